// Argument block and launchers of the single-GPU pull / push / lookup kernels (sparse_local.cu).
#pragma once
#include "sparse_fused.h"

namespace psb {

struct LocalArgs {
    unsigned n, bag_size, dim, flags;
    unsigned item_len, big_min, big_len;   // occurrences per work item of a lane group; a key with more than big_min is cut into
                                           // CTA items of big_len (set by launch_local_pull)
    unsigned once_shift;         // push: a block of keys that occur once has 1 << once_shift positions (set by launch_local_push)
    const long long* keys;       // [n]
    void* out;                   // [n / bag_size][dim] fp32, or bf16 with FUSED_OUT_BF16
    const float* grads;          // [n / bag_size][dim]
    const TableView* table;      // device memory, see FusedArgs::table
    KernelCtl* ctl;
    const KernelCtl* plan_ctl;   // push: control block of the pull family
    unsigned* counters;          // [2][16] per epoch parity of the pull: 0 distinct keys, 2 occurrences listed,
                                 // 3 work items, 5 keys with several items, 6 work items of whole CTAs, 8 new rows and
                                 // 9 new entries of the index (one 64-bit word)
    unsigned long long limit_ns;
    unsigned long long* prof;
    unsigned long long* usage_mirror;   // pinned host words {row_bump, free_count}
    unsigned* plan_gen;          // GpuTable's erase counter when the plan was made
    // ---- the plan, filled by a pull -------------------------------------------------------------------------------
    // A distinct key is known by the number of the entry that met it first: a place in the batch, below n.
    unsigned* id_of;             // [N] the key's number, of every position (kNoSlot: the index was full)
    unsigned* rank_of;           // [N] how many earlier occurrences the position's key has (upper bit: behind the owner's) ...
    unsigned* push_row;          // [N] ... and, in the same memory, from phase C on: the table row of a key that occurs
                                 //     once, kRemoteRow where a work item covers the position, kNoRow without a row
    unsigned* row_of;            // [N] table row of every position (kNoRow: reads as the initial value)
    unsigned* slot_of_id;        // [N] table slot of the key with this number (kNoSlot: nobody's number)
    unsigned* own;               // [N] occurrences of the key with this number in the tile of that entry
    unsigned* count;             // [N] its occurrences in all other tiles: zero between calls
    uint2* info;                 // [N] of the key with this number: table row (kNoRow: none), 1 + first of its occurrences or 0
    unsigned* new_list;          // [N] slots whose rows this call attached
    unsigned* occ;               // [N] positions of the repeated keys, one contiguous segment per key (phase A: slots of
                                 //     the keys that this call inserted)
    uint4* items;                // [N/2] {row, first occurrence, length | items of the key << 8, 1 + hot index or 0}
    uint4* big_items;            // [2 (N/256) + 1] the same for keys that whole CTAs sum (length | items << 11)
    long long* key_copy;         // [N] lookup: the keys, in case a push follows
    float* hot_sum;              // [N/16 + 1][dim] sums of keys with several items: zero between calls
    unsigned* hot_cnt;           // [N/16 + 1] items of the key that have arrived: zero between calls
    OptConfig opt;
};

// Arrays of the general push (FusedArgs) that a plan of the local pull is turned into.
struct GeneralPlan {
    int* inverse;
    long long* send_keys;
    unsigned* send_ret;
    unsigned* res_slot;
    unsigned* in_cnt;
};

// Rows of hot_sum / hot_cnt that a batch of n keys can need.
unsigned local_hot_rows(unsigned n);
// Entries of big_items that a batch of n keys can need.
unsigned local_big_items(unsigned n);
// Shared-memory attributes, and how many CTAs of the two pull shapes the GPU holds at a time.
int local_prepare(int* pull_blocks_small, int* pull_blocks_wide, int num_sms);
// `wide`: 1024-thread CTAs (at most max_blocks SMs are used); otherwise 256 threads.
int launch_local_pull(const LocalArgs& a, int max_blocks, bool wide, void* stream);
int launch_local_push(const LocalArgs& a, int max_blocks, bool wide, bool sync, unsigned table_slots, void* stream);
int launch_local_lookup(const LocalArgs& a, int max_blocks, bool wide, void* stream);
int launch_plan_to_general(const LocalArgs& a, const GeneralPlan& g, int num_sms, void* stream);

}  // namespace psb
