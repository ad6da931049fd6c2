// Pull, push and read-only lookup of a table that lives on ONE GPU (world == 1): the owner, the requester and the
// transport of the fused kernels of sparse_fused.cu collapse into one device, so nothing is staged per owner and the
// table's own index is the dedup structure of a batch.
//
// local_pull_kernel (cooperative)
//   A  a CTA folds the duplicates of a tile of keys in shared memory; one thread per distinct key of the tile finds or
//      inserts it in the table and swaps the entry's own number (its place in the batch) into the slot's `aux` word, which
//      is kNoRow at rest. Whoever swaps first owns the key; everybody else reads the owner's number there. From here on
//      all bookkeeping is in arrays indexed by that number. The occurrences are counted there, and the count returned
//      tells each tile where its own begin.
//   B  per number: a new row is initialised, a key that occurs more than once gets a segment
//      of the occurrence list and work items for the push
//   C  per position: row and segment of its key's number; the `aux` words go back to rest; then the rows are gathered and
//      pooled
//   What bounds A is the number of scattered requests to the index (a few hundred MB: about 25 G/s for the whole GPU, whatever
//   their width): one probe (1.5 with the chains), one swap and one reset per (tile, key), none per position.
// local_push_kernel (plain launch, no barrier)
//   every distinct row is touched once: the gradients of a repeated key are summed in registers straight from the
//   gradient buffer (no aggregation rows, no fp32 atomics except one partial row per item of a key with more than
//   item_len occurrences, whose last item applies the step), a key that occurs once is updated from its gradient row
// local_lookup_kernel (plain launch, no barrier)
//   a pull that inserts nothing: probe and gather, one pass, no dedup. The keys are kept so that a push that follows
//   all the same can have its plan made then.
//
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "sparse_local.h"

namespace psb {

namespace {

// How the occurrences of a repeated key are cut into work items of the push. Up to item_len go to one lane group, and a key with
// more has several such items. Their sums meet in one row of fp32 atomics, which costs about 80 ns each time: with one
// row per 32 occurrences the hottest key of 4 Mi Zipf(1.05) keys (210 000 of them) took 548 us. So a key with more than
// big_min is summed by whole CTAs, big_len occurrences each. Those items are a string of memory latencies and CTA
// barriers (eight rows requested at a time), up to 10 us each even when short (with big_min 128 the five hundred of a 213 Ki batch took 50 of the
// push's 78 us on 96 SMs): few of them, and no longer than the batch allows. By the batch's size alone: the cost is that of the
// longest item against the push's time. Pull and push in us with the first / second / third cut for all sizes, Adagrad:
//   dim 64, Zipf 1.05      64 Ki 57.2 / 58.4 / 59.7   256 Ki 110 / 113 / 115   1 Mi 292 / 292 / 289   4 Mi 969 / 946 / 950
//   dim 16, Zipf 1.1       64 Ki 54.6 / 53.8 / 54.3   256 Ki  71 /  71 /  72   1 Mi 200 / 187 / 185   4 Mi 682 / 611 / 608
//   dim 128, Zipf 1.1      64 Ki 70.4 / 70.1 / 77.6   256 Ki 146 / 150 / 159   1 Mi 412 / 410 / 409   2 Mi 761 / 752 / 748
//   dim 128 on 96 SMs      64 Ki 70.7 / 72.4 / 72.1   256 Ki 162 / 159 / 156   1 Mi 512 / 475 / 465   2 Mi 984 / 892 / 865
// Where two cuts cross depends on dim and SMs (first and second: near 2^17 keys at dim 16, 2^19 at dim 128 on all SMs), but
// these lines cost nowhere more than 3 us or 5 %.
struct Cut {
    unsigned item_len, big_min, big_len;
};
constexpr unsigned kMinItem = 16, kMinBig = 256;
inline Cut cut_of(unsigned n) {
    if (n < (1u << 18)) return {kMinItem, 1024, kMinBig};
    if (n < (1u << 21)) return {32, 2048, 512};
    return {32, 2048, 1024};
}
constexpr unsigned kDupRow = kRemoteRow;   // LocalArgs::push_row: the position's key is handled by a work item

constexpr unsigned kBehindOwner = 0x80000000u;   // LocalArgs::rank_of: counted from the end of the owner's own occurrences

struct Slot4 {
    long long key;
    unsigned row, aux;
};
// One slot in one 16-byte access that does not allocate in L1 (other CTAs change the words behind our back). Two 64-bit
// elements, since each element of a vector access is single-copy atomic by itself: the key is read whole beside a 64-bit
// CAS of another CTA. Row and aux may be older than it; each user re-checks what it needs with an atomic or after a barrier.
__device__ __forceinline__ Slot4 ld_slot(const Slot* p) {
    unsigned long long key, rest;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];" : "=l"(key), "=l"(rest) : "l"(p) : "memory");
    Slot4 s;
    s.key = (long long)key;
    s.row = (unsigned)rest;
    s.aux = (unsigned)(rest >> 32);
    return s;
}

__device__ __forceinline__ uint2 pack4(const float4& v) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    uint2 p;
    p.x = *(const unsigned*)&lo;
    p.y = *(const unsigned*)&hi;
    return p;
}

// Initial value of four columns of a key that has no row: rare, so out of line.
__device__ __noinline__ float4 init_row4(long long key, unsigned d, unsigned long long seed, float range) {
    float4 v;
    v.x = init_uniform(key, d + 0, seed, range);
    v.y = init_uniform(key, d + 1, seed, range);
    v.z = init_uniform(key, d + 2, seed, range);
    v.w = init_uniform(key, d + 3, seed, range);
    return v;
}

// The grid barrier of common.cuh in two halves, so that work can stand between arriving and waiting. An error status does
// not break it: no CTA of these kernels leaves early except on a time-out, so every call ends with its scratch clean.
// It carries one bit: whether any thread of any CTA arrived with `flag`, in the upper half of the count and then in the step
// of the generation (a word of its own, read behind the barrier, cost every pull 0.5 to 1 us).
__device__ __forceinline__ unsigned grid_arrive(KernelCtl* ctl, unsigned nblocks, bool flag = false) {
    const unsigned me = __syncthreads_or(flag) ? 0x10001u : 1u;
    unsigned gen = 0;
    if (threadIdx.x == 0) {
        gen = ld_acquire_gpu(&ctl->bar_gen);
        __threadfence();
        const unsigned arrived = atomicAdd(&ctl->bar_count, me) + me;
        if ((arrived & 0xffffu) == nblocks) {
            ctl->bar_count = 0;
            __threadfence();
            atomicAdd(&ctl->bar_gen, arrived >> 16 ? 3u : 1u);
        }
    }
    return gen;   // meaningful in thread 0
}
// `flagged` (shared memory, or null): set to that bit.
__device__ __forceinline__ bool grid_wait(KernelCtl* ctl, unsigned gen, unsigned long long limit_ns, unsigned where, unsigned* flagged = nullptr) {
    int ok = 1;
    if (threadIdx.x == 0) {
        const unsigned long long t0 = global_timer_ns();
        unsigned spins = 0, now;
        while ((now = ld_acquire_gpu(&ctl->bar_gen)) == gen) {
            if ((++spins & 63u) == 0) {
                if (ld_acquire_gpu(&ctl->status) == kStTimeout) { ok = 0; break; }
                if (global_timer_ns() - t0 > limit_ns) {
                    set_status(ctl, kStTimeout, where);
                    ok = 0;
                    break;
                }
            }
        }
        if (flagged != nullptr) *flagged = now - gen != 1u;
        __threadfence();
    }
    return __syncthreads_and(ok) != 0;
}

enum Where : unsigned { W_P1 = 1, W_P3A = 4, W_P3B = 5, W_INDEX_FULL = 9, W_POOL_FULL = 10, W_RESERVED_KEY = 12, W_NOROW = 38 };

#define PROF(slot)                                                                                      \
    do {                                                                                                \
        if (a.prof != nullptr && blockIdx.x == 0 && threadIdx.x == 0) a.prof[slot] = global_timer_ns(); \
    } while (0)
#define PROF_CTA(k)                                                                                                  \
    do {                                                                                                             \
        if (a.prof != nullptr && threadIdx.x == 0 && blockIdx.x < kProfMaxCtas)                                      \
            a.prof[16 + (k) * kProfMaxCtas + blockIdx.x] = global_timer_ns();                                        \
    } while (0)

// Gather + pool: bags [b_lo, b_hi) of this CTA, `rows` = table row (or kNoRow) of every key position.
__device__ __forceinline__ void gather_bags(const TableView& T, const LocalArgs& a, const unsigned* rows, unsigned b_lo, unsigned b_hi) {
    const unsigned L = a.bag_size, lanes = lanes_for_dim(a.dim);
    const unsigned lgroup = threadIdx.x / lanes, lgroups = blockDim.x / lanes, lane = threadIdx.x % lanes;
    const bool out16 = (a.flags & FUSED_OUT_BF16) != 0;
    float* outf = (float*)a.out;
    __nv_bfloat16* outh = (__nv_bfloat16*)a.out;
    if (L == 1) {
        // Four bags per lane group and iteration, the row indexes of the next four requested before this four's rows
        // are stored: the chain index -> slab pointer -> row is then never exposed twice.
        constexpr int kBags = 4;
        unsigned nx[kBags];
#pragma unroll
        for (int k = 0; k < kBags; ++k) {
            const unsigned b = b_lo + (unsigned)k * lgroups + lgroup;
            nx[k] = b < b_hi ? rows[b] : kNoRow;
        }
        for (unsigned b0 = b_lo; b0 < b_hi; b0 += lgroups * kBags) {
            const float* src[kBags];
#pragma unroll
            for (int k = 0; k < kBags; ++k) src[k] = nx[k] < kRowPending ? T.row_ptr(nx[k]) : nullptr;
#pragma unroll
            for (int k = 0; k < kBags; ++k) {
                const unsigned b = b0 + (unsigned)(kBags + k) * lgroups + lgroup;
                nx[k] = b < b_hi ? rows[b] : kNoRow;
            }
            for (unsigned d = lane * 4; d < a.dim; d += lanes * 4) {
                float4 v[kBags];
#pragma unroll
                for (int k = 0; k < kBags; ++k) {
                    const unsigned b = b0 + (unsigned)k * lgroups + lgroup;
                    if (b < b_hi) v[k] = src[k] != nullptr ? *(const float4*)(src[k] + d) : init_row4(a.keys[b], d, T.init_seed, T.init_range);
                }
#pragma unroll
                for (int k = 0; k < kBags; ++k) {
                    const unsigned b = b0 + (unsigned)k * lgroups + lgroup;
                    if (b >= b_hi) continue;
                    if (out16) *(uint2*)(outh + (size_t)b * a.dim + d) = pack4(v[k]);
                    else *(float4*)(outf + (size_t)b * a.dim + d) = v[k];
                }
            }
        }
        return;
    }
    const float scale = (a.flags & FUSED_MEAN) ? 1.0f / (float)L : 1.0f;
    for (unsigned b = b_lo + lgroup; b < b_hi; b += lgroups) {
        const unsigned* br = rows + (size_t)b * L;
        const long long* bk = a.keys + (size_t)b * L;
        for (unsigned d = lane * 4; d < a.dim; d += lanes * 4) {
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            auto fetch = [&](unsigned j) -> float4 {
                const unsigned row = br[j];
                if (row < kRowPending) return *(const float4*)(T.row_ptr(row) + d);
                return init_row4(bk[j], d, T.init_seed, T.init_range);
            };
            auto add = [&](const float4& v) { acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w; };
            unsigned j = 0;
            for (; j + 4 <= L; j += 4) {   // added front to back, requested four at a time
                const float4 v0 = fetch(j), v1 = fetch(j + 1), v2 = fetch(j + 2), v3 = fetch(j + 3);
                add(v0); add(v1); add(v2); add(v3);
            }
            for (; j < L; ++j) add(fetch(j));
            acc.x *= scale; acc.y *= scale; acc.z *= scale; acc.w *= scale;
            if (out16) *(uint2*)(outh + (size_t)b * a.dim + d) = pack4(acc);
            else *(float4*)(outf + (size_t)b * a.dim + d) = acc;
        }
    }
}

// A reserved key refuses the whole batch, but it is found when other CTAs have inserted their keys (a barrier in front of
// the first insertion cost 1.5 us of a step of 8192 keys, 4.7 us of 65536). The refused call takes them out again: a slot
// that was empty before the call ends no chain but those of the call's own keys, so it may be empty again. Rows go
// to the free stack; whoever gets one initialises it.
__device__ __noinline__ void undo_inserts(const TableView* table, const unsigned* new_rows, const unsigned* new_keys, const unsigned* counts,
                                          const unsigned* slot_of_id, unsigned n) {
    const TableView& T = *table;
    const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
    const unsigned n_rows = __ldcg(counts), n_keys = __ldcg(counts + 1);
    for (unsigned j = tid; j < n_rows; j += nthreads) {
        const unsigned slot = __ldcg(new_rows + j), row = __ldcg(&T.slots[slot].row);
        T.slots[slot].row = kNoRow;
        T.free_rows[atomicAdd(T.free_count, 1)] = row;
    }
    for (unsigned j = tid; j < n_keys; j += nthreads) T.slots[__ldcg(new_keys + j)].key = kEmptyKey;
    for (unsigned u = tid; u < n; u += nthreads) {
        const unsigned slot = __ldcg(slot_of_id + u);
        if (slot != kNoSlot) T.slots[slot].aux = kNoRow;
    }
    if (tid == 0) atomicAdd(T.n_items, 0ull - n_keys);
}

// Tile of the shared-memory dedup: positions per tile, and twice as many table slots (load at most one half).
template <int kThreads> struct Tile {
    static constexpr int kPer = kThreads >= 1024 ? 2 : 4;
    static constexpr int kKeys = kThreads * kPer;
    static constexpr int kSlots = 2 * kKeys;
    static constexpr size_t kSmem = (size_t)kSlots * (8 + 4) + (size_t)kKeys * 2;
};

// 1 Mi keys of dim 64, Zipf(1.05), 8 Mi rows: 64 + 14 + 82 us for A, B, C (the general kernel: 91 for dedup and resolve, 141 for
// the gather, 4.9 TB/s there now); 8192 keys of dim 16: 8 + 7 + 2 us, a handful of memory latencies and two barriers.
// Both CTA shapes fill the register file with 64 registers a thread; the 1024-thread one is for set_sm_budget.
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads) local_pull_kernel(const LocalArgs a) {
    using TL = Tile<kThreads>;
    constexpr int kPer = TL::kPer;
    extern __shared__ __align__(16) unsigned char s_raw[];
    unsigned long long* s_key = (unsigned long long*)s_raw;              // [kSlots] key; after the resolve step (slot, base)
    unsigned* s_cnt = (unsigned*)(s_key + TL::kSlots);                   // [kSlots] occurrences in the tile
    unsigned short* s_list = (unsigned short*)(s_cnt + TL::kSlots);      // [kKeys] occupied slots
    __shared__ unsigned s_n, s_sum[3], s_base[3];
    const unsigned nblocks = gridDim.x;
    const unsigned tid = blockIdx.x * kThreads + threadIdx.x, nthreads = nblocks * kThreads;
    const unsigned wlane = threadIdx.x & 31u, lt = (1u << wlane) - 1u;
    if (ld_acquire_gpu(&a.ctl->status) != 0u) return;
    const unsigned epoch = *((volatile unsigned*)&a.ctl->epoch) + 1u;
    const unsigned par = epoch & 1u;
    unsigned* cnt = a.counters + par * 16;   // see LocalArgs::counters
    const TableView T = *a.table;
    PROF(0);
    PROF_CTA(0);

    // Every CTA owns a contiguous range of bags, cut into tiles of equal length.
    const unsigned L = a.bag_size, nbags = a.n / L;
    const unsigned per = (nbags + nblocks - 1) / nblocks;
    const unsigned b_lo = min(nbags, blockIdx.x * per), b_hi = min(nbags, b_lo + per);
    const unsigned lo = b_lo * L, hi = b_hi * L;

    // ---- A ------------------------------------------------------------------------------------------------------
    bool reserved = false;
    const unsigned ntiles = (hi - lo + TL::kKeys - 1) / TL::kKeys;
    const unsigned tlen = ntiles ? (hi - lo + ntiles - 1) / ntiles : 0;
    for (unsigned t0 = lo; t0 < hi; t0 += tlen) {
        const unsigned t1 = min(hi, t0 + tlen);
        for (unsigned s = threadIdx.x; s < (unsigned)TL::kSlots / 2; s += kThreads)
            ((ulonglong2*)s_key)[s] = make_ulonglong2((unsigned long long)kEmptyKey, (unsigned long long)kEmptyKey);
        for (unsigned s = threadIdx.x; s < (unsigned)TL::kSlots / 4; s += kThreads) ((uint4*)s_cnt)[s] = make_uint4(0u, 0u, 0u, 0u);
        if (threadIdx.x == 0) { s_n = 0; s_sum[0] = s_sum[1] = s_sum[2] = 0; }
        long long key[kPer];
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const unsigned i = t0 + (unsigned)q * kThreads + threadIdx.x;
            key[q] = kEmptyKey;
            if (i < t1) {
                key[q] = a.keys[i];
                if (key[q] <= kTombstoneKey) {   // the two reserved values can never be stored
                    reserved = true;
                    key[q] = kEmptyKey;
                }
            }
        }
        __syncthreads();
        unsigned hs[kPer], rank[kPer];
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            hs[q] = 0xFFFFFFFFu;
            if (key[q] == kEmptyKey) continue;
            unsigned h = (unsigned)(slot_hash(key[q]) >> 40) & (TL::kSlots - 1);
            for (;;) {   // ends: the table holds twice as many slots as the tile has keys
                unsigned long long cur = *((volatile unsigned long long*)&s_key[h]);
                if (cur == (unsigned long long)kEmptyKey) {
                    cur = atomicCAS(&s_key[h], (unsigned long long)kEmptyKey, (unsigned long long)key[q]);
                    if (cur == (unsigned long long)kEmptyKey) {
                        s_list[atomicAdd(&s_n, 1u)] = (unsigned short)h;
                        break;
                    }
                }
                if (cur == (unsigned long long)key[q]) break;
                h = (h + 1) & (TL::kSlots - 1);
            }
            hs[q] = h;
            rank[q] = atomicAdd(&s_cnt[h], 1u);
        }
        __syncthreads();
        // Resolve. Sweeps over the thread's entries, so that their probes, and then their atomics, are in flight together.
        const unsigned m = s_n, tile_keys = t1 - t0;
        constexpr unsigned kDone = 0xFFFFFFF0u;   // probes[q]: found; kDone + 1: no entry, or the index is full
        unsigned eslot[kPer], probes[kPer], owner[kPer], before[kPer];
        bool won[kPer], inserted[kPer];
        Slot4 c[kPer];
        bool pending = false;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const unsigned e = (unsigned)q * kThreads + threadIdx.x;
            inserted[q] = won[q] = false;
            probes[q] = kDone + 1u;
            if (e < m) {
                probes[q] = 0;
                pending = true;
                eslot[q] = (unsigned)(slot_hash((long long)s_key[s_list[e]]) & T.mask);
                c[q] = ld_slot(T.slots + eslot[q]);
            }
        }
        while (pending) {
            pending = false;
#pragma unroll
            for (int q = 0; q < kPer; ++q) {
                if (probes[q] >= kDone) continue;
                const long long k = (long long)s_key[s_list[(unsigned)q * kThreads + threadIdx.x]];
                if (c[q].key == k) { probes[q] = kDone; continue; }
                if (c[q].key == kEmptyKey) {
                    const long long prev = (long long)atomicCAS((unsigned long long*)&T.slots[eslot[q]].key, (unsigned long long)kEmptyKey, (unsigned long long)k);
                    if (prev == kEmptyKey || prev == k) {
                        inserted[q] = prev == kEmptyKey;
                        c[q].row = c[q].aux = kNoRow;   // as far as known
                        probes[q] = kDone;
                        continue;
                    }
                }
                if (++probes[q] >= T.max_probe) {
                    probes[q] = kDone + 1u;
                    set_soft_status(a.ctl, kStOom, W_INDEX_FULL);
                    continue;
                }
                eslot[q] = (unsigned)((eslot[q] + 1ull) & T.mask);
                pending = true;
            }
#pragma unroll
            for (int q = 0; q < kPer; ++q)
                if (probes[q] < kDone) c[q] = ld_slot(T.slots + eslot[q]);
        }
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            if (probes[q] != kDone) continue;
            const unsigned id = t0 + (unsigned)q * kThreads + threadIdx.x;
            owner[q] = c[q].aux;
            if (owner[q] == kNoRow) {
                const unsigned prev = atomicCAS(&T.slots[eslot[q]].aux, kNoRow, id);
                won[q] = prev == kNoRow;
                owner[q] = won[q] ? id : prev;
            }
        }
#pragma unroll
        for (int q = 0; q < kPer; ++q)
            if (probes[q] == kDone) {
                // the owner's own occurrences come first and need no atomic (three entries in four, in a batch of 1 Mi)
                const unsigned n_here = s_cnt[s_list[(unsigned)q * kThreads + threadIdx.x]];
                before[q] = won[q] ? n_here : atomicAdd(&a.count[owner[q]], n_here) | kBehindOwner;
            }
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const unsigned e = (unsigned)q * kThreads + threadIdx.x;
            bool attached = false;
            if (won[q]) {
                unsigned row = c[q].row;
                if (row == kNoRow) {
                    bool oom = false;
                    attached = table_attach_row(T, eslot[q], &oom);
                    if (oom) set_soft_status(a.ctl, kStOom, W_POOL_FULL);
                    row = *((volatile unsigned*)&T.slots[eslot[q]].row);
                }
                a.info[t0 + e] = make_uint2(row < kRowPending ? row : kNoRow, 0u);
            }
            if (e < tile_keys) {
                a.slot_of_id[t0 + e] = won[q] ? eslot[q] : kNoSlot;
                a.own[t0 + e] = won[q] ? before[q] : 0u;
            }
            if (won[q]) before[q] = 0;
            // counters: one shared-memory atomic per warp, one global one per tile (new rows and entries, rare, one per warp)
            const unsigned wm = __ballot_sync(0xffffffffu, won[q]), im = __ballot_sync(0xffffffffu, inserted[q]);
            const unsigned am = __ballot_sync(0xffffffffu, attached);
            if (wlane == 0) {
                if (wm) atomicAdd(&s_sum[0], (unsigned)__popc(wm));
                if (im) atomicAdd(&s_sum[1], (unsigned)__popc(im));
            }
            if (am | im) {
                unsigned long long ab = 0;
                if (wlane == 0) ab = atomicAdd((unsigned long long*)&cnt[8], (unsigned long long)__popc(im) << 32 | (unsigned)__popc(am));
                ab = __shfl_sync(0xffffffffu, ab, 0);
                if (attached) a.new_list[(unsigned)ab + __popc(am & lt)] = eslot[q];
                if (inserted[q]) a.occ[(unsigned)(ab >> 32) + __popc(im & lt)] = eslot[q];   // for undo_inserts
            }
        }
        __syncthreads();   // every entry has read its key
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const unsigned e = (unsigned)q * kThreads + threadIdx.x;
            if (e < m) s_key[s_list[e]] = probes[q] == kDone ? ((unsigned long long)owner[q] << 32) | before[q] : (unsigned long long)kNoSlot << 32;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            if (s_sum[0]) atomicAdd(&cnt[0], s_sum[0]);
            if (s_sum[1]) atomicAdd(T.n_items, (unsigned long long)s_sum[1]);
        }
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const unsigned i = t0 + (unsigned)q * kThreads + threadIdx.x;
            if (i < t1) {
                unsigned id = kNoSlot, first = 0;
                if (hs[q] != 0xFFFFFFFFu) {
                    const unsigned long long p = s_key[hs[q]];
                    id = (unsigned)(p >> 32);
                    first = (unsigned)p;
                }
                a.id_of[i] = id;
                a.rank_of[i] = first + (id != kNoSlot ? rank[q] : 0u);
            }
        }
        __syncthreads();   // the tables are emptied for the next tile
    }
    PROF_CTA(1);
    unsigned gen = grid_arrive(a.ctl, nblocks, reserved);
    if (!grid_wait(a.ctl, gen, a.limit_ns, W_P1, &s_n)) return;
    if (s_n != 0u) {   // a reserved key in the batch
        undo_inserts(a.table, a.new_list, a.occ, cnt + 8, a.slot_of_id, a.n);
        // reported only now: a CTA that had not started yet would take the word for an earlier call's and leave
        if (tid == 0) set_status(a.ctl, kStError, W_RESERVED_KEY);
        return;
    }
    PROF(1);
    PROF(2);

    // ---- B ------------------------------------------------------------------------------------------------------
    const unsigned n_new = *((volatile unsigned*)&cnt[8]);
    if (blockIdx.x == 0 && threadIdx.x == 0 && a.usage_mirror != nullptr) {
        // the allocation counters that the host's next reservation reads (no copy engine, no extra launch)
        a.usage_mirror[0] = *((volatile unsigned*)T.row_bump);
        a.usage_mirror[1] = (unsigned)*((volatile int*)T.free_count);
        *a.plan_gen = *((volatile unsigned*)T.erase_gen);
    }
    {
        constexpr int kU = 4;   // numbers per thread
        for (unsigned u0 = blockIdx.x * (kThreads * kU); u0 < a.n; u0 += nthreads * kU) {
            unsigned row[kU], c[kU];
            unsigned seg = 0, items = 0, multi = 0;
#pragma unroll
            for (int q = 0; q < kU; ++q) {
                const unsigned u = u0 + (unsigned)q * kThreads + threadIdx.x;
                c[q] = 0;
                if (u >= a.n) continue;
                c[q] = __ldcg(a.count + u);
                const unsigned own = __ldcg(a.own + u);
                if (c[q] != 0u) a.count[u] = 0;
                c[q] += own;
            }
#pragma unroll
            for (int q = 0; q < kU; ++q) {
                const unsigned u = u0 + (unsigned)q * kThreads + threadIdx.x;
                if (c[q] >= 2u) row[q] = __ldcg(&a.info[u].x);
            }
#pragma unroll
            for (int q = 0; q < kU; ++q)
                if (c[q] >= 2u) {
                    seg += c[q];
                    if (c[q] <= a.big_min) {
                        items += (c[q] + a.item_len - 1) / a.item_len;
                        multi += c[q] > a.item_len ? 1u : 0u;
                    }
                }
            // exclusive offsets inside the warp, the warp's inside the CTA, the CTA's from the global counters
            unsigned xs = seg, xi = items, xm = multi;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned ys = __shfl_up_sync(0xffffffffu, xs, o), yi = __shfl_up_sync(0xffffffffu, xi, o), ym = __shfl_up_sync(0xffffffffu, xm, o);
                if (wlane >= (unsigned)o) { xs += ys; xi += yi; xm += ym; }
            }
            unsigned bs = 0, bi = 0, bm = 0;
            if (threadIdx.x < 3) s_sum[threadIdx.x] = 0;
            __syncthreads();
            if (wlane == 31u && xs) {
                bs = atomicAdd(&s_sum[0], xs);
                if (xi) bi = atomicAdd(&s_sum[1], xi);
                if (xm) bm = atomicAdd(&s_sum[2], xm);
            }
            __syncthreads();
            if (threadIdx.x < 3) s_base[threadIdx.x] = s_sum[threadIdx.x] ? atomicAdd(&cnt[threadIdx.x == 2 ? 5 : 2 + threadIdx.x], s_sum[threadIdx.x]) : 0u;
            __syncthreads();
            bs = __shfl_sync(0xffffffffu, bs, 31) + s_base[0] + xs - seg;
            bi = __shfl_sync(0xffffffffu, bi, 31) + s_base[1] + xi - items;
            bm = __shfl_sync(0xffffffffu, bm, 31) + s_base[2] + xm - multi;
#pragma unroll
            for (int q = 0; q < kU; ++q) {
                const bool dup = c[q] >= 2u;
                const bool big = c[q] > a.big_min;
                const unsigned nch = dup && !big ? (c[q] + a.item_len - 1) / a.item_len : 0u;
                unsigned mid = 0;
                if (dup) {
                    a.info[u0 + (unsigned)q * kThreads + threadIdx.x].y = bs + 1u;   // 0 stays the mark of a key that occurs once
                    if (big) {   // a handful of keys at the head of the batch
                        const unsigned nb = (c[q] + a.big_len - 1) / a.big_len, b0 = atomicAdd(&cnt[6], nb), md = atomicAdd(&cnt[5], 1u) + 1u;
                        for (unsigned j = 0; j < nb; ++j)
                            a.big_items[b0 + j] = make_uint4(row[q], bs + j * a.big_len, min(a.big_len, c[q] - j * a.big_len) | (nb << 11), md);
                    } else if (nch > 1u) mid = ++bm;
                    else a.items[bi] = make_uint4(row[q], bs, c[q], 0u);
                }
                // the items of a hot key are written by the whole warp
                unsigned todo = __ballot_sync(0xffffffffu, nch > 1u);
                while (todo) {
                    const int src = __ffs(todo) - 1;
                    todo &= todo - 1;
                    const unsigned r = __shfl_sync(0xffffffffu, row[q], src), o = __shfl_sync(0xffffffffu, bs, src), cc = __shfl_sync(0xffffffffu, c[q], src);
                    const unsigned it = __shfl_sync(0xffffffffu, bi, src), n = __shfl_sync(0xffffffffu, nch, src), md = __shfl_sync(0xffffffffu, mid, src);
                    for (unsigned j = wlane; j < n; j += 32)
                        a.items[it + j] = make_uint4(r, o + j * a.item_len, min(a.item_len, cc - j * a.item_len) | (n << 8), md);
                }
                if (dup) { bs += c[q]; bi += nch; }
            }
        }
        // rows attached by this call
        const unsigned lanes = lanes_for_dim(a.dim);
        for (unsigned j = tid / lanes; j < n_new; j += nthreads / lanes) {
            const unsigned slot = a.new_list[j];
            row_init(T, T.row_ptr(T.slots[slot].row), T.slots[slot].key, tid % lanes, lanes);
        }
    }
    PROF_CTA(2);
    gen = grid_arrive(a.ctl, nblocks);
    if (!grid_wait(a.ctl, gen, a.limit_ns, W_P3A)) return;
    PROF(3);
    PROF(4);
    PROF(5);

    // ---- C ------------------------------------------------------------------------------------------------------
    {
        constexpr int kU = 4;
        for (unsigned i0 = lo + threadIdx.x; i0 < hi; i0 += kThreads * kU) {
            unsigned id[kU], rank[kU];
            uint2 f[kU];
#pragma unroll
            for (int q = 0; q < kU; ++q) {
                const unsigned i = i0 + (unsigned)q * kThreads;
                id[q] = i < hi ? a.id_of[i] : kNoSlot;
                rank[q] = i < hi ? a.rank_of[i] : 0u;
            }
#pragma unroll
            for (int q = 0; q < kU; ++q)
                if (id[q] != kNoSlot) f[q] = __ldcg(a.info + id[q]);
#pragma unroll
            for (int q = 0; q < kU; ++q) {
                const unsigned i = i0 + (unsigned)q * kThreads;
                if (i >= hi) continue;
                unsigned row = kNoRow, pr = kNoRow;
                if (id[q] != kNoSlot) {
                    pr = row = f[q].x;
                    if (f[q].y != 0u) {
                        const unsigned first = (rank[q] & kBehindOwner) ? __ldcg(a.own + id[q]) : 0u;
                        a.occ[f[q].y - 1u + first + (rank[q] & ~kBehindOwner)] = i;
                        pr = kDupRow;
                    }
                }
                a.row_of[i] = row;
                a.push_row[i] = pr;   // the same word as rank_of[i], which was read above
            }
        }
    }
    // The `aux` words go back to rest: scattered stores that nothing waits for here (in front of a barrier something would).
    for (unsigned u = tid; u < a.n; u += nthreads) {
        const unsigned slot = __ldcg(a.slot_of_id + u);
        if (slot != kNoSlot) T.slots[slot].aux = kNoRow;
    }
    __syncthreads();
    if (a.flags & FUSED_COPY_ROWS) gather_bags(T, a, a.row_of, b_lo, b_hi);
    if (blockIdx.x == 0 && threadIdx.x < 16) a.counters[(par ^ 1u) * 16 + threadIdx.x] = 0;
    PROF(6);
    if (blockIdx.x == 0 && threadIdx.x == 0) a.ctl->epoch = epoch;
}

// ---- push ---------------------------------------------------------------------------------------------------------
// kOpt: the update rule at compile time (-1: looked up per coordinate, and the slot count comes from the table).
template <int kOpt, bool kSync>
struct RowUpdate {
    static constexpr int kSlots = kOpt == OPT_ADAGRAD ? 1 : (kOpt == OPT_FTRL || kOpt == OPT_ADAM) ? 2 : 0;
    float4 w, s0, s1;
    __device__ __forceinline__ int slots(const TableView& T) const { return kOpt >= 0 ? kSlots : (int)T.n_opt_slots; }
    __device__ __forceinline__ void load(const TableView& T, const float* p, unsigned dim) {
        if (kSync) {
            w = *(const float4*)(p + (size_t)(T.n_opt_slots + 1) * dim);
            return;
        }
        w = *(const float4*)p;
        s0 = s1 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (slots(T) > 0) s0 = *(const float4*)(p + dim);
        if (slots(T) > 1) s1 = *(const float4*)(p + 2 * dim);
    }
    __device__ __forceinline__ void apply(const TableView& T, const OptConfig& opt, float* p, unsigned dim, const float4& g) {
        if (kSync) {
            w.x += g.x; w.y += g.y; w.z += g.z; w.w += g.w;
            *(float4*)(p + (size_t)(T.n_opt_slots + 1) * dim) = w;
            return;
        }
        opt_update<kOpt>(opt, w.x, s0.x, s1.x, g.x);
        opt_update<kOpt>(opt, w.y, s0.y, s1.y, g.y);
        opt_update<kOpt>(opt, w.z, s0.z, s1.z, g.z);
        opt_update<kOpt>(opt, w.w, s0.w, s1.w, g.w);
        *(float4*)p = w;
        if (slots(T) > 0) *(float4*)(p + dim) = s0;
        if (slots(T) > 1) *(float4*)(p + 2 * dim) = s1;
    }
};

template <bool kSync>
__device__ __forceinline__ void note_row(const TableView& T, KernelCtl* ctl, unsigned row) {
    if (kSync) {
        const unsigned bit = 1u << (row & 31u);
        if (!(atomicOr(&T.touched_bits[row >> 5], bit) & bit)) {
            const unsigned j = atomicAdd(T.touched_count, 1u);
            if (j < T.touched_cap) T.touched_list[j] = row;
            else set_soft_status(ctl, kStOom, W_NOROW);
        }
    }
    if (T.dirty_bits != nullptr) atomicOr(&T.dirty_bits[row >> 5], 1u << (row & 31u));
}

// 1 Mi keys of dim 64 (0.53 Mi distinct) with an Adagrad slot: 110 to 140 us for 830 MB, against 274 of the general kernel; the
// rest of the way to 125 us at copy speed is the tail of the longest work items. A kernel per update rule: at 64 registers the
// loops spill 268 bytes a thread with the rule looked up per coordinate, 20 with sgd, 24 Adagrad, 104 Adam, 116 FTRL.
// kFull: blocks of 32 positions (once_shift); with the shift in a register FTRL's push was 4 us longer at 512 Ki keys of
// dim 32 and at 256 Ki of dim 64, the others up to 1 us.
template <int kThreads, int kOpt, bool kSync, bool kFull>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads) local_push_kernel(const LocalArgs a) {
    if (ld_acquire_gpu(&a.ctl->status) != 0u || ld_acquire_gpu(&a.plan_ctl->status) != 0u) return;
    const unsigned epoch = *((volatile unsigned*)&a.ctl->epoch) + 1u;
    const unsigned* cnt = a.counters + (*((volatile const unsigned*)&a.plan_ctl->epoch) & 1u) * 16;
    const TableView T = *a.table;
    // rows were erased since the plan was made: ask the slots again (an erased key's gradient is dropped). A key that found
    // the pool exhausted is asked for in any case: it may have been given a row since.
    const bool stale = *((volatile unsigned*)T.erase_gen) != *((volatile unsigned*)a.plan_gen);
    // only Adam's rule changes with the call number; the others read their options where the parameters lie
    OptConfig stepped;
    if (kOpt < 0 || kOpt == OPT_ADAM) {
        stepped = a.opt;
        if (stepped.step_from_epoch) opt_set_step(stepped, epoch);
    }
    const OptConfig& opt = (kOpt < 0 || kOpt == OPT_ADAM) ? stepped : a.opt;
    const unsigned dim = a.dim, L = a.bag_size;
    const unsigned lanes = lanes_for_dim(dim);
    const unsigned tid = blockIdx.x * kThreads + threadIdx.x, nthreads = gridDim.x * kThreads;
    const unsigned group = tid / lanes, ngroups = nthreads / lanes, lane = tid % lanes;
    const unsigned wlane = threadIdx.x & 31u, gl0 = wlane / lanes * lanes;
    const unsigned gmask = (lanes >= 32u ? 0xffffffffu : ((1u << lanes) - 1u)) << gl0;
    const bool mean = L > 1 && (a.flags & FUSED_MEAN) != 0;
    const float scale = mean ? 1.0f / (float)L : 1.0f;
    auto grad4 = [&](unsigned pos, unsigned d) -> float4 {
        float4 v = *(const float4*)(a.grads + (size_t)(L == 1 ? pos : pos / L) * dim + d);
        if (mean) { v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale; }
        return v;
    };
    PROF(8);
    // ---- the head of a skewed batch: one CTA per work item, its lane groups share the occurrences ----------------------
    {
        const unsigned n_big = *((volatile const unsigned*)&cnt[6]);
        const unsigned lgroup = threadIdx.x / lanes, lgroups = kThreads / lanes;
        __shared__ float4 s_part[kThreads];
        __shared__ unsigned s_last;
        for (unsigned e = blockIdx.x; e < n_big; e += gridDim.x) {
            const uint4 it = a.big_items[e];
            const unsigned len = it.z & 2047u, n_parts = it.z >> 11;
            const unsigned* occ = a.occ + it.y;
            unsigned row = it.x;
            if (stale || row == kNoRow) row = T.slots[a.slot_of_id[a.id_of[occ[0]]]].row;
            if (row >= kRowPending) {
                if (threadIdx.x == 0) set_soft_status(a.ctl, kStOom, W_NOROW);
                continue;
            }
            float* sum = a.hot_sum + (size_t)(it.w - 1u) * dim;
            for (unsigned d0 = 0; d0 < dim; d0 += lanes * 4) {
                const unsigned d = d0 + lane * 4;
                float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                if (d < dim) {
                    auto add = [&](const float4& v) { acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w; };
                    constexpr int kBig = 8;
                    unsigned j = lgroup;
                    for (; j + (kBig - 1) * lgroups < len; j += kBig * lgroups) {
                        unsigned q[kBig];
                        float4 v[kBig];
#pragma unroll
                        for (int k = 0; k < kBig; ++k) q[k] = occ[j + k * lgroups];
#pragma unroll
                        for (int k = 0; k < kBig; ++k) v[k] = grad4(q[k], d);
#pragma unroll
                        for (int k = 0; k < kBig; ++k) add(v[k]);
                    }
                    for (; j < len; j += lgroups) add(grad4(occ[j], d));
                }
                s_part[threadIdx.x] = acc;
                __syncthreads();
                for (unsigned h = lgroups / 2; h > 0; h /= 2) {
                    if (lgroup < h) {
                        const float4 v = s_part[threadIdx.x + h * lanes];
                        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
                        s_part[threadIdx.x] = acc;
                    }
                    __syncthreads();
                }
                if (lgroup == 0 && d < dim) atomicAdd((float4*)(sum + d), acc);
            }
            // the item that arrives last finds the whole sum, applies the step and leaves sum and counter at zero
            if (lgroup == 0) __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) s_last = atomicAdd(&a.hot_cnt[it.w - 1u], 1u) + 1u == n_parts ? 1u : 0u;
            __syncthreads();
            if (s_last != 0u && lgroup == 0) {
                __threadfence();
                float* w = T.row_ptr(row);
                for (unsigned d = lane * 4; d < dim; d += lanes * 4) {
                    RowUpdate<kOpt, kSync> up;
                    up.load(T, w + d, dim);
                    const float4 g = __ldcg((const float4*)(sum + d));
                    __stcg((float4*)(sum + d), make_float4(0.f, 0.f, 0.f, 0.f));
                    up.apply(T, opt, w + d, dim, g);
                }
                if (lane == 0) {
                    a.hot_cnt[it.w - 1u] = 0;
                    note_row<kSync>(T, a.ctl, row);
                }
            }
            __syncthreads();
        }
    }
    PROF(13);
    // ---- repeated keys: one lane group per work item -----------------------------------------------------------
    const unsigned n_items = *((volatile const unsigned*)&cnt[3]);
    // A batch of occurrences is requested while the gradients of the one before it are on their way, across items too: a
    // batch then costs one memory latency, not two or three.
    constexpr int kBatch = 4;
    unsigned p[kBatch];   // the batch whose gradients are requested next
    auto batch_of = [&](const uint4& it, unsigned j) {
#pragma unroll
        for (int k = 0; k < kBatch; ++k) p[k] = j + k < (it.z & 255u) ? a.occ[it.y + j + k] : 0u;
    };
    uint4 nx = make_uint4(kNoRow, 0, 0, 0);
    if (group < n_items) {
        nx = a.items[group];
        batch_of(nx, 0);
    }
    for (unsigned e = group; e < n_items; e += ngroups) {
        const uint4 cur = nx;
        nx.z = 0;
        if (e + ngroups < n_items) nx = a.items[e + ngroups];
        const unsigned len = cur.z & 255u;
        unsigned row = cur.x;
        if (stale || row == kNoRow) row = T.slots[a.slot_of_id[a.id_of[p[0]]]].row;
        if (row >= kRowPending) {
            if (lane == 0) set_soft_status(a.ctl, kStOom, W_NOROW);
            batch_of(nx, 0);
            continue;
        }
        float* w = T.row_ptr(row);
        for (unsigned d = lane * 4;;) {
            const bool on = d < dim, last = d + lanes * 4 >= dim;   // dim need not fill the lanes
            RowUpdate<kOpt, kSync> up;
            if (cur.w == 0u && on) up.load(T, w + d, dim);
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            for (unsigned j = 0; j < len; j += kBatch) {
                float4 v[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; ++k)
                    if (on && j + k < len) v[k] = grad4(p[k], d);
                const bool more = j + kBatch < len;
                batch_of(more || !last ? cur : nx, more ? j + kBatch : 0);
#pragma unroll
                for (int k = 0; k < kBatch; ++k)
                    if (on && j + k < len) { acc.x += v[k].x; acc.y += v[k].y; acc.z += v[k].z; acc.w += v[k].w; }
            }
            if (on) {
                if (cur.w == 0u) up.apply(T, opt, w + d, dim, acc);
                else atomicAdd((float4*)(a.hot_sum + (size_t)(cur.w - 1u) * dim + d), acc);
            }
            if (last) break;
            d += lanes * 4;
        }
        if (cur.w != 0u) {
            // the item that arrives last finds the whole sum, applies the step and leaves sum and counter at zero
            __threadfence();
            __syncwarp(gmask);
            unsigned prev = 0;
            if (lane == 0) prev = atomicAdd(&a.hot_cnt[cur.w - 1u], 1u);
            prev = __shfl_sync(gmask, prev, gl0);
            if (prev + 1u != cur.z >> 8) continue;
            __threadfence();
            float* sum = a.hot_sum + (size_t)(cur.w - 1u) * dim;
            for (unsigned d = lane * 4; d < dim; d += lanes * 4) {
                RowUpdate<kOpt, kSync> up;
                up.load(T, w + d, dim);
                const float4 g = __ldcg((const float4*)(sum + d));
                __stcg((float4*)(sum + d), make_float4(0.f, 0.f, 0.f, 0.f));
                up.apply(T, opt, w + d, dim, g);
            }
            if (lane == 0) a.hot_cnt[cur.w - 1u] = 0;
        }
        if (lane == 0) note_row<kSync>(T, a.ctl, row);
    }
    PROF(10);
    PROF(11);
    PROF(14);
    PROF(15);
    PROF_CTA(3);
    // ---- keys that occur once: a warp takes a block of consecutive positions, its lane groups share the ones that qualify ---
    {
        // rows in flight per lane group: two where a row and its slots are at most three 16-byte loads a thread, else one (the
        // kernels spill a few values either way)
        constexpr int kIn = kOpt == OPT_FTRL || kOpt == OPT_ADAM || (kOpt < 0 && !kSync) ? 1 : 2;
        __shared__ uint2 s_todo[kThreads / 32][32];
        const unsigned warp = tid >> 5, nwarps = nthreads >> 5, gpw = 32u / lanes, g = wlane / lanes;
        const unsigned sh = kFull ? 5u : a.once_shift;
        const unsigned nblk = (a.n + (1u << sh) - 1u) >> sh;
        // Half of the blocks are dealt out by number, the rest from a counter to whoever is through with its work items, in
        // pieces that shrink towards the end (all of them dealt out left the CTAs with long items behind the others by half the
        // kernel's time; pieces of four to the end did the same to a batch of two blocks per warp).
        const unsigned fixed = max(1u, nblk / nwarps / 2u) * nwarps;
        auto rows_of = [&](unsigned b) -> unsigned { return b < nblk && wlane >> sh == 0u && (b << sh) + wlane < a.n ? a.push_row[(b << sh) + wlane] : kDupRow; };
        unsigned at = warp, end = 0;   // the last block handed out; the end of the piece it is from
        auto next_block = [&]() -> unsigned {
            if (at + nwarps < fixed) return at += nwarps;
            if (end != 0u && at + 1u < end) return ++at;
            if (fixed >= nblk) return nblk;
            const unsigned left = end == 0u ? nblk - fixed : (at < nblk ? nblk - at : 0u);
            const unsigned piece = min(8u, max(1u, left / (2u * nwarps)));
            unsigned b = 0;
            if (wlane == 0) b = atomicAdd(&a.ctl->pad[3], piece);
            at = fixed + __shfl_sync(0xffffffffu, b, 0);
            end = at + piece;
            return at;
        };
        unsigned blk = warp;
        unsigned nxr = rows_of(blk);
        while (blk < nblk) {
            const unsigned i0 = blk << sh;
            unsigned row = nxr;
            blk = next_block();
            nxr = rows_of(blk);
            if (row != kDupRow && (stale || row == kNoRow)) {
                const unsigned id = a.id_of[i0 + wlane];
                if (id != kNoSlot) row = T.slots[a.slot_of_id[id]].row;
            }
            if (row == kNoRow || row == kRowPending) {
                set_soft_status(a.ctl, kStOom, W_NOROW);
                row = kDupRow;
            }
            if (row != kDupRow && (kSync || T.dirty_bits != nullptr)) note_row<kSync>(T, a.ctl, row);
            // the positions that qualify, packed to the front of the warp's list; group g takes entries g, g + gpw, ...
            const unsigned mask = __ballot_sync(0xffffffffu, row != kDupRow), n_here = (unsigned)__popc(mask);
            __syncwarp();
            if (row != kDupRow) s_todo[threadIdx.x >> 5][__popc(mask & ((1u << wlane) - 1u))] = make_uint2(row, i0 + wlane);
            __syncwarp();
            for (unsigned e0 = g; e0 < n_here; e0 += gpw * kIn) {
                unsigned pos[kIn];
                float* w[kIn];
#pragma unroll
                for (int k = 0; k < kIn; ++k) {
                    const unsigned e = e0 + (unsigned)k * gpw;
                    w[k] = nullptr;
                    if (e < n_here) {
                        const uint2 t = s_todo[threadIdx.x >> 5][e];
                        w[k] = T.row_ptr(t.x);
                        pos[k] = t.y;
                    }
                }
                for (unsigned d = lane * 4; d < dim; d += lanes * 4) {
                    RowUpdate<kOpt, kSync> up[kIn];
                    float4 gv[kIn];
#pragma unroll
                    for (int k = 0; k < kIn; ++k)
                        if (w[k] != nullptr) {
                            gv[k] = grad4(pos[k], d);
                            up[k].load(T, w[k] + d, dim);
                        }
#pragma unroll
                    for (int k = 0; k < kIn; ++k)
                        if (w[k] != nullptr) up[k].apply(T, opt, w[k] + d, dim, gv[k]);
                }
            }
        }
    }
    PROF(12);
    // the last CTA out publishes the call's number (every CTA has read the old one by then)
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&a.ctl->done_blocks, 1u) == gridDim.x - 1u) {
        a.ctl->done_blocks = 0;
        a.ctl->pad[3] = 0;
        a.ctl->epoch = epoch;
    }
}

// ---- lookup ---------------------------------------------------------------------------------------------------------
// 1000 keys of dim 64: 21.2 us a call through the general kernel, 12.5 like this, most of it the host's; 151 663 keys of dim
// 128 in bags of 37: 63 and 18.4 us.
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads) local_lookup_kernel(const LocalArgs a) {
    if (ld_acquire_gpu(&a.ctl->status) != 0u) return;
    const TableView T = *a.table;
    const unsigned L = a.bag_size, nbags = a.n / L;
    const unsigned per = (nbags + gridDim.x - 1) / gridDim.x;
    const unsigned b_lo = min(nbags, blockIdx.x * per), b_hi = min(nbags, b_lo + per);
    const unsigned lo = b_lo * L, hi = b_hi * L;
    constexpr int kU = 4;   // keys per thread: their first probes are requested together
    for (unsigned i0 = lo + threadIdx.x; i0 < hi; i0 += kThreads * kU) {
        long long key[kU];
        unsigned h[kU];
        Slot4 s[kU];
#pragma unroll
        for (int q = 0; q < kU; ++q) {
            const unsigned i = i0 + (unsigned)q * kThreads;
            key[q] = i < hi ? a.keys[i] : kEmptyKey;
        }
#pragma unroll
        for (int q = 0; q < kU; ++q) {
            if (key[q] <= kTombstoneKey) continue;
            h[q] = (unsigned)(slot_hash(key[q]) & T.mask);
            s[q] = ld_slot(T.slots + h[q]);
        }
#pragma unroll
        for (int q = 0; q < kU; ++q) {
            const unsigned i = i0 + (unsigned)q * kThreads;
            if (i >= hi) continue;
            unsigned row = kNoRow;
            if (key[q] <= kTombstoneKey) {
                set_status(a.ctl, kStError, W_RESERVED_KEY);
            } else {
                unsigned p = 0;
                while (s[q].key != key[q] && s[q].key != kEmptyKey && ++p < T.max_probe) {
                    h[q] = (unsigned)((h[q] + 1ull) & T.mask);
                    s[q] = ld_slot(T.slots + h[q]);
                }
                if (s[q].key == key[q] && s[q].row < kRowPending) row = s[q].row;
            }
            a.row_of[i] = row;
            a.key_copy[i] = key[q];
        }
    }
    __syncthreads();
    gather_bags(T, a, a.row_of, b_lo, b_hi);
}

// ---- a plan of the local pull turned into one of the general push ---------------------------------------------------
// After a pull that left early there is no plan: its arrays are of an earlier call, perhaps of the general kernel's.
__global__ void __launch_bounds__(256) plan_entries_kernel(const LocalArgs a, const GeneralPlan g, unsigned* n_entries) {
    if (a.plan_ctl->status != 0u) return;
    for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < a.n; i += gridDim.x * 256) {
        const unsigned slot = a.slot_of_id[i];
        if (slot == kNoSlot) continue;
        const unsigned u = atomicAdd(n_entries, 1u);
        a.info[i].x = u;
        g.send_keys[u] = a.table->slots[slot].key;
        g.send_ret[u] = u;
        g.res_slot[u] = slot;
    }
}
__global__ void __launch_bounds__(256) plan_positions_kernel(const LocalArgs a, const GeneralPlan g, unsigned* n_entries) {
    if (a.plan_ctl->status != 0u) return;
    for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < a.n; i += gridDim.x * 256) {
        const unsigned id = a.id_of[i];
        unsigned u, bit = 0;
        if (id == kNoSlot) {   // the index was full: an entry without a row, whose gradient the push drops
            u = atomicAdd(n_entries, 1u);
            g.send_ret[u] = u;
            g.res_slot[u] = kNoSlot;
        } else {
            u = a.info[id].x;
            if (a.push_row[i] == kDupRow) bit = kDupBit;
        }
        g.inverse[i] = (int)(u | bit);   // the same word as push_row[i]
    }
}
__global__ void plan_finish_kernel(const LocalArgs a, const GeneralPlan g, unsigned* n_entries) {
    if (a.plan_ctl->status != 0u) return;
    const unsigned par = a.plan_ctl->epoch & 1u, n = *n_entries;
    *n_entries = 0;
    a.counters[par * 16] = n;
    a.counters[par * 16 + 4] = n;
    g.in_cnt[par * kMaxWorld] = n;
}

template <int kThreads, bool kFull>
const void* push_kernel_of(int opt, bool sync) {
    if (sync) return (const void*)local_push_kernel<kThreads, -1, true, false>;
    switch (opt) {
        case OPT_SGD: return (const void*)local_push_kernel<kThreads, OPT_SGD, false, kFull>;
        case OPT_ADAGRAD: return (const void*)local_push_kernel<kThreads, OPT_ADAGRAD, false, kFull>;
        case OPT_FTRL: return (const void*)local_push_kernel<kThreads, OPT_FTRL, false, kFull>;
        case OPT_ADAM: return (const void*)local_push_kernel<kThreads, OPT_ADAM, false, kFull>;
        default: return (const void*)local_push_kernel<kThreads, -1, false, false>;
    }
}

unsigned ceil_div(unsigned long long a, unsigned long long b) { return (unsigned)((a + b - 1) / b); }

// Positions per block of the keys that occur once (its logarithm): 32, fewer while that leaves warps without a block, but not
// fewer than the warp has lane groups. A wide row is a whole warp's work: 32 of them in a string took 41.2 us at 13312
// distinct keys of dim 256 (most of 4736 warps idle; the general kernel 27.1), 15.4 us like this; dim 128, 26.1 and 14.8.
// More blocks than one per warp cost more than their balance gives (65536 keys of dim 64, two: 19.4 to 23.0 us).
unsigned once_shift(unsigned n, unsigned dim, unsigned warps) {
    const unsigned groups = 32u / lanes_for_dim(dim);
    unsigned sh = 5;
    while ((1u << sh) > groups && n >> sh < warps) --sh;
    return sh;
}

}  // namespace

unsigned local_hot_rows(unsigned n) { return n / kMinItem + 1; }
unsigned local_big_items(unsigned n) { return 2 * (n / kMinBig) + 1; }   // a big key has at least one whole item

int local_prepare(int* pull_blocks_small, int* pull_blocks_wide, int num_sms) {
    int per_sm = 0;
    cudaError_t e = cudaFuncSetAttribute(local_pull_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Tile<256>::kSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(local_pull_kernel<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Tile<1024>::kSmem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, local_pull_kernel<256>, 256, Tile<256>::kSmem);
    *pull_blocks_small = per_sm * num_sms;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, local_pull_kernel<1024>, 1024, Tile<1024>::kSmem);
    *pull_blocks_wide = per_sm * num_sms;
    return (int)e;
}

int launch_local_pull(const LocalArgs& args, int max_blocks, bool wide, void* stream) {
    LocalArgs a = args;
    const Cut cut = cut_of(a.n);
    a.item_len = cut.item_len;
    a.big_min = cut.big_min;
    a.big_len = cut.big_len;
    void* params[] = {(void*)&a};
    // A small batch gets fewer CTAs, 64 keys each: fewer arrivals at the barriers, and still a row gather per lane group.
    const unsigned want = ceil_div(a.n, wide ? 256 : 64);
    const unsigned grid = want < 1 ? 1 : (want < (unsigned)max_blocks ? want : (unsigned)max_blocks);
    const void* k = wide ? (const void*)local_pull_kernel<1024> : (const void*)local_pull_kernel<256>;
    return (int)cudaLaunchCooperativeKernel(k, dim3(grid), dim3(wide ? 1024 : 256), params, wide ? Tile<1024>::kSmem : Tile<256>::kSmem, (cudaStream_t)stream);
}

int launch_local_push(const LocalArgs& args, int max_blocks, bool wide, bool sync, unsigned table_slots, void* stream) {
    LocalArgs a = args;
    void* params[] = {(void*)&a};
    const int opt = (unsigned)opt_num_slots(a.opt.type) == table_slots ? a.opt.type : -1;
    const unsigned threads = wide ? 1024 : 256;
    const unsigned want = ceil_div((unsigned long long)a.n * lanes_for_dim(a.dim), threads);
    const unsigned grid = want < 1 ? 1 : (want < (unsigned)max_blocks ? want : (unsigned)max_blocks);
    a.once_shift = once_shift(a.n, a.dim, grid * (threads / 32));
    const void* k = a.once_shift == 5 ? (wide ? push_kernel_of<1024, true>(opt, sync) : push_kernel_of<256, true>(opt, sync))
                                      : (wide ? push_kernel_of<1024, false>(opt, sync) : push_kernel_of<256, false>(opt, sync));
    return (int)cudaLaunchKernel(k, dim3(grid), dim3(threads), params, 0, (cudaStream_t)stream);
}

int launch_local_lookup(const LocalArgs& a, int max_blocks, bool wide, void* stream) {
    // A lane group per bag, but no CTA with more keys than it probes at a time while there are bags to hand to others: 64 bags
    // of 16384 keys of dim 16 stood on one CTA (6446 us; 3221 through the general kernel, whose dedup has every SM).
    const unsigned threads = wide ? 1024 : 256, bags = a.n / a.bag_size, by_keys = ceil_div(a.n, threads * 4);
    const unsigned by_bags = ceil_div((unsigned long long)bags * lanes_for_dim(a.dim), threads), most = by_keys < bags ? by_keys : bags;
    const unsigned want = by_bags > most ? by_bags : most;
    const unsigned grid = want < 1 ? 1 : (want < (unsigned)max_blocks ? want : (unsigned)max_blocks);
    if (wide) local_lookup_kernel<1024><<<grid, 1024, 0, (cudaStream_t)stream>>>(a);
    else local_lookup_kernel<256><<<grid, 256, 0, (cudaStream_t)stream>>>(a);
    return (int)cudaGetLastError();
}

int launch_plan_to_general(const LocalArgs& a, const GeneralPlan& g, int num_sms, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned want = ceil_div(a.n, 256), cap = (unsigned)num_sms * 8, grid = want < 1 ? 1 : (want < cap ? want : cap);
    unsigned* n_entries = a.hot_cnt;   // a word that is zero between calls
    plan_entries_kernel<<<grid, 256, 0, s>>>(a, g, n_entries);
    plan_positions_kernel<<<grid, 256, 0, s>>>(a, g, n_entries);
    plan_finish_kernel<<<1, 1, 0, s>>>(a, g, n_entries);
    return (int)cudaGetLastError();
}

}  // namespace psb
