// See segment_sum.h. The sort is cub::DeviceRadixSort (a stable LSD radix sort that ships with the CUDA toolkit);
// the segmented, ordered sum is the kernel below.
#include "segment_sum.h"

#include <cub/device/device_radix_sort.cuh>

#include "common.cuh"

namespace psb {

namespace {

constexpr int kThreads = 256;

__global__ void iota_kernel(unsigned* p, unsigned n, unsigned* long_cnt) {
    if (blockIdx.x == 0 && threadIdx.x < 2) long_cnt[threadIdx.x] = 0;
    for (unsigned i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) p[i] = i;
}

constexpr unsigned kBlock = 64;   // occurrences per block of the blocked sum

// What the pull left behind. The counters live in the half selected by the parity of the pull's call epoch (device
// memory: a launch replayed from a CUDA graph sees the current one). A pull that left early (a reserved key, a wait that
// ran out) published no epoch: inverse map and counters are then of different calls, and the ids need not have runs. The
// host learns of it at its next check only, so every pass looks at the status words itself, as the push does behind them.
struct PlanWords {
    const unsigned* counters;
    const KernelCtl* pull;
    const KernelCtl* push;
    __device__ __forceinline__ bool cut_short() const { return (pull->status | push->status) != 0u; }
    __device__ __forceinline__ unsigned n_uniq(unsigned n) const { return min(n, counters[(pull->epoch & 1u) * 16]); }
};

__device__ __forceinline__ float4 load_grad(const float* grads, unsigned pos, unsigned bag, unsigned dim, unsigned d, float scale) {
    float4 v = *(const float4*)(grads + (size_t)(pos / bag) * dim + d);
    if (scale != 1.0f) {
        v.x = __fmul_rn(v.x, scale); v.y = __fmul_rn(v.y, scale);
        v.z = __fmul_rn(v.z, scale); v.w = __fmul_rn(v.w, scale);
    }
    return v;
}
__device__ __forceinline__ void add_rn(float4& acc, const float4& v) {
    acc.x = __fadd_rn(acc.x, v.x); acc.y = __fadd_rn(acc.y, v.y);
    acc.z = __fadd_rn(acc.z, v.z); acc.w = __fadd_rn(acc.w, v.w);
}

// Left-to-right sum of the gradient rows of sorted entries [lo, end) for the lane's 4 columns at d. The adds are
// chained, the loads are not: four rows are requested before the first is added.
__device__ __forceinline__ float4 run_sum(const unsigned* __restrict__ sorted_pos, unsigned lo, unsigned end,
                                          const float* __restrict__ grads, unsigned bag, unsigned dim, unsigned d, float scale) {
    float4 acc = load_grad(grads, sorted_pos[lo], bag, dim, d, scale);
    unsigned j = lo + 1;
    for (; j + 4 <= end; j += 4) {
        const unsigned p0 = sorted_pos[j], p1 = sorted_pos[j + 1], p2 = sorted_pos[j + 2], p3 = sorted_pos[j + 3];
        const float4 v0 = load_grad(grads, p0, bag, dim, d, scale), v1 = load_grad(grads, p1, bag, dim, d, scale);
        const float4 v2 = load_grad(grads, p2, bag, dim, d, scale), v3 = load_grad(grads, p3, bag, dim, d, scale);
        add_rn(acc, v0); add_rn(acc, v1); add_rn(acc, v2); add_rn(acc, v3);
    }
    for (; j < end; ++j) add_rn(acc, load_grad(grads, sorted_pos[j], bag, dim, d, scale));
    return acc;
}

// The order of the sum (the definition the tests' oracle restates): the occurrences of a key, in position order, are
// cut into blocks of kBlock; every block is added front to back, then the block sums are added front to back. A key
// with up to kBlock occurrences is thus a plain left-to-right sum. The order depends on the batch alone, not on
// which unique id a key happened to get, and the blocks of a hot key are summed by different lane groups.
//
// Pass 1, one thread per sorted entry: the first entry of a run writes the run's start (every id below n_uniq has a run,
// so the next id's start is its end), and n behind the last.
__global__ void __launch_bounds__(kThreads) run_starts_kernel(const unsigned* __restrict__ sorted_ids, unsigned n, const PlanWords plan,
                                                              unsigned* __restrict__ starts) {
    if (plan.cut_short()) return;
    const unsigned n_uniq = plan.n_uniq(n);
    for (unsigned j = blockIdx.x * kThreads + threadIdx.x; j < n; j += gridDim.x * kThreads) {
        const unsigned id = sorted_ids[j] & 0x7fffffffu;
        if (id < n_uniq && (j == 0 || (sorted_ids[j - 1] & 0x7fffffffu) != id)) starts[id] = j;
        if (j == 0) starts[n_uniq] = n;
    }
}

// Pass 2, one lane group per unique id u: a run of up to kBlock entries is summed here; a longer one gets a row of
// partial sums and a work item per block, on which the whole GPU works in pass 3. One CTA per long run left the hottest
// key's 20 000 occurrences of a 213 Ki batch of dim 128 to eight lane groups, and two binary searches per key (36 dependent
// loads) came before: a step of 763 us, 267 us with these passes. What bounds them now is the latency of short kernels.
__global__ void __launch_bounds__(kThreads) ordered_sum_kernel(const unsigned* __restrict__ starts,
                                                              const unsigned* __restrict__ sorted_pos, unsigned n, const PlanWords plan,
                                                              const float* __restrict__ grads, unsigned bag, unsigned dim,
                                                              float scale, float* __restrict__ agg, unsigned* __restrict__ long_cnt,
                                                              uint4* __restrict__ long_runs, uint4* __restrict__ blocks, unsigned max_blocks) {
    if (plan.cut_short()) return;
    const unsigned lanes = lanes_for_dim(dim);
    const unsigned tid = blockIdx.x * kThreads + threadIdx.x;
    const unsigned group = tid / lanes, ngroups = (gridDim.x * kThreads) / lanes, lane = tid % lanes;
    const unsigned n_uniq = plan.n_uniq(n);
    unsigned nlo = 0, nend = 0;
    if (group < n_uniq) { nlo = starts[group]; nend = starts[group + 1]; }
    for (unsigned u = group; u < n_uniq; u += ngroups) {
        const unsigned lo = nlo, end = nend;
        if (u + ngroups < n_uniq) { nlo = starts[u + ngroups]; nend = starts[u + ngroups + 1]; }
        if (lo >= end || end > n) continue;   // an id without a run: nothing below may leave the arrays for it
        if (end - lo > kBlock) {
            const unsigned nblk = (end - lo + kBlock - 1) / kBlock;
            unsigned base = 0, run = 0;
            if (lane == 0) {
                base = atomicAdd(long_cnt + 1, nblk);   // work items, and rows of the scratch area for their sums
                if (base + nblk <= max_blocks) {
                    run = atomicAdd(long_cnt, 1u);
                    long_runs[run] = make_uint4(u, base, nblk, 0u);
                }
            }
            const unsigned wl = threadIdx.x & 31u, gl0 = wl / lanes * lanes;
            const unsigned gmask = (lanes >= 32u ? 0xffffffffu : ((1u << lanes) - 1u)) << gl0;
            base = __shfl_sync(gmask, base, gl0);
            run = __shfl_sync(gmask, run, gl0);
            if (base + nblk > max_blocks) continue;
            for (unsigned k = lane; k < nblk; k += lanes) blocks[base + k] = make_uint4(lo + k * kBlock, min(end, lo + (k + 1) * kBlock), run, 0u);
            continue;
        }
        for (unsigned d = lane * 4; d < dim; d += lanes * 4)
            *(float4*)(agg + (size_t)u * dim + d) = run_sum(sorted_pos, lo, end, grads, bag, dim, d, scale);
    }
}

// The block sums of a long run, front to back. The adds are chained; sixteen loads at a time are not.
__device__ __forceinline__ float4 fold(const float* part, unsigned n, unsigned dim) {
    constexpr unsigned kIn = 16;
    float4 acc = __ldcg((const float4*)part);
    unsigned k = 1;
    for (; k + kIn <= n; k += kIn) {
        float4 v[kIn];
#pragma unroll
        for (unsigned t = 0; t < kIn; ++t) v[t] = __ldcg((const float4*)(part + (size_t)(k + t) * dim));
#pragma unroll
        for (unsigned t = 0; t < kIn; ++t) add_rn(acc, v[t]);
    }
    for (; k < n; ++k) add_rn(acc, __ldcg((const float4*)(part + (size_t)k * dim)));
    return acc;
}

// Pass 3, one lane group per block of a long run; the group that stores the last block sum of a run folds them. (The folds in a
// launch of their own, and a memset of the two counters, cost a batch of 256 to 8192 keys 3 to 11 % of its step.)
__global__ void __launch_bounds__(kThreads) block_sum_kernel(const unsigned* __restrict__ sorted_pos, unsigned n, const float* __restrict__ grads,
                                                            unsigned bag, unsigned dim, float scale, const unsigned* __restrict__ long_cnt,
                                                            uint4* long_runs, const uint4* __restrict__ blocks, unsigned max_blocks,
                                                            float* partials, float* __restrict__ agg) {
    const unsigned lanes = lanes_for_dim(dim);
    const unsigned tid = blockIdx.x * kThreads + threadIdx.x;
    const unsigned n_blocks = min(long_cnt[1], max_blocks), lane = tid % lanes;
    const unsigned gl0 = (threadIdx.x & 31u) / lanes * lanes, gmask = (lanes >= 32u ? 0xffffffffu : ((1u << lanes) - 1u)) << gl0;
    for (unsigned k = tid / lanes; k < n_blocks; k += (gridDim.x * kThreads) / lanes) {
        const uint4 b = blocks[k];
        if (b.x >= b.y || b.y > n || b.z >= max_blocks / 2) continue;
        for (unsigned d = lane * 4; d < dim; d += lanes * 4)
            *(float4*)(partials + (size_t)k * dim + d) = run_sum(sorted_pos, b.x, b.y, grads, bag, dim, d, scale);
        __threadfence();
        __syncwarp(gmask);
        const uint4 run = __ldcg(long_runs + b.z);   // (its last word changes meanwhile)
        unsigned stored = 0;
        if (lane == 0) stored = atomicAdd(&long_runs[b.z].w, 1u) + 1u;
        if (__shfl_sync(gmask, stored, gl0) != run.z) continue;
        __threadfence();
        for (unsigned d = lane * 4; d < dim; d += lanes * 4)
            *(float4*)(agg + (size_t)run.x * dim + d) = fold(partials + (size_t)run.y * dim + d, run.z, dim);
    }
}

}  // namespace

namespace {
// layout of the temporary storage after the identity permutation and cub's own scratch
struct Scratch {
    size_t counters, starts, runs, blocks, partials, total;
    unsigned max_blocks;
};
Scratch scratch_layout(unsigned max_n, unsigned dim, size_t cub_bytes) {
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    Scratch l;
    size_t o = up((size_t)max_n * sizeof(unsigned)) + up(cub_bytes);
    l.counters = o; o += 256;
    const size_t max_long = (size_t)max_n / kBlock + 1;                 // runs longer than kBlock
    l.starts = o; o += up(((size_t)max_n + 1) * sizeof(unsigned));
    l.runs = o; o += up(max_long * sizeof(uint4));
    l.max_blocks = (unsigned)(2 * max_long + 1);                        // sum of ceil(len / kBlock) over the long runs
    l.blocks = o; o += up(l.max_blocks * sizeof(uint4));
    l.partials = o; o += up(l.max_blocks * (size_t)dim * sizeof(float));
    l.total = o;
    return l;
}
size_t cub_sort_bytes(unsigned max_n) {
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const unsigned*)nullptr, (unsigned*)nullptr, (const unsigned*)nullptr,
                                    (unsigned*)nullptr, (int)max_n);
    return bytes;
}
}  // namespace

size_t ordered_segment_sum_temp_bytes(unsigned max_n, unsigned dim) { return scratch_layout(max_n, dim, cub_sort_bytes(max_n)).total; }

int ordered_segment_sum(const int* inverse, unsigned n, unsigned max_n, const unsigned* counters, const KernelCtl* pull_ctl,
                        const KernelCtl* push_ctl, const float* grads, unsigned bag, unsigned dim, float scale, float* agg,
                        unsigned* sorted_ids, unsigned* sorted_pos, void* temp, size_t temp_bytes, void* stream) {
    if (n == 0) return 0;
    if (n > max_n) return (int)cudaErrorInvalidValue;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t cub_bytes = cub_sort_bytes(max_n);
    const Scratch l = scratch_layout(max_n, dim, cub_bytes);
    if (l.total > temp_bytes) return (int)cudaErrorInvalidValue;
    unsigned* iota = (unsigned*)temp;
    void* cub_temp = (char*)temp + ((size_t)max_n * sizeof(unsigned) + 255) / 256 * 256;
    unsigned* long_cnt = (unsigned*)((char*)temp + l.counters);
    unsigned* starts = (unsigned*)((char*)temp + l.starts);
    uint4* long_runs = (uint4*)((char*)temp + l.runs);
    uint4* blocks = (uint4*)((char*)temp + l.blocks);
    float* partials = (float*)((char*)temp + l.partials);
    const PlanWords plan = {counters, pull_ctl, push_ctl};
    iota_kernel<<<148 * 2, kThreads, 0, s>>>(iota, n, long_cnt);
    int bits = 1;
    while (bits < 31 && (1ull << bits) < (unsigned long long)n) ++bits;   // unique ids are below n; bit 31 is a flag, not part of the id
    size_t cb = cub_bytes;
    const cudaError_t e = cub::DeviceRadixSort::SortPairs(cub_temp, cb, (const unsigned*)inverse, sorted_ids, (const unsigned*)iota, sorted_pos, (int)n, 0,
                                        bits, s);
    if (e != cudaSuccess) return (int)e;
    const unsigned lanes = lanes_for_dim(dim);
    const unsigned long long want = ((unsigned long long)n * lanes + kThreads - 1) / kThreads;
    const unsigned grid = (unsigned)(want < 148 * 16 ? want : 148 * 16);
    const unsigned grid_n = (unsigned)(((unsigned long long)n + kThreads - 1) / kThreads);
    run_starts_kernel<<<grid_n < 148 * 8 ? grid_n : 148 * 8, kThreads, 0, s>>>(sorted_ids, n, plan, starts);
    ordered_sum_kernel<<<grid, kThreads, 0, s>>>(starts, sorted_pos, n, plan, grads, bag, dim, scale, agg, long_cnt, long_runs, blocks, l.max_blocks);
    // at most n / kBlock + (long runs) blocks, and a long run has more than kBlock entries
    const unsigned long long want_blocks = (2ull * n / kBlock * lanes + kThreads - 1) / kThreads + 1;
    block_sum_kernel<<<(unsigned)(want_blocks < 148 * 8 ? want_blocks : 148 * 8), kThreads, 0, s>>>(sorted_pos, n, grads, bag, dim, scale, long_cnt, long_runs, blocks,
                                                                                                             l.max_blocks, partials, agg);
    return (int)cudaGetLastError();
}

}  // namespace psb
