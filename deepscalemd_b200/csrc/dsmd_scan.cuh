// Exclusive sums over the counts of cells, for tables of up to two million of them; without waits between blocks, and launched to
// overlap like the kernels around it.
//
// What bounds it: latency. A block turns kScanItems counts into starts and needs to know what lies before them: of few blocks each
// adds up all counts before its own (they are in the L2), of more each adds up the blocks' sums that a launch before left. The
// library's scan is two launches at any size, neither of which overlaps with its neighbours (rebuild of 864 and of 32,000
// Lennard-Jones atoms: 51 and 61 us with it, 41 and 55 us without it, the launch that cleared the counts and the one for the quads).
// Larger tables do not feel that and stay with it.
#pragma once

#include <cuda_runtime.h>

#include "dsmd_launch.cuh"

namespace dsmd {

constexpr int kScanThreads = 1024, kScanEach = 8, kScanItems = kScanThreads * kScanEach;
constexpr int kScanAlone = 8;              // blocks that work without sums
constexpr int kScanBlocksMost = 256;
constexpr int kScanMost = kScanItems * kScanBlocksMost;

// Counts [first, first + kScanEach) of n, whether or not they lie on 16 bytes.
__device__ __forceinline__ int scan_load(const int* counts, int first, int n, int (&v)[kScanEach]) {
    if (first + kScanEach <= n && (reinterpret_cast<size_t>(counts) & 15) == 0) {
#pragma unroll
        for (int q = 0; q < kScanEach; q += 4) {
            const int4 w = *reinterpret_cast<const int4*>(counts + first + q);
            v[q] = w.x; v[q + 1] = w.y; v[q + 2] = w.z; v[q + 3] = w.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kScanEach; ++k) v[k] = first + k < n ? counts[first + k] : 0;
    }
    int sum = 0;
#pragma unroll
    for (int k = 0; k < kScanEach; ++k) sum += v[k];
    return sum;
}

// Sum over the block, in every thread.
__device__ __forceinline__ int scan_block_sum(int v) {
    __shared__ int s_sum[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = v;
    __syncthreads();
    v = s_sum[threadIdx.x & 31];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    return v;
}

static __global__ void __launch_bounds__(kScanThreads) k_cell_sums(int n, const int* counts, int* __restrict__ sums) {
    if (!after_previous()) return;
    int v[kScanEach];
    const int all = scan_block_sum(scan_load(counts, blockIdx.x * kScanItems + threadIdx.x * kScanEach, n, v));
    if (threadIdx.x == 0) sums[blockIdx.x] = all;
}

// starts[k] = init + counts[0] + ... + counts[k - 1] for k < n. sums: of the blocks' counts, or null.
static __global__ void __launch_bounds__(kScanThreads) k_cell_starts(int n, int init, const int* counts, const int* sums,
                                                                     int* __restrict__ starts) {
    if (!after_previous()) return;
    __shared__ int s_warp[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, block = blockIdx.x;
    int v[kScanEach], before = 0;
    if (sums) {
        if (static_cast<int>(threadIdx.x) < block) before = sums[threadIdx.x];   // (at most kScanBlocksMost)
    } else {
        for (int b = 0; b < block; ++b) before += scan_load(counts, b * kScanItems + threadIdx.x * kScanEach, n, v);
    }
    if (block > 0) before = scan_block_sum(before);
    const int first = block * kScanItems + threadIdx.x * kScanEach, sum = scan_load(counts, first, n, v);
    int incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    int of_warps = s_warp[lane];   // sums of the warps, then of those before each
    const int mine = of_warps;
    for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, of_warps, o);
        if (lane >= o) of_warps += up;
    }
    int at = init + before + __shfl_sync(0xffffffffu, of_warps - mine, w) + incl - sum;
#pragma unroll
    for (int k = 0; k < kScanEach; ++k) {
        if (first + k < n) starts[first + k] = at;
        at += v[k];
    }
}

// n <= kScanMost. sums: room for kScanBlocksMost. Returns how many kernels it launched, or a negative number after an error.
inline int launch_cell_scan(int n, int init, const int* counts, int* sums, int* starts, cudaStream_t s) {
    const unsigned blocks = static_cast<unsigned>((n + kScanItems - 1) / kScanItems);
    const bool alone = blocks <= static_cast<unsigned>(kScanAlone);
    if (!alone && launch_next(k_cell_sums, blocks, kScanThreads, 0, s, n, counts, sums) != cudaSuccess) return -1;
    const int* const of_blocks = alone ? nullptr : sums;
    if (launch_next(k_cell_starts, blocks, kScanThreads, 0, s, n, init, counts, of_blocks, starts) != cudaSuccess) return -1;
    return alone ? 1 : 2;
}

}  // namespace dsmd
