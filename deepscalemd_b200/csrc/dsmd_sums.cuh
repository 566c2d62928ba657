// Largest displacement and sums over the blocks of a grid, reported to the host by the block that finishes last, or by a launch behind it.
#pragma once

#include "dsmd_force.cuh"

namespace {

using dsmd::DisplacementReport;
using dsmd::Mail;
using dsmd::post;

// The status word with the largest squared displacement goes to the host and becomes the gate of the launches behind.
__device__ __forceinline__ void post_displacement(const DisplacementReport& r) {   // one thread
    const double out[2] = {__longlong_as_double(static_cast<long long>(__ldcg(&r.st->max_disp2))), static_cast<double>(__ldcg(&r.st->out_of_domain))};
    r.st->gate = out[1] != 0.0 ? __longlong_as_double(0x7FF0000000000000ll) : out[0];
    post(r.mail, out, 2, r.seq);
}

// The block's largest squared displacement goes into the status word. With a ticket the last block of the grid reports the word.
// Without one (large grids, or nobody to report to) nothing waits for anything: every warp adds its own, if it is larger than what it reads
// there, and a launch behind this one reports the word (k_post_displacement), if there is to be a report.
__device__ __forceinline__ void report_displacement(double v, const DisplacementReport& r) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (!r.ticket) {
        const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(v));
        if (lane == 0 && v > 0.0 && bits > __ldcg(&r.st->max_disp2)) atomicMax(&r.st->max_disp2, bits);
        return;
    }
    __shared__ double warp_max[32];
    if (lane == 0) warp_max[w] = v;
    __syncthreads();
    if (w == 0) {
        v = lane < (blockDim.x >> 5) ? warp_max[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
        if (lane == 0) {
            if (v > 0.0) atomicMax(&r.st->max_disp2, static_cast<unsigned long long>(__double_as_longlong(v)));
            __threadfence();
            if (atomicAdd(r.ticket, 1u) == gridDim.x - 1) {
                __threadfence();
                *r.ticket = 0u;
                post_displacement(r);
            }
        }
    }
}

// Deterministic sums over a grid: every block leaves its partial sums, and the block that finishes last adds them up in a
// fixed order (one launch instead of two). `ticket` counts finished blocks and is left at zero.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double (&sh)[32][NV]) {   // thread 0 has the sums
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k)
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    if (lane == 0)
        for (int k = 0; k < NV; ++k) sh[w][k] = v[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        const int nw = blockDim.x >> 5;
        for (int k = 0; k < NV; ++k) {
            v[k] = 0.0;
            for (int q = 0; q < nw; ++q) v[k] += sh[q][k];
        }
    }
}

template <int NV>
__device__ __forceinline__ void sum_over_grid(double (&v)[NV], double* partials, unsigned* ticket, double* out, bool accumulate,
                                              Mail* mail = nullptr, unsigned long long seq = 0) {
    __shared__ double sh[32][NV];
    __shared__ bool last;
    block_sum<NV>(v, sh);
    if (threadIdx.x == 0) {
        for (int k = 0; k < NV; ++k) partials[static_cast<size_t>(blockIdx.x) * NV + k] = v[k];
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int k = 0; k < NV; ++k) v[k] = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x)
        for (int k = 0; k < NV; ++k) v[k] += __ldcg(&partials[static_cast<size_t>(b) * NV + k]);
    block_sum<NV>(v, sh);
    if (threadIdx.x == 0) {
        for (int k = 0; k < NV; ++k) out[k] = v[k] = accumulate ? out[k] + v[k] : v[k];
        *ticket = 0u;
        if (mail) post(mail, v, NV, seq);
    }
}

}  // namespace
