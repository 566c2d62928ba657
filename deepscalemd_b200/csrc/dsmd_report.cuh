// Values that the host waits for leave a kernel through pinned host memory: the block that finishes last writes them (or, for
// displacement checks of large grids, a launch of one thread behind them: report_displacement), each
// half of a value in one 64-bit word with the number of the launch, which the host polls (dsmd_ctx::mail). That saves the
// copy behind the kernel and the wait for the copy; and, as every word says by itself whether it has arrived, the fence
// between values and number (1.4 us each: it waits for the host's memory).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstring>

namespace dsmd {

constexpr int kMailValues = 7;

struct Mail {
    unsigned long long word[2 * kMailValues];   // 32 bits of a value, 32 bits of the launch's number
    unsigned long long pad[2];

    double value(int k) const {   // behind wait_report
        const unsigned long long bits = (word[2 * k] >> 32 << 32) | (word[2 * k + 1] >> 32);
        double v;
        std::memcpy(&v, &bits, sizeof(v));
        return v;
    }
};

#ifdef __CUDACC__
__device__ __forceinline__ void post(Mail* mail, const double* v, int n, unsigned long long seq) {   // one thread
    volatile Mail* m = mail;
    const unsigned long long tag = seq & 0xFFFFFFFFull;
    for (int k = 0; k < n; ++k) {
        const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(v[k]));
        m->word[2 * k] = (bits >> 32 << 32) | tag;
        m->word[2 * k + 1] = (bits << 32) | tag;
    }
}

// True in the block that finishes last. Every thread of every block calls it, after what it has written for the last one.
__device__ __forceinline__ bool last_block(unsigned* ticket) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (last) __threadfence();
    return last;
}
#endif

// Waits for the n values of report `seq` of a launch in `s`. The loop ends with an error when the stream has run dry (or
// failed) without them.
inline cudaError_t wait_report(const Mail* mail, int n, unsigned long long seq, cudaStream_t s) {
    const volatile Mail* m = mail;
    const unsigned tag = static_cast<unsigned>(seq);
    for (int k = 0; k < 2 * n; ++k)
        for (unsigned spins = 1; static_cast<unsigned>(m->word[k]) != tag; ++spins) {
            if ((spins & 0x3FFu) != 0) continue;
            cudaError_t q = cudaStreamQuery(s);
            if (q == cudaErrorNotReady) continue;
            // done or failed; the caller may have named another stream than the launch's
            if (q == cudaSuccess) q = cudaDeviceSynchronize();
            if (q != cudaSuccess) return q;
            if (static_cast<unsigned>(m->word[k]) != tag) return cudaErrorUnknown;
        }
    std::atomic_thread_fence(std::memory_order_acquire);
    return cudaSuccess;
}

}  // namespace dsmd
