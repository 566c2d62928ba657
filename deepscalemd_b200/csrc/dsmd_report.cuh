// Values that the host waits for leave a kernel through pinned host memory: the block that finishes last writes them and then
// the number of the launch, which the host polls. That saves the copy behind the kernel and the wait for the copy: 3 us
// instead of 9 per value.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace dsmd {

struct Mail {
    double value[7];
    unsigned long long seq;
};

#ifdef __CUDACC__
__device__ __forceinline__ void post(Mail* mail, const double* v, int n, unsigned long long seq) {   // one thread
    volatile Mail* m = mail;
    for (int k = 0; k < n; ++k) m->value[k] = v[k];
    __threadfence_system();
    m->seq = seq;
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

// Waits for report `seq` of a launch in `s`. The loop ends with an error when the stream has run dry (or failed) without it.
inline cudaError_t wait_report(const Mail* mail, unsigned long long seq, cudaStream_t s) {
    const volatile Mail* m = mail;
    for (unsigned spins = 1; m->seq != seq; ++spins) {
        if ((spins & 0x3FFu) != 0) continue;
        cudaError_t q = cudaStreamQuery(s);
        if (q == cudaErrorNotReady) continue;
        // done or failed; the caller may have named another stream than the launch's
        if (q == cudaSuccess) q = cudaDeviceSynchronize();
        if (q != cudaSuccess) return q;
        if (m->seq != seq) return cudaErrorUnknown;
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    return cudaSuccess;
}

}  // namespace dsmd
