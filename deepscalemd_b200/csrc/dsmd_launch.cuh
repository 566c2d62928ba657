// Launches that overlap the end of the launch before them in the stream (programmatic dependent launch): the blocks of the next
// kernel are placed, and set up, while the last blocks of this one are still at work, and wait in after_previous() until all
// that came before is done and visible. What it gives: 1.6 us per launch of a chain of short kernels (step of 864
// Lennard-Jones atoms 8.9 -> 7.4 us, of 32,000 16.1 -> 14.4 us).
#pragma once

#include <cuda_runtime.h>

namespace dsmd {

#ifdef __CUDACC__
// Every thread of a kernel launched by launch_next calls it before it touches anything that a launch before it may read or
// write, and returns if it is told false. (It never is: the compiler cannot know that, and so keeps behind it also the loads that it may
// otherwise move, __ldca.) From then on the next launch may place its blocks.
// What the launches before have written is visible behind it to ordinary loads. Not so to loads by the read-only path, for which memory
// has to stay as it is as long as the grid lives, and this one lived already while the launch before wrote. So these kernels
// have no __ldg, and none of their pointers to memory that they only read is __restrict__, from which the compiler would
// conclude the same. (What it costs: nothing; passes of 864, 32,000 and 4,000,000 Lennard-Jones atoms 349, 584 and 9,501 us, by the read-only
// path 348, 583 and 9,502.)
__device__ __forceinline__ bool after_previous() {
    unsigned multiprocessors;
    asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;\n\tmov.u32 %0, %%nsmid;" : "=r"(multiprocessors)::"memory");
    return multiprocessors != 0u;
}

// overlap = false: an ordinary launch (the wait in the kernel is over at once).
template <class... Params, class... Args>
cudaError_t launch_next_if(bool overlap, void (*kernel)(Params...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t s, Args&&... args) {
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(blocks);
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
    config.stream = s;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attribute;
    config.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

template <class... Params, class... Args>
cudaError_t launch_next(void (*kernel)(Params...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t s, Args&&... args) {
    return launch_next_if(true, kernel, blocks, threads, smem, s, static_cast<Params>(args)...);
}
#endif

}  // namespace dsmd
