// Force kernels: Lennard-Jones with long rows and energy sums.
#include "dsmd_pair.cuh"

template cudaError_t dsmd::launch_pair<0, true, kLongOrder>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
