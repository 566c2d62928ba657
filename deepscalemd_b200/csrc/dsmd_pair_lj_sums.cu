// Force kernels: Lennard-Jones with energy sums.
#include "dsmd_pair.cuh"

template cudaError_t dsmd::launch_pair<0, true>(const PairParams&, const ForceArgs&, bool, unsigned, cudaStream_t);
