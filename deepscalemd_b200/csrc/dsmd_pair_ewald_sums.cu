// Force kernels: Ewald with short rows and energy sums.
#include "dsmd_pair.cuh"

template cudaError_t dsmd::launch_pair<1, true, 0>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
