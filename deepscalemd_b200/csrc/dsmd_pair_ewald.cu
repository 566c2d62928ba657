// Force kernels: Ewald with short rows, forces alone.
#include "dsmd_pair.cuh"

template cudaError_t dsmd::launch_pair<1, false, 0>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
