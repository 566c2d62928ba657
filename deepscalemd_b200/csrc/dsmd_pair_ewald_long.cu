// Force kernels: Ewald with long rows, forces alone.
#include "dsmd_pair.cuh"

template cudaError_t dsmd::launch_pair<dsmd::kEwaldCopiesMost, false, kLongOrder>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
