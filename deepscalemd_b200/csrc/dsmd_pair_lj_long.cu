// Force kernels: Lennard-Jones with long rows, forces alone; and the step of the MD loop.
#include "dsmd_pair.cuh"

template cudaError_t dsmd::launch_pair<0, false, kLongOrder>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
template cudaError_t dsmd::launch_step<kLongOrder>(const PairParams&, const ForceArgs&, const Grid&, const StepArgs&, const DisplacementReport&, bool, unsigned,
                                                cudaStream_t);
