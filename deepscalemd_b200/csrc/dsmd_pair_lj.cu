// Force kernels: Lennard-Jones with short rows, forces alone; and the step of the MD loop.
#include "dsmd_pair.cuh"

template cudaError_t dsmd::launch_pair<0, false, 0>(const PairParams&, const ForceArgs&, bool, unsigned, bool, cudaStream_t);
template cudaError_t dsmd::launch_step<0>(const PairParams&, const ForceArgs&, const Grid&, const StepArgs&, const DisplacementReport&, bool, unsigned,
                                                cudaStream_t);
