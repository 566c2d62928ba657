// Force kernels: Lennard-Jones, forces alone; and the step of the MD loop.
#include "dsmd_pair.cuh"

template cudaError_t dsmd::launch_pair<0, false>(const PairParams&, const ForceArgs&, bool, unsigned, cudaStream_t);

cudaError_t dsmd::launch_step(const PairParams& p, const ForceArgs& a, const Grid& g, const StepArgs& at, const DisplacementReport& report,
                              bool sw, unsigned blocks, cudaStream_t s) {
    const auto launch = [&](auto types) {
        constexpr int TYPES = decltype(types)::value;
        const size_t smem = PairTables<0, false, TYPES, false>::bytes(p.ntypes, 0);
        const auto kernel = sw ? k_step<TYPES, true> : k_step<TYPES, false>;
        kernel<<<blocks, kPairThreads<0, TYPES>, smem, s>>>(p, a, g, at, report);
        return cudaGetLastError();
    };
    if (p.ntypes == 1) return launch(std::integral_constant<int, kOneType>());
    if (p.ntypes <= kFewTypesMost) return launch(std::integral_constant<int, kFewTypes>());
    return launch(std::integral_constant<int, kManyTypes>());
}
