// Fused step kernels with float population storage in both lattices (see step_kernels.cuh).
#include "step_kernels.cuh"

namespace xac {
template void launch_staged_step<float, float>(const StepLaunch&);
template void launch_row_step<float, float>(const StepLaunch&);
template void launch_split_fluid<float>(const SplitArgs&, int, bool, cudaStream_t);
template void launch_split_thermal<float>(const SplitArgs&, int, bool, cudaStream_t);
}  // namespace xac
