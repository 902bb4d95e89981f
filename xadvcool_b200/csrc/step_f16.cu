// Fused step kernels with __half populations in both lattices (see step_kernels.cuh).
#include "step_kernels.cuh"

namespace xac {
template void launch_staged_step<__half, __half>(const StepLaunch&);
template void launch_row_step<__half, __half>(const StepLaunch&);
template void launch_split_fluid<__half>(const SplitArgs&, int, bool, cudaStream_t);
template void launch_split_thermal<__half>(const SplitArgs&, int, bool, cudaStream_t);
}  // namespace xac
