// Fused step kernels with __nv_bfloat16 fluid populations and __half thermal populations (see step_kernels.cuh):
// BF16's 8-bit significand is used for the fluid lattice only.
#include "step_kernels.cuh"

namespace xac {
template void launch_staged_step<__nv_bfloat16, __half>(const StepLaunch&);
template void launch_row_step<__nv_bfloat16, __half>(const StepLaunch&);
template void launch_split_fluid<__nv_bfloat16>(const SplitArgs&, int, bool, cudaStream_t);
}  // namespace xac
