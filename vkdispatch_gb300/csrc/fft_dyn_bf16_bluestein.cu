// Runtime-plan Bluestein kernels for storage bf16c with float butterflies.
#include "fft_launch.cuh"

namespace vdx {
template <>
cudaError_t launch_dyn_bluestein<bf16c, float>(const FftArgs& a, const Launch& l, bool strided) {
  return launch_bluestein<DynConvPlanOf<bf16c, float>, bf16c, float>(a, l, strided);
}
}  // namespace vdx
