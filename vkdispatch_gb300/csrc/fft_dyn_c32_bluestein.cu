// Runtime-plan Bluestein kernels for storage c32s with float butterflies.
#include "fft_launch.cuh"

namespace vdx {
template <>
cudaError_t launch_dyn_bluestein<c32s, float>(const FftArgs& a, const Launch& l, bool strided) {
  return launch_bluestein<DynConvPlanOf<c32s, float>, c32s, float>(a, l, strided);
}
}  // namespace vdx
