// Runtime-plan Bluestein kernels for storage Cx<float> with float butterflies.
#include "fft_launch.cuh"

namespace vdx {
template <>
cudaError_t launch_dyn_bluestein<Cx<float>, float>(const FftArgs& a, const Launch& l, bool strided) {
  return launch_bluestein<DynConvPlanOf<Cx<float>, float>, Cx<float>, float>(a, l, strided);
}
}  // namespace vdx
