// Runtime-plan Bluestein kernels for storage Cx<double> with double butterflies.
#include "fft_launch.cuh"

namespace vdx {
template <>
cudaError_t launch_dyn_bluestein<Cx<double>, double>(const FftArgs& a, const Launch& l, bool strided) {
  return launch_bluestein<DynConvPlanOf<Cx<double>, double>, Cx<double>, double>(a, l, strided);
}
}  // namespace vdx
