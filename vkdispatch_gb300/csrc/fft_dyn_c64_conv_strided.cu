// Runtime-plan complex64 convolution kernels, strided axes.
#include "fft_launch.cuh"

namespace vdx {
template <>
cudaError_t launch_dyn_conv_layout<Cx<float>, float, true>(const FftArgs& a, const Launch& l, int kop, int variant) {
  using Plan = DynConvPlanOf<Cx<float>, float>;
  if (kop == 0) return launch_conv_layout<Plan, 0, true, Cx<float>, float>(a, l, variant);
  return launch_conv_layout<Plan, 1, true, Cx<float>, float>(a, l, variant);
}
}  // namespace vdx
