// Runtime-plan C2C kernels for storage Cx<float>, contiguous rows.
#include "fft_launch.cuh"

namespace vdx {
template <>
cudaError_t launch_dyn_c2c_layout<Cx<float>, float, false>(const FftArgs& a, const Launch& l, int op, int variant) {
  using Plan = DynPlanOf<Cx<float>, float>;
  if (op == OP_C2C_FWD) return launch_c2c_layout<Plan, false, false, Cx<float>, float>(a, l, variant);
  return launch_c2c_layout<Plan, true, false, Cx<float>, float>(a, l, variant);
}
}  // namespace vdx
