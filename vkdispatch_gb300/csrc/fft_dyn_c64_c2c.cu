// Runtime-plan C2C kernels for storage Cx<float> with float butterflies: the
// layouts are two translation units (fft_dyn_c64_c2c_contig.cu and
// fft_dyn_c64_c2c_strided.cu), so they compile in parallel.
#include "fft_launch.cuh"

namespace vdx {
template <>
cudaError_t launch_dyn_c2c<Cx<float>, float>(const FftArgs& a, const Launch& l, int op, bool strided, int variant) {
  if (strided) return launch_dyn_c2c_layout<Cx<float>, float, true>(a, l, op, variant);
  return launch_dyn_c2c_layout<Cx<float>, float, false>(a, l, op, variant);
}
}  // namespace vdx
