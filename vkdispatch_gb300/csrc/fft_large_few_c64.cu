// Four-step pass kernels of launches of few CTAs, for storage Cx<float>.
#include "fft_large.cuh"

namespace vdx {
cudaError_t launch_fs_few_c64(const FsArgs& a, const Launch& l, bool inv, int mode) {
  return launch_few<Cx<float>>(a, l, inv, mode);
}
}  // namespace vdx
