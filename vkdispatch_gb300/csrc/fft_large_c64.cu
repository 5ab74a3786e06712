// Four-step pass kernels for storage Cx<float>.
#include "fft_large.cuh"

namespace vdx {
cudaError_t launch_fs_c64(const FsArgs& a, const Launch& l, bool inv, int mode) {
  return launch_any<Cx<float>>(a, l, inv, mode);
}
}  // namespace vdx
