// Four-step pass kernels for storage c32s.
#include "fft_large.cuh"

namespace vdx {
cudaError_t launch_fs_c32(const FsArgs& a, const Launch& l, bool inv, int mode) {
  return launch_any<c32s>(a, l, inv, mode);
}
}  // namespace vdx
