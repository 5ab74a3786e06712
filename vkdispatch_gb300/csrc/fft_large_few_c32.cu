// Four-step pass kernels of launches of few CTAs, for storage c32s.
#include "fft_large.cuh"

namespace vdx {
cudaError_t launch_fs_few_c32(const FsArgs& a, const Launch& l, bool inv, int mode) {
  return launch_few<c32s>(a, l, inv, mode);
}
}  // namespace vdx
