// Four-step pass kernels for storage bf16c.
#include "fft_large.cuh"

namespace vdx {
cudaError_t launch_fs_bf16(const FsArgs& a, const Launch& l, bool inv, int mode) {
  return launch_any<bf16c>(a, l, inv, mode);
}
}  // namespace vdx
