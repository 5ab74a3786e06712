// Four-step pass kernels of launches of few CTAs, for storage bf16c.
#include "fft_large.cuh"

namespace vdx {
cudaError_t launch_fs_few_bf16(const FsArgs& a, const Launch& l, bool inv, int mode) {
  return launch_few<bf16c>(a, l, inv, mode);
}
}  // namespace vdx
