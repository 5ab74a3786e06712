// Four-step pass kernels for storage bf16c.
#include "fft_large.cuh"

namespace vdx {
cudaError_t launch_fs_bf16(const CUtensorMap& m, const FsArgs& a, const TmaTile& tt, const Launch& l, bool inv,
                        int mode) {
  return launch_any<bf16c>(m, a, tt, l, inv, mode);
}
}  // namespace vdx
