// Four-step pass kernels for storage c32s.
#include "fft_large.cuh"

namespace vdx {
cudaError_t launch_fs_c32(const CUtensorMap& m, const FsArgs& a, const TmaTile& tt, const Launch& l, bool inv,
                        int mode) {
  return launch_any<c32s>(m, a, tt, l, inv, mode);
}
}  // namespace vdx
