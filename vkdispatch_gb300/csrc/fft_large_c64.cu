// Four-step pass kernels for storage Cx<float>.
#include "fft_large.cuh"

namespace vdx {
cudaError_t launch_fs_c64(const CUtensorMap& m, const FsArgs& a, const TmaTile& tt, const Launch& l, bool inv,
                        int mode) {
  return launch_any<Cx<float>>(m, a, tt, l, inv, mode);
}
}  // namespace vdx
