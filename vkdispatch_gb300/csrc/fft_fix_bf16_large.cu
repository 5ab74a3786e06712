// C2C kernels for storage bf16c on the compile-time plans of 512 to 4096 points.
#include "fft_launch.cuh"

namespace vdx {
cudaError_t launch_fixed_bf16_large(int n, const FftArgs& a, const Launch& l, int op, bool strided) {
  switch (n) {
    case 512: return launch_c2c_any<Pow2Plan<512>, bf16c, float>(a, l, op, strided, 0);
    case 1024: return launch_c2c_any<Pow2Plan<1024>, bf16c, float>(a, l, op, strided, 0);
    case 2048: return launch_c2c_any<Pow2Plan<2048>, bf16c, float>(a, l, op, strided, 0);
    case 4096: return launch_c2c_any<Pow2Plan<4096>, bf16c, float>(a, l, op, strided, 0);
    default: return cudaErrorInvalidValue;
  }
}
}  // namespace vdx
