// C2C kernels for storage bf16c on the compile-time plans of 16 to 256 points.
#include "fft_launch.cuh"

namespace vdx {
cudaError_t launch_fixed_bf16_small(int n, const FftArgs& a, const Launch& l, int op, bool strided) {
  switch (n) {
    case 16: return launch_c2c_any<Pow2Plan<16>, bf16c, float>(a, l, op, strided, 0);
    case 32: return launch_c2c_any<Pow2Plan<32>, bf16c, float>(a, l, op, strided, 0);
    case 64: return launch_c2c_any<Pow2Plan<64>, bf16c, float>(a, l, op, strided, 0);
    case 128: return launch_c2c_any<Pow2Plan<128>, bf16c, float>(a, l, op, strided, 0);
    case 256: return launch_c2c_any<Pow2Plan<256>, bf16c, float>(a, l, op, strided, 0);
    default: return cudaErrorInvalidValue;
  }
}
}  // namespace vdx
