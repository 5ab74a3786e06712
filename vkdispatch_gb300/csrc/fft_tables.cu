// FP64-built twiddle tables.
#include "vdx_internal.h"

namespace vdx {

cudaError_t launch_twiddle(void* tab, int count, int den, bool f64, cudaStream_t s) {
  const int threads = 256;
  const int blocks = (count + threads - 1) / threads;
  if (f64)
    k_twiddle<double><<<blocks, threads, 0, s>>>(reinterpret_cast<Cx<double>*>(tab), count, den);
  else
    k_twiddle<float><<<blocks, threads, 0, s>>>(reinterpret_cast<Cx<float>*>(tab), count, den);
  return cudaGetLastError();
}

namespace {

// tab[k1 * N0 + b0] = W_{N1 N0}^{b0 k1}
__global__ void k_cross_twiddle(Cx<float>* tab, int N1, int N0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N1 * N0) return;
  const int k1 = i / N0, b0 = i - k1 * N0;
  double s, c;
  sincospi(2.0 * double(b0 * k1) / double(N1 * N0), &s, &c);  // b0 k1 < N1 N0 <= 2^28
  tab[i] = mk<float>(float(c), float(-s));
}

}  // namespace

cudaError_t launch_cross_twiddle(void* tab, int N1, int N0, cudaStream_t s) {
  const int threads = 256;
  k_cross_twiddle<<<(N1 * N0 + threads - 1) / threads, threads, 0, s>>>(reinterpret_cast<Cx<float>*>(tab), N1, N0);
  return cudaGetLastError();
}

cudaError_t launch_stage_twiddle(void* tab, const PassPlan& pp, bool f64, cudaStream_t s) {
  const int threads = 256;
  const int blocks = (pp.n + threads - 1) / threads;
  if (f64)
    k_stage_twiddle<double><<<blocks, threads, 0, s>>>(reinterpret_cast<Cx<double>*>(tab), pp);
  else
    k_stage_twiddle<float><<<blocks, threads, 0, s>>>(reinterpret_cast<Cx<float>*>(tab), pp);
  return cudaGetLastError();
}

}  // namespace vdx
