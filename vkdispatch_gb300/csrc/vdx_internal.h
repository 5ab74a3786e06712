// Internal launch interface between the C ABI (vdx_api.cu) and the kernel
// translation units.  Each launcher picks the template instantiation for a
// (storage, compute, direction, layout) combination and enqueues it.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "fft_kernels.cuh"

struct vdx_fft_desc;  // include/vdx.h

namespace vdx {

enum Store { ST_C64 = 0, ST_C32 = 1, ST_C128 = 2, ST_BF16 = 3 };

struct Launch {
  dim3 grid;
  dim3 block;
  size_t smem;
  cudaStream_t stream;
};

// Elements per thread of the instantiated kernels: registers hold MAXE
// complex values of the current pass, and every radix used by a plan must be
// <= MAXE.  fp32 compute keeps 16 (32 registers of data under the 64-register
// cap of 1024-thread CTAs); fp64 compute keeps 8.
template <class Re>
struct MaxE;
template <>
struct MaxE<float> {
  static constexpr int value = 16;
};
template <>
struct MaxE<double> {
  static constexpr int value = 8;
};

// Runtime-radix plan of a (storage, compute) pair: rows step linearly through
// their shared-memory slots in fp32, where the planner puts an odd radix first
// or the list is 16s and one last radix.  fp64 lists (radix 8) and the
// convolutions of 16-bit storage, whose powers of two have no compile-time
// plan and run their lists in both orders, compute every padded slot.
template <class S, class Re>
using DynPlanOf = DynPlan<MaxE<Re>::value, !Same<Re, float>::value>;
template <class S, class Re>
using DynConvPlanOf = DynPlan<MaxE<Re>::value, !Same<S, Cx<float>>::value>;

// Supported (storage, compute) pairs: complex64/fp32, complex32/fp32,
// bf16x2/fp32, complex128/fp64.
enum Op { OP_C2C_FWD, OP_C2C_INV, OP_CONV, OP_R2C_EVEN, OP_C2R_EVEN, OP_R2C_ODD, OP_C2R_ODD, OP_CONV2D_REAL, OP_BLUESTEIN };

template <class S, class Re>
cudaError_t launch_fft(const FftArgs& a, const Launch& l, int op, bool strided, int kop, int variant);
template <class S, class Re>
cudaError_t launch_dyn_c2c(const FftArgs& a, const Launch& l, int op, bool strided, int variant);
template <class S, class Re>
cudaError_t launch_dyn_conv(const FftArgs& a, const Launch& l, bool strided, int kop, int variant);
template <class S, class Re>
cudaError_t launch_dyn_real(const FftArgs& a, const Launch& l, int op);

cudaError_t launch_twiddle(void* tab, int count, int den, bool f64, cudaStream_t s);
// Four-step twiddles laid out like the intermediate: tab[k1 * N0 + b0] =
// W_{N1 N0}^{b0 k1}, so that a tile's lanes (neighbouring b0) read neighbouring
// entries; in a natural table W_N^i every lane's entry b0 k1 lies on a sector
// of its own.
cudaError_t launch_cross_twiddle(void* tab, int N1, int N0, cudaStream_t s);
cudaError_t launch_stage_twiddle(void* tab, const PassPlan& pp, bool f64, cudaStream_t s);

// One pass of a four-step long-axis transform (fft_large.cu): tiles of M
// adjacent columns, one pp.n-point transform per column.  Batch b of the
// launch starts at (b / split) * bs1 + (b % split) * bs2 elements; point pos
// of column c is at c + pos * ps on input, and at c * out_cs + pos * out_ps
// on output.  Grid = batches * col_tiles, block = pp.T * pp.M.
struct FsArgs {
  PassPlan pp;
  const void* in;
  void* out;
  const void* tw;   // stage-ordered twiddles of the short transform (tensor-core passes: W_n^k)
  const void* twl;  // pass A: cross twiddles W_N^{b0 k1} at b0 * tw_b + k1 * tw_p (tensor-core passes: W_N^k)
  int tw_b, tw_p;
  long long split;
  long long in_bs1, in_bs2, out_bs1, out_bs2;
  long long in_ps, out_ps, out_cs;
  int ncols, col_tiles;
  int tw_from_batch;  // pass A: b0 is b % split (strided axes) or the column (contiguous axes)
  float scale;
  long long nbatch;   // batches of this launch (grid = nbatch * col_tiles)
};
// mode 0: plain store; 1: twiddle, unit-stride columns; 2: twiddle, transposed store (out_ps == 1).
// Whether a short length runs on a compile-time plan, whose transposed stores
// read the cross twiddles along k1, and the exchange pitch of those stores.
inline bool fourstep_fixed(const PassPlan& pp) {
  return (pp.n == 128 && pp.T == 8) || (pp.n == 256 && pp.T == 16) || (pp.n == 64 && pp.T == 4);
}
int fourstep_pitch(const PassPlan& pp);
// Whether every CTA of a launch runs at once at 128 registers a thread (512
// threads an SM).  Such a launch waits for instructions and loads, not for
// issue slots: its runtime plans take a kernel of twice the registers, without
// spills, whose middle and last passes share their code (one 8575-point row
// 20.1 us for both passes with 64 registers, 17.1 with 128; 1 x 16807 x 4 18.3
// and 14.8, 1 x 28561 x 4 17.1 and 13.0).  Launches of more CTAs lose their
// second CTA per SM by it (1 x 240240 x 4: 22.4 and 27.0).
inline bool fourstep_few(const Launch& l, int sms) {
  const int per_sm = 512 / (((int)l.block.x + 31) / 32 * 32);
  return (long long)l.grid.x <= (long long)per_sm * sms;
}
cudaError_t launch_fourstep_pass(const FsArgs& a, const Launch& l, int store, bool inv, int mode, bool few);
// The same pass with the 128-point short transforms on the tensor cores
// (fft_tc.cu); a.pp.n must be 128 and a.pp.M 16 or 32.  bmat = the DFT
// operand image from tc_dft_operands; *status is set to 1 if an MMA
// completion wait gives up.
cudaError_t launch_fourstep_pass_tc(const FsArgs& a, const Launch& l, int store, bool inv, int mode,
                                    const void* bmat, int* status);
cudaError_t tc_dft_operands(int dev, bool inv, const void** out);
size_t tc_pass_smem(int mt);

// Both passes of a four-step long axis in one persistent launch with an
// L2-resident ring for the intermediate (fft_fused4.cu).  Square splits
// (N0 == N1, the same compile-time short plan for both passes) only.
struct FusedLaunch {
  PassPlan ppA, ppB;  // short-transform plans; M = columns per tile, equal for both
  const void* in;
  void* out;
  void* ring;  // R slots: N * M elements each (strided axes) or N (contiguous)
  const void* twA;
  const void* twB;
  const void* twl;
  long long N, N0, N1, inner, outer;
  int M;
  float scale;
  int L, R;
  unsigned* ticket;
  int* doneA;  // R counters each
  int* doneB;
  int* status;
  long long wait_limit;  // 0 = default
  int store;
  bool inverse, strided;
  unsigned grid;
  size_t smem;
};
cudaError_t fused_fourstep_ctas_per_sm(int store, const PassPlan& pp, size_t smem, int* per_sm);
cudaError_t launch_fused_fourstep(const FusedLaunch& fl, cudaStream_t s);

// One-launch 2-D convolution of real images (fft_conv2d.cu): one image per
// thread-block cluster, the half spectrum held in the cluster's shared memory.
struct Conv2dArgs {
  Cx<float>* data;          // (images, H, W/2 + 1) packed RFFT rows, in place
  const Cx<float>* ker;     // kernel spectrum, (images or 1, H, W/2 + 1)
  long long ker_bs;         // elements between images' kernel spectra (0 = broadcast)
  const Cx<float>* tw_row;  // stage-ordered twiddles of the W/2-point rows
  const Cx<float>* tw2;     // W_W^k, k <= W/2
  const Cx<float>* tw_col;  // and of the H-point columns, in both pass orders
  const Cx<float>* tw_colr;
  float col_scale, row_scale;
};
// Bluestein transforms (bluestein.cu): chirp tables w (N) and b (M), the
// conj(FFT(b)) kernel slab replicated over `inner` columns, and the
// chirp-in (zero-padded, to the (outer, M, inner) workspace) / chirp-out
// (cropped, scaled) element-wise launches.
cudaError_t launch_chirp_tables(void* w, void* b, int N, int M, int sign, bool f64, cudaStream_t s);
cudaError_t launch_conj_slab(void* K, const void* B, int M, long long inner, bool f64, cudaStream_t s);
cudaError_t launch_bluestein_mul(void* ws, const void* K, long long outer, int M, long long inner, cudaStream_t s);
cudaError_t launch_bluestein_io(bool in_phase, int store, const void* x, void* ws, const void* w, long long outer,
                                int N, int M, long long inner, float scale, cudaStream_t s);

bool conv2d_real_supported(int H, int W);
cudaError_t conv2d_real_max_clusters(int H, int W, int* count);
cudaError_t launch_conv2d_real(const Conv2dArgs& a, int H, int W, long long images, int kop, cudaStream_t s);

// complex64 kernels specialised at compile time for power-of-two n in
// [16, 16384] (radix-16 passes, n/16 threads per transform)
template <int N>
cudaError_t launch_fixed_c64(const FftArgs& a, const Launch& l, int op, bool strided, int kop, int variant);
bool has_fixed_c64(int n);
cudaError_t launch_fixed_c64_any(int n, const FftArgs& a, const Launch& l, int op, bool strided, int kop,
                                 int variant);
// C2C kernels of 16-bit storage on the same plans, n in [16, 4096]: their
// bytes are half of complex64's, so they are bound by instructions, which the
// runtime-radix kernels spend on addresses (32768 x 1024 bf16 points: 95.1 us
// on the runtime passes, 67.8 us here; 256^3 fp16 along axis 0: 43.3 and 36.3)
bool has_fixed_half(int n);
cudaError_t launch_fixed_half(int store, int n, const FftArgs& a, const Launch& l, int op, bool strided);
cudaError_t launch_fixed_c32_small(int n, const FftArgs& a, const Launch& l, int op, bool strided);
cudaError_t launch_fixed_c32_large(int n, const FftArgs& a, const Launch& l, int op, bool strided);
cudaError_t launch_fixed_bf16_small(int n, const FftArgs& a, const Launch& l, int op, bool strided);
cudaError_t launch_fixed_bf16_large(int n, const FftArgs& a, const Launch& l, int op, bool strided);
// complex64 kernels on the alternative compile-time plans: pts = 32 (two
// passes: radix 32 x 16 for n = 512, 32 x 32 for n = 1024; n/32 threads per
// transform) for every operation, and pts = 8 (radix-8 passes, n/8 threads)
// for strided convolutions of n = 512
template <int N>
cudaError_t launch_fixedpts_conv_c64(int pts, const FftArgs& a, const Launch& l, int kop, int variant);
template <int N>
cudaError_t launch_fixed32_c64(const FftArgs& a, const Launch& l, int op, bool strided, int kop, int variant);
bool has_fixedpts_c64(int n, int pts, bool conv, bool strided);

// fused multi-kernel convolution on the runtime-plan kernels (ST_C64 or
// ST_C128 storage); conv_multi_points = the kernel's points per thread
cudaError_t launch_conv_multi(int store, bool strided, const FftArgs& a, const Launch& l, int kop, int K,
                              long long kstride, long long ostride);
int conv_multi_points(bool f64);
// the same on the compile-time complex64 plans (n = 16 .. 512 and 1024 ..
// 16384 in two translation units)
// pts = 16 (Pow2Plan) or 32 (the two-pass plans of 512 and 1024 points)
cudaError_t launch_fixed_conv_multi_small(int n, int pts, bool strided, const FftArgs& a, const Launch& l, int kop,
                                          int K, long long kstride, long long ostride);
cudaError_t launch_fixed_conv_multi_large(int n, int pts, bool strided, const FftArgs& a, const Launch& l, int kop,
                                          int K, long long kstride, long long ostride);
cudaError_t launch_fixedpts_c64_any(int n, int pts, const FftArgs& a, const Launch& l, int op, bool strided, int kop,
                                    int variant);

// Opt a kernel into more than 48 KB of dynamic shared memory once.
template <class K>
inline cudaError_t prepare_smem(K kernel, size_t smem) {
  if (smem <= 48 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

template <class K, class... Args>
inline cudaError_t enqueue(K kernel, const Launch& l, Args... args) {
  cudaError_t e = prepare_smem(kernel, l.smem);
  if (e != cudaSuccess) return e;
  kernel<<<l.grid, l.block, l.smem, l.stream>>>(args...);
  return cudaGetLastError();
}

// Programmatic dependent launch for the kernels that open with pdl_enter()
// (fft_kernels.cuh): on unless VDX_PDL=0.
bool pdl_enabled();

template <class... KArgs, class... Args>
inline cudaError_t enqueue_pdl(void (*kernel)(KArgs...), const Launch& l, Args... args) {
  if (!pdl_enabled()) return enqueue(kernel, l, args...);
  cudaError_t e = prepare_smem(kernel, l.smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = l.grid;
  cfg.blockDim = l.block;
  cfg.dynamicSmemBytes = l.smem;
  cfg.stream = l.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Geometry of a single-CTA-per-transform plan (no four-step, no Bluestein)
// for the run-time compiled map kernels of jit.cu: the planner's pass plan,
// launch shape and twiddle table for the descriptor's axis.
struct MapGeometry {
  FftArgs args;
  Launch launch;
  std::vector<int> radices;
  bool strided;
  bool f64;
  int N;
  int dev;
};
int map_plan_geometry(const ::vdx_fft_desc& d, MapGeometry* g);

// error reporting and argument checks shared by the C entry points
int set_error(int code, const char* msg);
int check_reduce_args(int op, int map, int in_type, const void* in, long long n, long long batch, const void* out);
int reduce_out_bytes(int in_type);

// reductions
cudaError_t launch_reduce(int op, int map, int in_type, const void* in, long long n, long long batch, void* out,
                          void* partials, int nparts, cudaStream_t s);

}  // namespace vdx
