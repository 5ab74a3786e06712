// Kernel of one four-step pass (see fft_large.cu) and its launch by storage
// type; the storage types are separate translation units, so they compile in
// parallel.
#pragma once

#include "fft_kernels.cuh"
#include "vdx_internal.h"

namespace vdx {

// thread placement inside a column tile: m = column, t = thread of the column
// (the interface run_passes / FixPlan::run use)
struct FsPlace {
  int t, m, M;
  static constexpr bool kLinear = true;
  __device__ __forceinline__ int sidx(const PassPlan&, int i) const { return i * M + m; }
  __device__ __forceinline__ int pitch(const PassPlan&) const { return M; }
  __device__ __forceinline__ int pad(const PassPlan&) const { return 0; }
};

// source: point pos of this thread's column at p + pos * ps
template <class S>
struct FsIn {
  const S* p;
  long long ps;
  bool valid;
  template <int R>
  __device__ __forceinline__ void load(Cx<float>* v, int j, int nb) const {
    const S* q = p + j * ps;
    const long long step = nb * ps;
#pragma unroll
    for (int r = 0; r < R; ++r, q += step) v[r] = valid ? Conv<S, float>::ld(q) : mk<float>(0.f, 0.f);
  }
};
// sink: [times the cross twiddle at w + pos * ld,] times s, to p + pos * ps
template <class S, bool INV, bool TW>
struct FsOut {
  S* p;
  long long ps;
  const Cx<float>* w;
  int ld;
  float s;
  bool valid;
  template <int R>
  __device__ __forceinline__ void store(const Cx<float>* v, int j, int nb) const {
    if (!valid) return;
    S* q = p + j * ps;
    const long long step = nb * ps;
    const Cx<float>* f = w + j * ld;
    const int fstep = nb * ld;
#pragma unroll
    for (int r = 0; r < R; ++r, q += step, f += fstep) {
      Cx<float> y = v[r];
      if constexpr (TW) {
        const Cx<float> t = ldg(f);
        y = INV ? cmulc(y, t) : cmul(y, t);
      }
      Conv<S, float>::st(q, scale(y, s));
    }
  }
};

// MODE 0: plain store (pass B).  MODE 1: four-step twiddle, then a store
// whose columns are unit-stride (strided axes).  MODE 2: four-step twiddle,
// then a transposed store through shared memory so that each column's points
// land contiguously (out_ps == 1; contiguous axes).
template <bool INV, class S, int MODE, class Plan, class In>
__device__ __forceinline__ void fs_transform(const Plan& P, const FsPlace& pl, const FsArgs& a, const In& in, S* out,
                                             const Cx<float>* twl, int col, bool valid, Cx<float>* sm) {
  const Cx<float>* tw = reinterpret_cast<const Cx<float>*>(a.tw);
  if constexpr (MODE == 2) {
    // odd row pitch n + 1: the column-major writes spread over the banks
    P.template transform<INV, false, true>(
        pl, sm, tw, in, FsOut<Cx<float>, INV, true>{sm + pl.m * (P.n() + 1), 1, twl, a.tw_ld, a.scale, true});
  } else {
    P.template transform<INV, false, false>(
        pl, sm, tw, in, FsOut<S, INV, MODE == 1>{out + col, a.out_ps, twl, a.tw_ld, a.scale, valid});
  }
}

template <class Plan, bool INV, class S, int MODE>
__global__ void __launch_bounds__(512, 2) k_fs(FsArgs a) {
  using Re = float;
  const Plan P(a.pp);
  const int M = a.pp.M;
  FsPlace pl;
  pl.M = M;
  pl.m = threadIdx.x % M;
  pl.t = threadIdx.x / M;
  P.assume_t(pl.t);
  const int n = P.n();
  const int tile = blockIdx.x % a.col_tiles;
  const long long b = blockIdx.x / a.col_tiles;
  const long long bq = b / a.split, br = b - bq * a.split;
  const int col = tile * M + pl.m;
  const bool valid = col < a.ncols;
  Cx<Re>* sm = smem_base<Re>();
  S* out = reinterpret_cast<S*>(a.out) + bq * a.out_bs1 + br * a.out_bs2;
  // cross twiddles of column b0 < N0.  Columns past the last one of a partial
  // tile (col >= ncols) take b0 = 0: theirs would lie past the table
  const int b0 = a.tw_from_batch ? (int)br : (valid ? col : 0);
  const Cx<Re>* twl = reinterpret_cast<const Cx<Re>*>(a.twl) + b0;
  fs_transform<INV, S, MODE>(
      P, pl, a, FsIn<S>{reinterpret_cast<const S*>(a.in) + bq * a.in_bs1 + br * a.in_bs2 + col, a.in_ps, valid}, out,
      twl, col, valid, sm);
  if constexpr (MODE == 2) {
    __syncthreads();
    const long long ocs = a.out_cs;
    const int total = n * M, ld = n + 1;
    const unsigned nmag = inv_magic(n);
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
      const int mm = n > 1 ? int(__umulhi(unsigned(idx), nmag)) : idx, pos = idx - mm * n;  // idx < 2^20, n <= 4096
      const int c = tile * M + mm;
      if (c < a.ncols) Conv<S, Re>::st(out + c * ocs + pos, sm[mm * ld + pos]);
    }
  }
}

template <class Plan, class S>
cudaError_t launch_mode(const FsArgs& a, const Launch& l, bool inv, int mode) {
  switch (mode * 2 + (inv ? 1 : 0)) {
    case 0: return enqueue(k_fs<Plan, false, S, 0>, l, a);
    case 1: return enqueue(k_fs<Plan, true, S, 0>, l, a);
    case 2: return enqueue(k_fs<Plan, false, S, 1>, l, a);
    case 3: return enqueue(k_fs<Plan, true, S, 1>, l, a);
    case 4: return enqueue(k_fs<Plan, false, S, 2>, l, a);
    default: return enqueue(k_fs<Plan, true, S, 2>, l, a);
  }
}

template <class S>
cudaError_t launch_any(const FsArgs& a, const Launch& l, bool inv, int mode) {
  const int n = a.pp.n, T = a.pp.T;
  if (n == 128 && T == 8) return launch_mode<FixPlan<128, 8, RList<16, 8>>, S>(a, l, inv, mode);
  if (n == 256 && T == 16) return launch_mode<FixPlan<256, 16, RList<16, 16>>, S>(a, l, inv, mode);
  if (n == 64 && T == 4) return launch_mode<FixPlan<64, 4, RList<16, 4>>, S>(a, l, inv, mode);
  return launch_mode<DynPlan<16, false>, S>(a, l, inv, mode);
}

// the instantiations of one storage type (fft_large_c64.cu, _c32.cu, _bf16.cu)
cudaError_t launch_fs_c64(const FsArgs& a, const Launch& l, bool inv, int mode);
cudaError_t launch_fs_c32(const FsArgs& a, const Launch& l, bool inv, int mode);
cudaError_t launch_fs_bf16(const FsArgs& a, const Launch& l, bool inv, int mode);

}  // namespace vdx
