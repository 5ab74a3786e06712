// Kernel of one four-step pass (see fft_large.cu) and its launch by storage
// type; the storage types are separate translation units, so they compile in
// parallel.
#pragma once

#include "fft_kernels.cuh"
#include "vdx_internal.h"

namespace vdx {

// thread placement inside a column tile: m = column, t = thread of the column
// (the interface FixPlan::run uses)
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
// then a store in which each column's points land contiguously (out_ps == 1;
// contiguous axes).  Compile-time plans transpose in the exchange they make
// anyway: the first pass runs with neighbouring columns in neighbouring lanes,
// as the loads want, and the last with neighbouring points, as the stores want
// (16384^2 bf16 along rows: 1047 -> 917 us for both passes; 384 x 65536: 145.5
// -> 131.3 us).  Runtime plans transpose through shared memory after the last
// pass.
template <bool INV, class S, int MODE, class Plan, class In>
__device__ __forceinline__ void fs_transform(const Plan& P, const FsPlace& pl, const FsArgs& a, const In& in, S* out,
                                             const Cx<float>* twl, int col, bool valid, Cx<float>* sm) {
  const Cx<float>* tw = reinterpret_cast<const Cx<float>*>(a.tw);
  if constexpr (MODE == 2) {
    // odd row pitch n + 1: the column-major writes spread over the banks
    P.template transform<INV, false, true>(
        pl, sm, tw, in, FsOut<Cx<float>, INV, true>{sm + pl.m * (P.n() + 1), 1, twl, a.tw_p, a.scale, true});
  } else {
    P.template transform<INV, false, false>(
        pl, sm, tw, in, FsOut<S, INV, MODE == 1>{out + col, a.out_ps, twl, a.tw_p, a.scale, valid});
  }
}

// slots between neighbouring points of a transposing exchange: columns in
// lanes on one side and T threads' points on the other without bank conflicts
__host__ __device__ constexpr int fs_pitch(int M, int T) { return T <= 16 ? M + 16 / T : M + 1; }

// MODE 2 of a two-pass compile-time plan
template <bool INV, class S, class Plan, class In>
__device__ __forceinline__ void fs_transpose(const Plan& P, const FsPlace& pl, const FsArgs& a, const In& in, S* out,
                                             int tile, Cx<float>* sm) {
  constexpr int R0 = Plan::kFirst, R1 = Plan::kLast, N = R0 * R1, T = Plan::T(), MAXE = Plan::MAXE;
  static_assert(Plan::n() == N, "two passes");
  const int pitch = fs_pitch(pl.M, T);
  Cx<float> v[MAXE];
  Plan::template each<R0>(pl.t, [&](auto b, int j) {
    in.template load<R0>(&v[b * R0], j, N / R0);
    Dft<R0, INV, float>::run(&v[b * R0]);
    Cx<float>* q = sm + j * R0 * pitch + pl.m;
#pragma unroll
    for (int r = 0; r < R0; ++r, q += pitch) *q = v[b * R0 + r];
  });
  __syncthreads();
  const int t = threadIdx.x % T, m = threadIdx.x / T;
  const int c = tile * pl.M + m;
  if (c >= a.ncols) return;
  const Cx<float>* tw = reinterpret_cast<const Cx<float>*>(a.tw);
  const Cx<float>* w = reinterpret_cast<const Cx<float>*>(a.twl) + c * a.tw_b;
  S* dst = out + c * a.out_cs;
  Plan::template each<R1>(t, [&](auto b, int j) {
    const Cx<float>* q = sm + j * pitch + m;
#pragma unroll
    for (int r = 0; r < R1; ++r, q += R0 * pitch) v[b * R1 + r] = *q;
    twiddled_dft<R1, INV>(&v[b * R1], j, R0, tw);
#pragma unroll
    for (int r = 0; r < R1; ++r) {
      const int pos = j + r * R0;
      const Cx<float> f = ldg(w + pos * a.tw_p);
      Conv<S, float>::st(dst + pos, scale(INV ? cmulc(v[b * R1 + r], f) : cmul(v[b * R1 + r], f), a.scale));
    }
  });
}

// Registers: 64 a thread (two CTAs of 512), or 128 on a merged plan, which the
// launches take whose CTAs all run at once (see fourstep_few).
template <class Plan, bool INV, class S, int MODE>
__global__ void __launch_bounds__(512, Plan::kMerged ? 1 : 2) k_fs(FsArgs a) {
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
  const Cx<Re>* twl = reinterpret_cast<const Cx<Re>*>(a.twl) + b0 * a.tw_b;
  const FsIn<S> in{reinterpret_cast<const S*>(a.in) + bq * a.in_bs1 + br * a.in_bs2 + col, a.in_ps, valid};
  if constexpr (MODE == 2 && IsFixPlan<Plan>::value) {
    fs_transpose<INV, S>(P, pl, a, in, out, tile, sm);
    return;
  } else {
    fs_transform<INV, S, MODE>(P, pl, a, in, out, twl, col, valid, sm);
  }
  if constexpr (MODE == 2 && !IsFixPlan<Plan>::value) {
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
  const int n = a.pp.n, T = a.pp.T;  // the lengths below: fourstep_fixed()
  if (n == 128 && T == 8) return launch_mode<FixPlan<128, 8, RList<16, 8>>, S>(a, l, inv, mode);
  if (n == 256 && T == 16) return launch_mode<FixPlan<256, 16, RList<16, 16>>, S>(a, l, inv, mode);
  if (n == 64 && T == 4) return launch_mode<FixPlan<64, 4, RList<16, 4>>, S>(a, l, inv, mode);
  return launch_mode<DynPlan<16, false>, S>(a, l, inv, mode);
}

template <class S>
cudaError_t launch_few(const FsArgs& a, const Launch& l, bool inv, int mode) {
  return launch_mode<DynPlan<16, false, true>, S>(a, l, inv, mode);
}

// the instantiations of one storage type (fft_large_c64.cu, _c32.cu, _bf16.cu,
// and fft_large_few_*.cu)
cudaError_t launch_fs_c64(const FsArgs& a, const Launch& l, bool inv, int mode);
cudaError_t launch_fs_c32(const FsArgs& a, const Launch& l, bool inv, int mode);
cudaError_t launch_fs_bf16(const FsArgs& a, const Launch& l, bool inv, int mode);
cudaError_t launch_fs_few_c64(const FsArgs& a, const Launch& l, bool inv, int mode);
cudaError_t launch_fs_few_c32(const FsArgs& a, const Launch& l, bool inv, int mode);
cudaError_t launch_fs_few_bf16(const FsArgs& a, const Launch& l, bool inv, int mode);

}  // namespace vdx
