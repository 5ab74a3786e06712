// Kernel of one four-step pass (see fft_large.cu) and its launch by storage
// type; the storage types are separate translation units, so they compile in
// parallel.
#pragma once

#include <cuda.h>

#include "fft_kernels.cuh"
#include "tc_ptx.cuh"
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

// source: point pos of this thread's column at p + pos * ps (global memory, or
// a TMA-staged tile in shared memory)
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
template <class S>
struct FsTileIn {
  const S* p;
  int ps;
  template <int R>
  __device__ __forceinline__ void load(Cx<float>* v, int j, int nb) const {
    const S* q = p + j * ps;
    const int step = nb * ps;
#pragma unroll
    for (int r = 0; r < R; ++r, q += step) v[r] = Conv<S, float>::ld(q);
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
// TMA tile copies: dims (columns, then the other axes by increasing stride),
// coordinates in that order; the box is M columns x n rows.
struct TmaTile {
  int rank;
  int row_dim, br_dim, bq_dim;  // position of each in the map (-1: not a dimension)
};
constexpr long long kTmaWait = 1ll << 24;  // polls before a tile-load wait gives up

template <int RANK>
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, const int* c, uint64_t* bar) {
  const uint64_t m = reinterpret_cast<uint64_t>(map);
  const uint32_t b = tc::smem_u32(bar);
  if constexpr (RANK == 2) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(m), "r"(c[0]), "r"(c[1]), "r"(b)
        : "memory");
  } else if constexpr (RANK == 3) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            dst),
        "l"(m), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(b)
        : "memory");
  } else {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(dst),
        "l"(m), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(b)
        : "memory");
  }
}

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

// TMA > 0: the input tile arrives by one bulk-tensor copy of rank TMA into
// shared memory behind the exchange area, and the first pass gathers from it.
template <class Plan, bool INV, class S, int MODE, int TMA>
__global__ void __launch_bounds__(512, 2) k_fs(const __grid_constant__ CUtensorMap tmap, FsArgs a, TmaTile tt) {
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
  if constexpr (TMA > 0) {
    // staging after the exchange area ((n + 1) * M complex slots), on the
    // 128-byte boundary a tensor copy's destination needs
    const uint32_t stg_addr = (tc::smem_u32(sm + (n + 1) * M) + 127u) & ~127u;
    const S* stg = reinterpret_cast<const S*>(reinterpret_cast<const unsigned char*>(sm) +
                                              (stg_addr - tc::smem_u32(sm)));
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
      tc::mbar_init(&bar, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const uint32_t bytes = uint32_t(n) * uint32_t(M) * uint32_t(sizeof(S));
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_u32(&bar)), "r"(bytes)
                   : "memory");
      int c[4] = {0, 0, 0, 0};
      c[0] = tile * M;
      if (tt.br_dim >= 0) c[tt.br_dim] = (int)br;
      if (tt.bq_dim >= 0) c[tt.bq_dim] = (int)bq;
      tma_load<TMA>(stg_addr, &tmap, c, &bar);
    }
    if (!__syncthreads_and(tc::mbar_wait(&bar, 0, kTmaWait))) {
      if (threadIdx.x == 0 && a.status) atomicExch(a.status, 1);
      tc::mbar_wait(&bar, 0, kTmaWait);  // the copy is still in flight: let it land before leaving
      return;
    }
    fs_transform<INV, S, MODE>(P, pl, a, FsTileIn<S>{stg + pl.m, M}, out, twl, col, valid, sm);
  } else {
    fs_transform<INV, S, MODE>(
        P, pl, a, FsIn<S>{reinterpret_cast<const S*>(a.in) + bq * a.in_bs1 + br * a.in_bs2 + col, a.in_ps, valid}, out,
        twl, col, valid, sm);
  }
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

template <class Plan, class S, int TMA>
cudaError_t launch_mode(const CUtensorMap& m, const FsArgs& a, const TmaTile& tt, const Launch& l, bool inv,
                        int mode) {
  switch (mode * 2 + (inv ? 1 : 0)) {
    case 0: return enqueue(k_fs<Plan, false, S, 0, TMA>, l, m, a, tt);
    case 1: return enqueue(k_fs<Plan, true, S, 0, TMA>, l, m, a, tt);
    case 2: return enqueue(k_fs<Plan, false, S, 1, TMA>, l, m, a, tt);
    case 3: return enqueue(k_fs<Plan, true, S, 1, TMA>, l, m, a, tt);
    case 4: return enqueue(k_fs<Plan, false, S, 2, TMA>, l, m, a, tt);
    default: return enqueue(k_fs<Plan, true, S, 2, TMA>, l, m, a, tt);
  }
}

template <class S, int TMA>
cudaError_t launch_store(const CUtensorMap& m, const FsArgs& a, const TmaTile& tt, const Launch& l, bool inv,
                         int mode) {
  const int n = a.pp.n, T = a.pp.T;
  if constexpr (TMA > 0) {  // staged passes exist for the 128-point short transforms only
    if (n == 128 && T == 8) return launch_mode<FixPlan<128, 8, RList<16, 8>>, S, TMA>(m, a, tt, l, inv, mode);
    return cudaErrorInvalidValue;
  } else {
    if (n == 128 && T == 8) return launch_mode<FixPlan<128, 8, RList<16, 8>>, S, 0>(m, a, tt, l, inv, mode);
    if (n == 256 && T == 16) return launch_mode<FixPlan<256, 16, RList<16, 16>>, S, 0>(m, a, tt, l, inv, mode);
    if (n == 64 && T == 4) return launch_mode<FixPlan<64, 4, RList<16, 4>>, S, 0>(m, a, tt, l, inv, mode);
    return launch_mode<DynPlan<16, false>, S, 0>(m, a, tt, l, inv, mode);
  }
}

template <class S>
cudaError_t launch_any(const CUtensorMap& m, const FsArgs& a, const TmaTile& tt, const Launch& l, bool inv,
                       int mode) {
  if constexpr (sizeof(S) == 4) {
    switch (tt.rank) {
      case 2: return launch_store<S, 2>(m, a, tt, l, inv, mode);
      case 3: return launch_store<S, 3>(m, a, tt, l, inv, mode);
      case 4: return launch_store<S, 4>(m, a, tt, l, inv, mode);
      default: break;
    }
  }
  return launch_store<S, 0>(m, a, tt, l, inv, mode);
}

// the instantiations of one storage type (fft_large_c64.cu, _c32.cu, _bf16.cu)
cudaError_t launch_fs_c64(const CUtensorMap& m, const FsArgs& a, const TmaTile& tt, const Launch& l, bool inv, int mode);
cudaError_t launch_fs_c32(const CUtensorMap& m, const FsArgs& a, const TmaTile& tt, const Launch& l, bool inv, int mode);
cudaError_t launch_fs_bf16(const CUtensorMap& m, const FsArgs& a, const TmaTile& tt, const Launch& l, bool inv, int mode);

}  // namespace vdx
