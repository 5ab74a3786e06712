// Batched 1-D FFT kernels along one axis of a C-order array, viewed as
// (outer, N, inner): contiguous axes (inner == 1) and strided axes
// (inner > 1, "columns").
//
// Algorithm: Stockham autosort with a runtime list of radix passes.  Pass p
// with radix R and Ns = product of the radices before it maps butterfly j to
//   inputs  j + r*(n/R)                     (r = 0..R-1)
//   twiddle W_{Ns*R}^{(j mod Ns) * r}
//   outputs (j - j mod Ns)*R + (j mod Ns) + r*Ns
// The inputs of the first pass and the outputs of the last pass both sit at
// j + r*(n/R), so the first pass loads straight from HBM into registers and
// the last pass stores straight to HBM, both coalesced across threads; only
// the exchanges between passes go through shared memory.  A fused
// convolution runs the inverse with the pass order reversed, so the spectrum
// never leaves registers between the forward and the inverse transform.
//
// The reference decomposes the same transforms into per-stage prime groups
// executed by generated code (vkdispatch/fft/context.py:152-179,
// vkdispatch/fft/stages.py:104-172); this file is an independent design.
#pragma once

#include "vdx_common.cuh"

namespace vdx {

constexpr int kMaxPasses = 12;

struct PassPlan {
  int n;      // complex points per transform
  int npass;  // number of radix passes
  int radix[kMaxPasses];
  int T;     // threads per transform
  int M;     // transforms (rows or columns) per CTA
  int npad;  // shared-memory slots per transform (contiguous layout)
  int pad;   // rows of a runtime plan pad one slot every 16 (see Slots)
  // inv_magic(ns) of each pass, ns = product of the radices run before it, in
  // forward and in reversed pass order (set_pass_tables)
  unsigned nsm[kMaxPasses];
  unsigned nsmr[kMaxPasses];
  int nb[kMaxPasses];  // n / radix[p]: butterflies of the pass
  unsigned tmag, mmag;  // inv_magic(T), inv_magic(M) where a kernel splits thread indices with them
};

// m = ceil(2^32 / d) for d >= 2 (0 for d < 2), the multiplier of mod_inv
__host__ __device__ __forceinline__ unsigned inv_magic(int d) { return d > 1 ? 0xFFFFFFFFu / unsigned(d) + 1u : 0u; }

// Fills the per-pass constants of a pass plan whose n and radix list are set.
inline void set_pass_tables(PassPlan& pp) {
  int ns = 1, nsr = 1;
  for (int q = 0; q < pp.npass; ++q) {
    pp.nsm[q] = inv_magic(ns);
    ns *= pp.radix[q];
    pp.nsmr[q] = inv_magic(nsr);
    pp.nb[q] = pp.n / pp.radix[q];
    nsr *= pp.radix[pp.npass - 1 - q];
  }
  // rows pad where stepping through padded slots stays exact: every radix but
  // the last is 16, so points are 1 apart inside a block of 16 or a multiple of
  // 16 apart
  pp.pad = pp.npass > 1;
  for (int q = 0; q + 1 < pp.npass; ++q)
    if (pp.radix[q] != 16) pp.pad = 0;
  pp.tmag = inv_magic(pp.T);
  pp.mmag = inv_magic(pp.M);
}

struct FftArgs {
  PassPlan pp;
  const void* in;
  void* out;
  const void* ker;        // convolution: kernel spectrum
  // stage-ordered twiddles of the n-point passes (k_stage_twiddle), in the
  // plan's pass order and, for convolutions, in reversed pass order
  const void* tw;
  const void* twr;
  const void* tw2;        // real transforms: W_{2n}^k, k in [0, n]
  long long ntrans;       // contiguous: number of transforms
  long long inner;        // strided: number of columns (axis stride in elements)
  long long outer;        // strided: number of outer batches
  long long in_bs;        // elements between transforms (contiguous) / outer batches (strided)
  long long out_bs;
  long long ker_bs;       // kernel batch stride (0 = one spectrum broadcast to all batches)
  int col_tiles;          // strided: ceil(inner / M)
  int sig_lo, sig_hi;     // input positions outside [lo, hi) read as zero
  double scale;           // applied at the final store
  int nreal;              // real transforms: logical real length N
  // fused element-wise operations (complex64 kernels; see vdx_exec_ops)
  const float* in_weight;  // C2C: input point *= in_weight[element] * in_weight_scale on load
  const float* in_weight_scale_ptr;  // optional device scalar multiplied into in_weight_scale
  float in_weight_scale;
  float spec_scale;        // CONV: spec_out = spec_aux * conj(S) * spec_scale (mode 2)
  void* spec_out;          // CONV: receives the forward spectrum S (mode 1) or the product (mode 2)
  const void* spec_aux;
  const float* loss_weight;  // C2C: per-CTA partial of sum(loss_weight * |out|^2)
  float* loss_partials;
  // BLUESTEIN: chirp w[0 .. chirp_n), the kernel spectrum (n entries, one for
  // all transforms) in `ker`, and the output scale besides the 1/n in `scale`
  const void* chirp;
  int chirp_n;
  double chirp_scale;
};

// ---------------------------------------------------------------------------
// thread placement
// ---------------------------------------------------------------------------
// PAD: rows pad one shared-memory slot every 16, which spreads the stride-R
// scatters of power-of-two radices over the banks.  Unpadded rows (and column
// tiles) have a linear slot layout, one addition per access instead of three
// operations; the planner puts an odd radix first, whose scatter does not
// conflict without padding.
template <bool STRIDED, bool PAD = true>
struct Place {
  static constexpr bool kLinear = STRIDED || !PAD;
  int t, m;
  bool valid;
  bool tile_full;  // every transform slot of this CTA exists (uniform per CTA)
  long long ps;    // point stride in elements
  const FftArgs& a;
  __device__ __forceinline__ Place(const FftArgs& args, int T) : a(args) {
    const int tid = threadIdx.x;
    if (STRIDED) {
      m = tid % a.pp.M;
      t = tid / a.pp.M;
      const long long c = col();
      valid = c < a.inner;
      tile_full = (long long)(blockIdx.x % a.col_tiles + 1) * a.pp.M <= a.inner;
      ps = a.inner;
    } else {
      t = tid % T;
      m = tid / T;
      valid = row() < a.ntrans;
      tile_full = (long long)(blockIdx.x + 1) * a.pp.M <= a.ntrans;
      ps = 1;
    }
  }
  // transform coordinates, recomputed where needed so that 64-bit offsets do
  // not stay live across the passes
  __device__ __forceinline__ long long col() const { return (long long)(blockIdx.x % a.col_tiles) * a.pp.M + m; }
  __device__ __forceinline__ long long row() const { return (long long)blockIdx.x * a.pp.M + m; }
  __device__ __forceinline__ long long off(long long bs) const {
    if (STRIDED) return (long long)(blockIdx.x / a.col_tiles) * bs + col();
    return row() * bs;
  }
  __device__ __forceinline__ long long in0() const { return off(a.in_bs); }
  __device__ __forceinline__ long long out0() const { return off(a.out_bs); }
  __device__ __forceinline__ long long ker0() const { return off(a.ker_bs); }
  // shared-memory slot of point i of this thread's transform
  __device__ __forceinline__ int sidx(const PassPlan& pp, int i) const {
    if (STRIDED) return i * pp.M + m;
    return PAD ? m * pp.npad + i + (i >> 4) : m * pp.npad + i;
  }
  // slots between neighbouring points of a linear layout
  __device__ __forceinline__ int pitch(const PassPlan& pp) const { return STRIDED ? pp.M : 1; }
  __device__ __forceinline__ int pad(const PassPlan& pp) const { return STRIDED ? 0 : pp.pad; }
  // unpadded slot, for exchanges whose accesses are unit-stride in either
  // direction (the mirrored k / n-k accesses of the real transforms)
  __device__ __forceinline__ int sidx_plain(const PassPlan& pp, int i) const {
    if (STRIDED) return i * pp.M + m;
    return m * pp.npad + i;
  }
};

// A placement whose transforms each occupy consecutive threads (t fastest)
// keeps every transform of T | 32 threads inside one warp, with shared-memory
// slots of its own: its exchanges between passes need only warp
// synchronisation.  Strided column tiles spread a transform over warps.
template <class PL>
struct WarpLocal : FalseT {};
template <bool PAD>
struct WarpLocal<Place<false, PAD>> : TrueT {};

__host__ __device__ constexpr bool warp_sized(int T) { return T >= 1 && T <= 32 && 32 % T == 0; }

template <bool WARP>
__device__ __forceinline__ void xsync() {
  if constexpr (WARP) __syncwarp();
  else __syncthreads();
}
// runtime scope; `warp` must be the same for the whole CTA
__device__ __forceinline__ void xsync(bool warp) {
  if (warp) __syncwarp();
  else __syncthreads();
}

template <int V>
using IC = IntConst<int, V>;

// Runtime radix -> compile-time radix.
template <class F>
__device__ __forceinline__ void radix_dispatch(int R, F&& f) {
  switch (R) {
    case 1: f(IC<1>{}); break;
    case 2: f(IC<2>{}); break;
    case 3: f(IC<3>{}); break;
    case 4: f(IC<4>{}); break;
    case 5: f(IC<5>{}); break;
    case 6: f(IC<6>{}); break;
    case 7: f(IC<7>{}); break;
    case 8: f(IC<8>{}); break;
    case 9: f(IC<9>{}); break;
    case 10: f(IC<10>{}); break;
    case 11: f(IC<11>{}); break;
    case 12: f(IC<12>{}); break;
    case 13: f(IC<13>{}); break;
    case 14: f(IC<14>{}); break;
    case 15: f(IC<15>{}); break;
    case 16: f(IC<16>{}); break;
    default: break;
  }
}

// v[b*R + r] <- f(j + r*nb) for the thread's butterflies j = t + b*T < nb
template <int R, int MAXE, class Re, class F>
__device__ __forceinline__ void gather(Cx<Re>* v, int nb, int T, int t, F&& f) {
  constexpr int B = MAXE / R;
#pragma unroll
  for (int b = 0; b < B; ++b) {
    const int j = t + b * T;
    if (j < nb) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[b * R + r] = f(j + r * nb);
    }
  }
}

// f(j + r*nb, v[b*R + r]) : natural-order positions (last pass outputs)
template <int R, int MAXE, class Re, class F>
__device__ __forceinline__ void each_natural(Cx<Re>* v, int nb, int T, int t, F&& f) {
  constexpr int B = MAXE / R;
#pragma unroll
  for (int b = 0; b < B; ++b) {
    const int j = t + b * T;
    if (j < nb) {
#pragma unroll
      for (int r = 0; r < R; ++r) f(j + r * nb, v[b * R + r]);
    }
  }
}

// j mod d for d >= 2 and j * d < 2^32, given m = ceil(2^32 / d): one
// multiply-high and a multiply-subtract instead of an integer division by a
// runtime value (division by invariant integers, Granlund & Montgomery,
// PLDI 1994: with m = (2^32 + e) / d, 0 <= e < d, the floor of j m / 2^32 is
// floor(j / d) while j e < 2^32).  Transform indices stay below 2^15, so
// j * d < 2^30 for every pass of every supported length.
__device__ __forceinline__ int mod_inv(int j, int d, unsigned m) {
  return j - int(__umulhi(unsigned(j), m)) * d;
}

// ns is a compile-time constant, so j % ns folds.
// tw is stage-ordered: entry k + r ns of a pass holds W_{ns R}^{k r}, so the
// lanes of a warp (consecutive j, hence consecutive k) read neighbouring
// entries.  A natural table W_n^i is read at k r n/(ns R) instead, a stride
// that puts every lane on a line of its own: those L1 wavefronts, not HBM,
// bounded the three-pass plans (32768 x 1024 points: 113.6 us from a natural
// table, 78.8 us from a stage-ordered one, which is the copy bandwidth; the
// 2048-point convolutions of 4096 x 1009 Bluestein rows: 123.9 -> 96.8 us
// with their chirp launches).
template <int R, int MAXE, bool INV, class Re>
__device__ __forceinline__ void butterflies(Cx<Re>* v, int nb, int T, int t, int ns, const Cx<Re>* tw) {
  constexpr int B = MAXE / R;
#pragma unroll
  for (int b = 0; b < B; ++b) {
    const int j = t + b * T;
    if (j < nb) {
      if (ns > 1) {
        const int k = j % ns;
#pragma unroll
        for (int r = 1; r < R; ++r) {
          const Cx<Re> w = ldg(&tw[k + r * ns]);
          v[b * R + r] = INV ? cmulc(v[b * R + r], w) : cmul(v[b * R + r], w);
        }
      }
      Dft<R, INV, Re>::run(&v[b * R]);
    }
  }
}

// ---------------------------------------------------------------------------
// sources and sinks of a transform.  Both see whole butterflies: a source
// loads the R inputs, a sink stores the R outputs, of butterfly j, which sit at
// points j + r*nb; the address steps by one precomputed stride, so a strided
// axis costs one 64-bit addition per point rather than a 64-bit product.
// ---------------------------------------------------------------------------
// complex input in global memory (signal-range masked).  CTAs whose slots all
// exist and whose range is the whole axis take the unpredicated path.
template <class S, class Re>
struct GlobalIn {
  const S* p;     // point 0 of the thread's transform
  long long ps;   // elements between points
  int lo, hi;     // points outside [lo, hi) read as zero
  bool full, valid;
  template <class PL>
  __device__ __forceinline__ GlobalIn(const FftArgs& a, const PL& pl, int n)
      : p(reinterpret_cast<const S*>(a.in) + pl.in0()), ps(pl.ps), lo(a.sig_lo), hi(a.sig_hi),
        full(pl.tile_full && a.sig_lo <= 0 && a.sig_hi >= n), valid(pl.valid) {}
  template <int R>
  __device__ __forceinline__ void load(Cx<Re>* v, int j, int nb) const {
    const S* q = p + j * ps;
    const long long step = nb * ps;
    if (full) {
#pragma unroll
      for (int r = 0; r < R; ++r, q += step) v[r] = Conv<S, Re>::ld(q);
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r, q += step) {
        const int pos = j + r * nb;
        v[r] = valid && pos >= lo && pos < hi ? Conv<S, Re>::ld(q) : mk<Re>(Re(0), Re(0));
      }
    }
  }
};

// GlobalIn times in_weight[element] * in_weight_scale
template <class S, class Re>
struct WeightedIn {
  GlobalIn<S, Re> in;
  const float* w;
  Re f;
  bool ok;
  template <class PL>
  __device__ __forceinline__ WeightedIn(const FftArgs& a, const PL& pl, int n)
      : in(a, pl, n), w(a.in_weight + pl.in0()),
        f(Re(a.in_weight_scale) * (a.in_weight_scale_ptr ? Re(__ldg(a.in_weight_scale_ptr)) : Re(1))),
        ok(pl.tile_full || pl.valid) {}
  template <int R>
  __device__ __forceinline__ void load(Cx<Re>* v, int j, int nb) const {
    in.template load<R>(v, j, nb);
    const float* q = w + j * in.ps;
    const long long step = nb * in.ps;
#pragma unroll
    for (int r = 0; r < R; ++r, q += step) v[r] = scale(v[r], ok ? Re(__ldg(q)) * f : Re(0));
  }
};

// natural-order points in shared memory
template <class Re>
struct SharedIn {
  const Cx<Re>* p;
  template <int R>
  __device__ __forceinline__ void load(Cx<Re>* v, int j, int nb) const {
    const Cx<Re>* q = p + j;
#pragma unroll
    for (int r = 0; r < R; ++r, q += nb) v[r] = *q;
  }
};
template <class Re>
struct SharedOut {
  Cx<Re>* p;
  template <int R>
  __device__ __forceinline__ void store(const Cx<Re>* v, int j, int nb) const {
    Cx<Re>* q = p + j;
#pragma unroll
    for (int r = 0; r < R; ++r, q += nb) *q = v[r];
  }
};

// scaled store to global memory (a.out unless `base` is given)
template <class S, class Re>
struct GlobalOut {
  S* p;
  long long ps;
  Re s;
  bool ok;
  template <class PL>
  __device__ __forceinline__ GlobalOut(const FftArgs& a, const PL& pl, S* base = nullptr)
      : p((base ? base : reinterpret_cast<S*>(a.out)) + pl.out0()), ps(pl.ps), s(Re(a.scale)),
        ok(pl.tile_full || pl.valid) {}
  template <int R>
  __device__ __forceinline__ void store(const Cx<Re>* v, int j, int nb) const {
    if (!ok) return;
    S* q = p + j * ps;
    const long long step = nb * ps;
#pragma unroll
    for (int r = 0; r < R; ++r, q += step) Conv<S, Re>::st(q, scale(v[r], s));
  }
};

// GlobalOut plus acc += loss_weight[element] * |output|^2
template <class S, class Re>
struct LossOut {
  GlobalOut<S, Re> out;
  const float* w;
  float* acc;
  template <class PL>
  __device__ __forceinline__ LossOut(const FftArgs& a, const PL& pl, float* sum)
      : out(a, pl), w(a.loss_weight + pl.out0()), acc(sum) {}
  template <int R>
  __device__ __forceinline__ void store(const Cx<Re>* v, int j, int nb) const {
    if (!out.ok) return;
    float lw[R];
    const float* q = w + j * out.ps;
    const long long step = nb * out.ps;
#pragma unroll
    for (int r = 0; r < R; ++r, q += step) lw[r] = __ldg(q);
    out.template store<R>(v, j, nb);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const Cx<Re> y = scale(v[r], out.s);
      *acc += lw[r] * float(y.x * y.x + y.y * y.y);
    }
  }
};

// the spectrum operation of a convolution, applied to the R natural-order
// spectrum points of one butterfly.  KOP 0 multiplies by conj(kernel), 1 by
// kernel; SPEC 1 also writes the forward spectrum to spec_out, SPEC 2 writes
// spec_aux * conj(spectrum) * spec_scale.
template <class S, class K, class Re, int KOP, int SPEC>
struct SpectrumOp {
  const K* ker;
  S* so;
  const S* sa;
  Re ss;
  long long ps;
  bool ok;
  template <class PL>
  __device__ __forceinline__ SpectrumOp(const FftArgs& a, const PL& pl)
      : ker(reinterpret_cast<const K*>(a.ker) + pl.ker0()), so(reinterpret_cast<S*>(a.spec_out) + pl.out0()),
        sa(reinterpret_cast<const S*>(a.spec_aux) + pl.out0()), ss(Re(a.spec_scale)), ps(pl.ps),
        ok(pl.tile_full || pl.valid) {}
  template <int R>
  __device__ __forceinline__ void apply(Cx<Re>* v, int j, int nb) const {
    const long long step = nb * ps;
    if constexpr (SPEC == 1) {
      if (ok) {
        S* q = so + j * ps;
#pragma unroll
        for (int r = 0; r < R; ++r, q += step) Conv<S, Re>::st(q, v[r]);
      }
    }
    if constexpr (SPEC == 2) {
      if (ok) {
        S* q = so + j * ps;
        const S* x = sa + j * ps;
#pragma unroll
        for (int r = 0; r < R; ++r, q += step, x += step)
          Conv<S, Re>::st(q, scale(cmulc(Conv<S, Re>::ld(x), v[r]), ss));
      }
    }
    const K* q = ker + j * ps;
#pragma unroll
    for (int r = 0; r < R; ++r, q += step) {
      const Cx<Re> k = ok ? Conv<K, Re>::ld(q) : mk<Re>(Re(0), Re(0));
      v[r] = KOP == 0 ? cmulc(v[r], k) : cmul(v[r], k);
    }
  }
};

// f(b, j) for the thread's butterflies j = t + b*T < nb of a pass, b a
// compile-time constant (so that the values' register array is never indexed
// by a loop counter)
template <int R, int MAXE, int B = 0, class F>
__device__ __forceinline__ void each_butterfly(int nb, int T, int t, F&& f) {
  if constexpr (B < MAXE / R) {
    const int j = t + B * T;
    if (j < nb) f(IntConst<int, B>{}, j);
    each_butterfly<R, MAXE, B + 1>(nb, T, t, f);
  }
}

// The exchange between two passes: the R values at points i0 + r*di of the
// transform in shared memory.  Placements with a linear slot layout step by
// one stride; the padded row layout computes each slot.
template <int R, class PL, class Re>
__device__ __forceinline__ void xload(Cx<Re>* v, const Cx<Re>* sm, const PassPlan& pp, const PL& pl, int i0, int di) {
  if constexpr (PL::kLinear) {
    const Cx<Re>* q = sm + pl.sidx(pp, i0);
    const int step = di * pl.pitch(pp);
#pragma unroll
    for (int r = 0; r < R; ++r, q += step) v[r] = *q;
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = sm[pl.sidx(pp, i0 + r * di)];
  }
}
template <int R, class PL, class Re>
__device__ __forceinline__ void xstore(const Cx<Re>* v, Cx<Re>* sm, const PassPlan& pp, const PL& pl, int i0, int di) {
  if constexpr (PL::kLinear) {
    Cx<Re>* q = sm + pl.sidx(pp, i0);
    const int step = di * pl.pitch(pp);
#pragma unroll
    for (int r = 0; r < R; ++r, q += step) *q = v[r];
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) sm[pl.sidx(pp, i0 + r * di)] = v[r];
  }
}

// v <- v * W_{ns R}^{k r}, then the radix-R butterfly
template <int R, bool INV, class Re>
__device__ __forceinline__ void twiddled_dft(Cx<Re>* v, int k, int ns, const Cx<Re>* tw) {
  if (ns > 1) {
    const Cx<Re>* q = tw + k + ns;
#pragma unroll
    for (int r = 1; r < R; ++r, q += ns) {
      const Cx<Re> w = ldg(q);
      v[r] = INV ? cmulc(v[r], w) : cmul(v[r], w);
    }
  }
  Dft<R, INV, Re>::run(v);
}

// ---------------------------------------------------------------------------
// runtime passes.  Each pass is a self-contained load -> twiddle -> butterfly
// -> store under one radix dispatch, so its values live in registers only
// inside the dispatched body.  (Keeping them across passes took two dispatches
// per pass, butterflies and the next gather, with both layouts live.)
// ---------------------------------------------------------------------------
// Where a thread's transform lives in the exchange's shared memory: point i at
// sm + i * pitch, padded by one slot every 16 points in rows of power-of-two
// plans.  PADDED computes every slot (any radix list); otherwise the R points
// of a butterfly, i0 + r di, are stepped through, one addition per access
// instead of three operations.
template <class Re, bool PADDED>
struct Slots {
  Cx<Re>* sm;  // slot of point 0
  int pitch;   // slots between neighbouring points
  int pad;     // 1 = padded rows (PassPlan::pad)
  __device__ __forceinline__ Cx<Re>* at(int i) const {
    return sm + (PADDED ? i + (i >> 4) : i * pitch + (i >> 4) * pad);
  }
  template <int R>
  __device__ __forceinline__ void load(Cx<Re>* v, int i0, int di) const {
    if constexpr (PADDED) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = *at(i0 + r * di);
    } else {
      const Cx<Re>* q = at(i0);
      const int step = di * pitch + (di >> 4) * pad;
#pragma unroll
      for (int r = 0; r < R; ++r, q += step) v[r] = *q;
    }
  }
  template <int R>
  __device__ __forceinline__ void store(const Cx<Re>* v, int i0, int di) const {
    if constexpr (PADDED) {
#pragma unroll
      for (int r = 0; r < R; ++r) *at(i0 + r * di) = v[r];
    } else {
      Cx<Re>* q = at(i0);
      const int step = di * pitch + (di >> 4) * pad;
#pragma unroll
      for (int r = 0; r < R; ++r, q += step) *q = v[r];
    }
  }
};

// The values of one pass.  They start as unspecified registers (no
// instruction): left uninitialised, a body inside a loop keeps the values of
// idle butterflies alive from one iteration to the next, for every radix of
// the switch at once, and all of them spill (13 KB of spill stores in a
// kernel of fifteen radices; 1500-point rows ran at 216 us).
template <int N, class Re>
struct Values {
  Cx<Re> v[N];
  __device__ __forceinline__ Values() {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if constexpr (sizeof(Re) == 4) asm("" : "=f"(v[i].x), "=f"(v[i].y));
      else asm("" : "=d"(v[i].x), "=d"(v[i].y));
    }
  }
  __device__ __forceinline__ Cx<Re>* at(int i) { return v + i; }
};

// one pass of a plan: t = the thread's index in its transform, T = threads of
// the transform, nb = butterflies, ns = product of the radices before it,
// nsm = inv_magic(ns)
struct PassAt {
  int t, T, nb, ns;
  unsigned nsm;
  bool warp;  // the exchange stays inside a warp
  __device__ __forceinline__ int k(int j) const { return ns > 1 ? mod_inv(j, ns, nsm) : 0; }
};

// source -> exchange (the plan's first pass, ns = 1).  smin: the source is the
// exchange's own shared memory, so a barrier lies between.
template <int R, int MAXE, bool INV, class Re, bool PADDED, class In>
__device__ __forceinline__ void pass_head(PassAt a, Slots<Re, PADDED> x, const In& in, bool smin) {
  Values<MAXE, Re> w;
  Cx<Re>* v = w.v;
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { in.template load<R>(&v[b * R], j, a.nb); });
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { Dft<R, INV, Re>::run(&v[b * R]); });
  if (smin) xsync(a.warp);
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { x.template store<R>(&v[b * R], j * R, 1); });
  xsync(a.warp);
}

// exchange -> exchange
template <int R, int MAXE, bool INV, class Re, bool PADDED>
__device__ __forceinline__ void pass_mid(PassAt a, Slots<Re, PADDED> x, const Cx<Re>* tw) {
  Values<MAXE, Re> w;
  Cx<Re>* v = w.v;
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { x.template load<R>(&v[b * R], j, a.nb); });
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { twiddled_dft<R, INV>(&v[b * R], a.k(j), a.ns, tw); });
  xsync(a.warp);
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) {
    const int k = a.k(j);
    x.template store<R>(&v[b * R], (j - k) * R + k, a.ns);
  });
  xsync(a.warp);
}

// exchange -> sink (the plan's last pass).  smout: the sink is the exchange's
// own shared memory.
template <int R, int MAXE, bool INV, class Re, bool PADDED, class Out>
__device__ __forceinline__ void pass_tail(PassAt a, Slots<Re, PADDED> x, const Cx<Re>* tw, const Out& out,
                                          bool smout) {
  Values<MAXE, Re> w;
  Cx<Re>* v = w.v;
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { x.template load<R>(&v[b * R], j, a.nb); });
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { twiddled_dft<R, INV>(&v[b * R], a.k(j), a.ns, tw); });
  if (smout) xsync(a.warp);
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { out.template store<R>(&v[b * R], j, a.nb); });
}

// pass_mid or, for the plan's last pass, pass_tail in one body
template <int R, int MAXE, bool INV, class Re, bool PADDED, class Out>
__device__ __forceinline__ void pass_rest(PassAt a, Slots<Re, PADDED> x, const Cx<Re>* tw, const Out& out, bool last,
                                          bool smout) {
  Values<MAXE, Re> w;
  Cx<Re>* v = w.v;
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { x.template load<R>(&v[b * R], j, a.nb); });
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { twiddled_dft<R, INV>(&v[b * R], a.k(j), a.ns, tw); });
  if (last) {
    if (smout) xsync(a.warp);
    each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { out.template store<R>(&v[b * R], j, a.nb); });
  } else {
    xsync(a.warp);
    each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) {
      const int k = a.k(j);
      x.template store<R>(&v[b * R], (j - k) * R + k, a.ns);
    });
    xsync(a.warp);
  }
}

// source -> sink (a plan of one pass: one thread holds a whole transform)
template <int R, int MAXE, bool INV, class Re, class In, class Out>
__device__ __forceinline__ void pass_only(PassAt a, const In& in, const Out& out) {
  Values<MAXE, Re> w;
  Cx<Re>* v = w.v;
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) {
    in.template load<R>(&v[b * R], j, a.nb);
    Dft<R, INV, Re>::run(&v[b * R]);
    out.template store<R>(&v[b * R], j, a.nb);
  });
}

// exchange -> last forward pass, spectrum operation, first inverse pass ->
// exchange: both passes have the same radix and the same points
template <int R, int MAXE, class Re, bool PADDED, class Op>
__device__ __forceinline__ void pass_turn(PassAt a, Slots<Re, PADDED> x, const Cx<Re>* tw, const Op& op) {
  Values<MAXE, Re> w;
  Cx<Re>* v = w.v;
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { x.template load<R>(&v[b * R], j, a.nb); });
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) {
    twiddled_dft<R, false>(&v[b * R], j, a.ns, tw);  // ns = nb in the last pass: k = j
    op.template apply<R>(&v[b * R], j, a.nb);
    Dft<R, true, Re>::run(&v[b * R]);
  });
  xsync(a.warp);
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) { x.template store<R>(&v[b * R], j * R, 1); });
  xsync(a.warp);
}
template <int R, int MAXE, class Re, class In, class Op, class Out>
__device__ __forceinline__ void pass_turn_only(PassAt a, const In& in, const Op& op, const Out& out) {
  Values<MAXE, Re> w;
  Cx<Re>* v = w.v;
  each_butterfly<R, MAXE>(a.nb, a.T, a.t, [&](auto b, int j) {
    in.template load<R>(&v[b * R], j, a.nb);
    Dft<R, false, Re>::run(&v[b * R]);
    op.template apply<R>(&v[b * R], j, a.nb);
    Dft<R, true, Re>::run(&v[b * R]);
    out.template store<R>(&v[b * R], j, a.nb);
  });
}

template <bool REV>
__device__ __forceinline__ PassAt pass_at(const PassPlan& pp, int q, int ns, int t, bool warp) {
  return PassAt{t, pp.T, pp.nb[REV ? pp.npass - 1 - q : q], ns, REV ? pp.nsmr[q] : pp.nsm[q], warp};
}

// passes 1 .. npass-2 (exchange to exchange) of a plan whose pass 0 ran radix
// ns; returns the product of the radices run so far
template <int MAXE, bool INV, bool REV, class Re, bool PADDED>
__device__ __forceinline__ int middle_passes(const PassPlan& pp, int ns, int t, const Slots<Re, PADDED>& x,
                                             const Cx<Re>* tw, bool warp) {
  const int P = pp.npass;
  for (int q = 1; q + 1 < P; ++q) {
    const int R = pp.radix[REV ? P - 1 - q : q];
    radix_dispatch(R, [&](auto rc) {
      pass_mid<decltype(rc)::value, MAXE, INV>(pass_at<REV>(pp, q, ns, t, warp), x, tw);
    });
    ns *= R;
  }
  return ns;
}

// A whole transform of a runtime plan from source `in` to sink `out`.  smin /
// smout: they live in the exchange's shared memory.
template <int MAXE, bool INV, class Re, bool PADDED, class In, class Out>
__device__ __forceinline__ void runtime_transform(const PassPlan& pp, int t, const Slots<Re, PADDED>& x,
                                                  const Cx<Re>* tw, const In& in, const Out& out, bool smin,
                                                  bool smout, bool warp) {
  const int P = pp.npass, R0 = pp.radix[0];
  if (P == 1) {
    radix_dispatch(R0, [&](auto rc) {
      pass_only<decltype(rc)::value, MAXE, INV, Re>(pass_at<false>(pp, 0, 1, t, warp), in, out);
    });
    return;
  }
  radix_dispatch(R0, [&](auto rc) {
    pass_head<decltype(rc)::value, MAXE, INV>(pass_at<false>(pp, 0, 1, t, warp), x, in, smin);
  });
  const int ns = middle_passes<MAXE, INV, false>(pp, R0, t, x, tw, warp);
  radix_dispatch(pp.radix[P - 1], [&](auto rc) {
    pass_tail<decltype(rc)::value, MAXE, INV>(pass_at<false>(pp, P - 1, ns, t, warp), x, tw, out, smout);
  });
}

// The same with one body per radix for the middle and the last pass.
template <int MAXE, bool INV, class Re, bool PADDED, class In, class Out>
__device__ __forceinline__ void merged_transform(const PassPlan& pp, int t, const Slots<Re, PADDED>& x,
                                                 const Cx<Re>* tw, const In& in, const Out& out, bool smin, bool smout,
                                                 bool warp) {
  const int P = pp.npass, R0 = pp.radix[0];
  if (P > 1) {
    radix_dispatch(R0, [&](auto rc) {
      pass_head<decltype(rc)::value, MAXE, INV>(pass_at<false>(pp, 0, 1, t, warp), x, in, smin);
    });
  } else {
    radix_dispatch(R0, [&](auto rc) {
      pass_only<decltype(rc)::value, MAXE, INV, Re>(pass_at<false>(pp, 0, 1, t, warp), in, out);
    });
    return;
  }
  int ns = R0;
  for (int q = 1; q < P; ++q) {
    const int R = pp.radix[q];
    radix_dispatch(R, [&](auto rc) {
      pass_rest<decltype(rc)::value, MAXE, INV>(pass_at<false>(pp, q, ns, t, warp), x, tw, out, q + 1 == P, smout);
    });
    ns *= R;
  }
}

// Forward transform, spectrum operation, inverse transform with the passes
// reversed.
template <int MAXE, class Re, bool PADDED, class In, class Op, class Out>
__device__ __forceinline__ void runtime_convolve(const PassPlan& pp, int t, const Slots<Re, PADDED>& x,
                                                 const Cx<Re>* tw, const Cx<Re>* twr, const In& in, const Op& op,
                                                 const Out& out, bool warp) {
  const int P = pp.npass, R0 = pp.radix[0], RL = pp.radix[P - 1];
  if (P == 1) {
    radix_dispatch(R0, [&](auto rc) {
      pass_turn_only<decltype(rc)::value, MAXE, Re>(pass_at<false>(pp, 0, 1, t, warp), in, op, out);
    });
    return;
  }
  radix_dispatch(R0, [&](auto rc) {
    pass_head<decltype(rc)::value, MAXE, false>(pass_at<false>(pp, 0, 1, t, warp), x, in, false);
  });
  int ns = middle_passes<MAXE, false, false>(pp, R0, t, x, tw, warp);
  radix_dispatch(RL, [&](auto rc) {
    pass_turn<decltype(rc)::value, MAXE>(pass_at<false>(pp, P - 1, ns, t, warp), x, tw, op);
  });
  ns = middle_passes<MAXE, true, true>(pp, RL, t, x, twr, warp);
  radix_dispatch(R0, [&](auto rc) {
    pass_tail<decltype(rc)::value, MAXE, true>(pass_at<true>(pp, P - 1, ns, t, warp), x, twr, out, false);
  });
}

// The inverse transform alone with the passes reversed, from a source in shared
// memory that an earlier transform's exchange may still be read from.
template <int MAXE, class Re, bool PADDED, class In, class Out>
__device__ __forceinline__ void runtime_inverse_reversed(const PassPlan& pp, int t, const Slots<Re, PADDED>& x,
                                                         const Cx<Re>* twr, const In& in, const Out& out, bool warp) {
  const int P = pp.npass, R0 = pp.radix[0], RL = pp.radix[P - 1];
  if (P == 1) {
    radix_dispatch(R0, [&](auto rc) {
      pass_only<decltype(rc)::value, MAXE, true, Re>(pass_at<false>(pp, 0, 1, t, warp), in, out);
    });
    return;
  }
  radix_dispatch(RL, [&](auto rc) {
    pass_head<decltype(rc)::value, MAXE, true>(pass_at<true>(pp, 0, 1, t, warp), x, in, true);
  });
  const int ns = middle_passes<MAXE, true, true>(pp, RL, t, x, twr, warp);
  radix_dispatch(R0, [&](auto rc) {
    pass_tail<decltype(rc)::value, MAXE, true>(pass_at<true>(pp, P - 1, ns, t, warp), x, twr, out, false);
  });
}

// ---------------------------------------------------------------------------
// plan policies: how the kernels below learn n, T and the radix passes.
//   DynPlan   - runtime pass list (any 13-smooth length), radix by switch
//   FixPlan   - compile-time length, threads per transform and radix list;
//               every index, division and twiddle stride folds at compile time
// ---------------------------------------------------------------------------
template <int... Rs>
struct RList {};

template <class L>
struct RFirst;
template <int R0, int... Rs>
struct RFirst<RList<R0, Rs...>> {
  static constexpr int value = R0;
};
template <class L>
struct RLast;
template <int R0>
struct RLast<RList<R0>> {
  static constexpr int value = R0;
};
template <int R0, int R1, int... Rs>
struct RLast<RList<R0, R1, Rs...>> {
  static constexpr int value = RLast<RList<R1, Rs...>>::value;
};
template <class In, class Out = RList<>>
struct RRev;
template <int R0, int... Rs, int... Os>
struct RRev<RList<R0, Rs...>, RList<Os...>> : RRev<RList<Rs...>, RList<R0, Os...>> {};
template <int... Os>
struct RRev<RList<>, RList<Os...>> {
  using type = RList<Os...>;
};

// MERGED: the middle and the last pass of a transform share one body per radix,
// so a list of equal radices runs the same instructions again instead of
// fetching others; the body needs more registers.
template <int MAXE_, bool PAD_ = true, bool MERGED_ = false>
struct DynPlan {
  static constexpr int MAXE = MAXE_;
  static constexpr bool PAD = PAD_;
  static constexpr bool kMerged = MERGED_;
  __device__ __forceinline__ void assume_t(int) const {}
  const PassPlan& pp;
  __device__ __forceinline__ explicit DynPlan(const PassPlan& p) : pp(p) {}
  __device__ __forceinline__ int n() const { return pp.n; }
  __device__ __forceinline__ int T() const { return pp.T; }
  template <class Re, class PL>
  __device__ __forceinline__ Slots<Re, !PL::kLinear> slots(const PL& pl, Cx<Re>* sm) const {
    return Slots<Re, !PL::kLinear>{sm + pl.sidx(pp, 0), pl.pitch(pp), pl.pad(pp)};
  }
  // whole transform from source `in` to sink `out`; SMIN / SMOUT: in the
  // exchange's shared memory
  template <bool INV, bool SMIN, bool SMOUT, class PL, class Re, class In, class Out>
  __device__ __forceinline__ void transform(const PL& pl, Cx<Re>* sm, const Cx<Re>* tw, const In& in,
                                            const Out& out) const {
    const bool warp = WarpLocal<PL>::value && warp_sized(pp.T);
    if constexpr (kMerged) merged_transform<MAXE, INV>(pp, pl.t, slots<Re>(pl, sm), tw, in, out, SMIN, SMOUT, warp);
    else runtime_transform<MAXE, INV>(pp, pl.t, slots<Re>(pl, sm), tw, in, out, SMIN, SMOUT, warp);
  }
  template <class PL, class Re, class In, class Out>
  __device__ __forceinline__ void inverse_reversed(const PL& pl, Cx<Re>* sm, const Cx<Re>* twr, const In& in,
                                                   const Out& out) const {
    runtime_inverse_reversed<MAXE>(pp, pl.t, slots<Re>(pl, sm), twr, in, out,
                                   WarpLocal<PL>::value && warp_sized(pp.T));
  }
  template <class PL, class Re, class In, class Op, class Out>
  __device__ __forceinline__ void convolve(const PL& pl, Cx<Re>* sm, const Cx<Re>* tw, const Cx<Re>* twr,
                                           const In& in, const Op& op, const Out& out) const {
    runtime_convolve<MAXE>(pp, pl.t, slots<Re>(pl, sm), tw, twr, in, op, out,
                           WarpLocal<PL>::value && warp_sized(pp.T));
  }
};

// FRESH: nothing in the exchange's shared memory is still being read, so the
// first scatter needs no barrier before it
template <int N, int T, int MAXE, bool INV, bool FRESH, class Re, class PL, int NS, int R, int... Rest>
__device__ __forceinline__ void chain(Cx<Re>* v, const PassPlan& pp, const PL& pl, Cx<Re>* sm, const Cx<Re>* tw) {
  constexpr bool W = WarpLocal<PL>::value && warp_sized(T);
  butterflies<R, MAXE, INV, Re>(v, N / R, T, pl.t, NS, tw);
  if constexpr (sizeof...(Rest) > 0) {
    if constexpr (!FRESH) xsync<W>();
    each_butterfly<R, MAXE>(N / R, T, pl.t, [&](auto b, int j) {
      const int k = j % NS;
      xstore<R>(&v[b * R], sm, pp, pl, (j - k) * R + k, NS);
    });
    xsync<W>();
    constexpr int R2 = RFirst<RList<Rest...>>::value;
    each_butterfly<R2, MAXE>(N / R2, T, pl.t, [&](auto b, int j) { xload<R2>(&v[b * R2], sm, pp, pl, j, N / R2); });
    chain<N, T, MAXE, INV, false, Re, PL, NS * R, Rest...>(v, pp, pl, sm, tw);
  }
}

template <int N, int T, int MAXE, bool INV, bool FRESH, class Re, class PL, int... Rs>
__device__ __forceinline__ void chain_list(RList<Rs...>, Cx<Re>* v, const PassPlan& pp, const PL& pl, Cx<Re>* sm,
                                           const Cx<Re>* tw) {
  chain<N, T, MAXE, INV, FRESH, Re, PL, 1, Rs...>(v, pp, pl, sm, tw);
}

template <int N_, int T_, class L, int MAXE_ = 16>
struct FixPlan {
  static constexpr int MAXE = MAXE_;
  static constexpr bool PAD = true;
  static constexpr bool kMerged = false;
  static constexpr int kFirst = RFirst<L>::value, kLast = RLast<L>::value;
  // the thread's index inside its transform is below T (lets the compiler
  // drop the j < n/R guards of exact plans)
  __device__ __forceinline__ void assume_t(int t) const { __builtin_assume(t >= 0 && t < T_); }
  const PassPlan& pp;
  __device__ __forceinline__ explicit FixPlan(const PassPlan& p) : pp(p) {}
  __device__ __forceinline__ static constexpr int n() { return N_; }
  __device__ __forceinline__ static constexpr int T() { return T_; }
  // radix of the first executed pass (REV: passes run last-to-first)
  template <bool REV, class F>
  __device__ __forceinline__ void first(F&& f) const {
    f(IC<REV ? RLast<L>::value : RFirst<L>::value>{});
  }
  template <bool REV, class F>
  __device__ __forceinline__ void last(F&& f) const {
    f(IC<REV ? RFirst<L>::value : RLast<L>::value>{});
  }
  // PL: a thread placement (Place<STRIDED> or any type with t and sidx(pp, i))
  template <bool INV, bool REV, bool FRESH = false, class PL, class Re>
  __device__ __forceinline__ void run(Cx<Re>* v, const PL& pl, Cx<Re>* sm, const Cx<Re>* tw) const {
    using Order = typename Cond<REV, typename RRev<L>::type, L>::type;
    chain_list<N_, T_, MAXE, INV, FRESH, Re, PL>(Order{}, v, pp, pl, sm, tw);
  }
  // f(b, j) over the thread's butterflies of radix R
  template <int R, class F>
  __device__ __forceinline__ static void each(int t, F&& f) {
    each_butterfly<R, MAXE>(N_ / R, T_, t, f);
  }
  template <bool INV, bool SMIN, bool SMOUT, class PL, class Re, class In, class Out>
  __device__ __forceinline__ void transform(const PL& pl, Cx<Re>* sm, const Cx<Re>* tw, const In& in,
                                            const Out& out) const {
    Cx<Re> v[MAXE];
    each<kFirst>(pl.t, [&](auto b, int j) { in.template load<kFirst>(&v[b * kFirst], j, N_ / kFirst); });
    run<INV, false, !SMIN>(v, pl, sm, tw);
    if constexpr (SMOUT) xsync<WarpLocal<PL>::value && warp_sized(T_)>();
    each<kLast>(pl.t, [&](auto b, int j) { out.template store<kLast>(&v[b * kLast], j, N_ / kLast); });
  }
  template <class PL, class Re, class In, class Op, class Out>
  __device__ __forceinline__ void convolve(const PL& pl, Cx<Re>* sm, const Cx<Re>* tw, const Cx<Re>* twr,
                                           const In& in, const Op& op, const Out& out) const {
    Cx<Re> v[MAXE];
    each<kFirst>(pl.t, [&](auto b, int j) { in.template load<kFirst>(&v[b * kFirst], j, N_ / kFirst); });
    run<false, false, true>(v, pl, sm, tw);
    each<kLast>(pl.t, [&](auto b, int j) { op.template apply<kLast>(&v[b * kLast], j, N_ / kLast); });
    run<true, true>(v, pl, sm, twr);
    each<kFirst>(pl.t, [&](auto b, int j) { out.template store<kFirst>(&v[b * kFirst], j, N_ / kFirst); });
  }
};

template <class P>
struct IsFixPlan : FalseT {};
template <int N_, int T_, class L, int MAXE_>
struct IsFixPlan<FixPlan<N_, T_, L, MAXE_>> : TrueT {};

// Programmatic dependent launch.  These kernels are launched with
// programmatic stream serialisation (enqueue_pdl): the next kernel of the
// stream may be scheduled while this one's last CTAs still run, and this one
// may have been scheduled before the previous kernel finished.  So every CTA
// first lets its successor launch, then waits until the previous kernel of
// the stream has completed and its writes are visible -- before any global
// memory access.  Launched without the attribute, both are no-ops.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class Re>
__device__ __forceinline__ Cx<Re>* smem_base() {
  extern __shared__ __align__(16) unsigned char vdx_smem_raw[];
  return reinterpret_cast<Cx<Re>*>(vdx_smem_raw);
}

// First-pass gather and last-pass store of kernels that keep a transform's
// values in registers across the passes.
template <class Plan, class S, class Re, bool STRIDED, bool PAD>
__device__ __forceinline__ void gather_input(const Plan& P, const Place<STRIDED, PAD>& pl, const FftArgs& a,
                                             Cx<Re>* v) {
  const GlobalIn<S, Re> in(a, pl, P.n());
  P.template first<false>([&](auto rc) {
    constexpr int RR = decltype(rc)::value;
    const int nb = P.n() / RR;
    each_butterfly<RR, Plan::MAXE>(nb, P.T(), pl.t, [&](auto b, int j) { in.template load<RR>(&v[b * RR], j, nb); });
  });
}

template <class Plan, bool REV, class S, class Re, bool STRIDED, bool PAD>
__device__ __forceinline__ void store_output(const Plan& P, const Place<STRIDED, PAD>& pl, const FftArgs& a, Cx<Re>* v,
                                             S* base = nullptr) {
  const GlobalOut<S, Re> out(a, pl, base);
  P.template last<REV>([&](auto rc) {
    constexpr int RR = decltype(rc)::value;
    const int nb = P.n() / RR;
    each_butterfly<RR, Plan::MAXE>(nb, P.T(), pl.t, [&](auto b, int j) { out.template store<RR>(&v[b * RR], j, nb); });
  });
}

// ---------------------------------------------------------------------------
// complex-to-complex
// ---------------------------------------------------------------------------
// IW: multiply each input point by in_weight[element] * in_weight_scale as it
// is loaded (the 2 w y of a weighted |y|^2 loss's gradient).
// LOSS: write one partial of sum(loss_weight[element] * |output|^2) per CTA.
// Plans of 32 points per thread run CTAs of at most 256 threads with up to
// 128 registers per thread.
template <class Plan, bool INV, bool STRIDED, class S, class Re, int IW = 0, int LOSS = 0>
__global__ void __launch_bounds__(Plan::MAXE >= 32 ? 256 : 1024, Plan::MAXE >= 32 ? 2 : 1) k_c2c(FftArgs a) {
  pdl_enter();
  const Plan P(a.pp);
  const Place<STRIDED, Plan::PAD> pl(a, P.T());
  Cx<Re>* sm = smem_base<Re>();
  const Cx<Re>* tw = reinterpret_cast<const Cx<Re>*>(a.tw);
  P.assume_t(pl.t);
  if constexpr (IW) {
    P.template transform<INV, false, false>(pl, sm, tw, WeightedIn<S, Re>(a, pl, P.n()), GlobalOut<S, Re>(a, pl));
  } else if constexpr (LOSS) {
    float acc = 0.f;
    P.template transform<INV, false, false>(pl, sm, tw, GlobalIn<S, Re>(a, pl, P.n()), LossOut<S, Re>(a, pl, &acc));
    // block sum in a fixed order through shared memory (any CTA size; the
    // plan reserves blockDim floats of dynamic shared memory)
    float* red = reinterpret_cast<float*>(sm);
    const int nt = blockDim.x, tid = threadIdx.x;
    __syncthreads();
    red[tid] = acc;
    __syncthreads();
    int span = 1;
    while (span < nt) span <<= 1;
    for (int h = span >> 1; h > 0; h >>= 1) {
      if (tid < h && tid + h < nt) red[tid] += red[tid + h];
      __syncthreads();
    }
    if (tid == 0) a.loss_partials[blockIdx.x] = red[0];
  } else {
    P.template transform<INV, false, false>(pl, sm, tw, GlobalIn<S, Re>(a, pl, P.n()), GlobalOut<S, Re>(a, pl));
  }
}

// ---------------------------------------------------------------------------
// fused convolution: forward FFT -> spectrum * op(kernel) -> inverse FFT
// kop: 0 = multiply by conj(kernel) (reference default,
// vkdispatch/fft/shader_factories.py:136-145), 1 = multiply by kernel.
// ---------------------------------------------------------------------------
// SPEC 1: also write the forward spectrum S to spec_out (kept for a backward
// pass).  SPEC 2: write spec_aux * conj(S) * spec_scale to spec_out instead
// (the kernel-spectrum gradient X conj(G) / N of an FFT convolution).
template <class Plan, bool STRIDED, class S, class K, class Re, int KOP, int SPEC = 0>
__global__ void __launch_bounds__(Plan::MAXE >= 32 ? 256 : 1024, Plan::MAXE >= 32 ? 2 : 1) k_conv(FftArgs a) {
  pdl_enter();
  const Plan P(a.pp);
  const Place<STRIDED, Plan::PAD> pl(a, P.T());
  Cx<Re>* sm = smem_base<Re>();
  const Cx<Re>* tw = reinterpret_cast<const Cx<Re>*>(a.tw);
  const Cx<Re>* twr = reinterpret_cast<const Cx<Re>*>(a.twr);
  P.assume_t(pl.t);
  P.convolve(pl, sm, tw, twr, GlobalIn<S, Re>(a, pl, P.n()), SpectrumOp<S, K, Re, KOP, SPEC>(a, pl),
             GlobalOut<S, Re>(a, pl));
}

// Fused convolution for CTAs of at most 256 threads, complex64 compile-time
// plans.  The launch bound allows 128 registers per thread (80 for plans of 8
// points per thread).  Plans of up to 16 points per thread load the kernel
// spectrum (and SPEC 2's spec_aux) into registers right after issuing the
// signal loads, so its HBM latency overlaps the forward passes instead of
// following them (rows: 65536 x 256 points 82.2 -> 67.0 us, 16384 x 1024 98.5 ->
// 77.0, 8192 x 2048 112.1 -> 85.3); with 32 points per thread the registers are
// full and it is loaded after the forward FFT.  The kernel spectrum is read
// once, with evict-first loads.
template <class Plan, bool STRIDED, class S, class Re, int KOP, int SPEC = 0>
__global__ void __launch_bounds__(256, Plan::MAXE <= 8 ? 3 : 2) k_conv_pf(FftArgs a) {
  pdl_enter();
  const Plan P(a.pp);
  constexpr int MAXE = Plan::MAXE, RR = Plan::kLast;
  const Place<STRIDED> pl(a, P.T());
  Cx<Re>* sm = smem_base<Re>();
  const Cx<Re>* tw = reinterpret_cast<const Cx<Re>*>(a.tw);
  const Cx<Re>* twr = reinterpret_cast<const Cx<Re>*>(a.twr);
  const S* ker = reinterpret_cast<const S*>(a.ker) + pl.ker0();
  P.assume_t(pl.t);
  const int n = P.n(), nb = n / RR;
  const bool kvalid = pl.tile_full || pl.valid;
  const long long step = nb * pl.ps;
  constexpr bool PF = MAXE <= 16;
  Cx<Re> v[MAXE];
  gather_input<Plan, S, Re>(P, pl, a, v);
  Cx<Re> kr[PF ? MAXE : 1], ar[PF && SPEC == 2 ? MAXE : 1];
  if constexpr (PF) {
    Plan::template each<RR>(pl.t, [&](auto b, int j) {
      const S* q = ker + j * pl.ps;
#pragma unroll
      for (int r = 0; r < RR; ++r, q += step) kr[b * RR + r] = kvalid ? ld_once<S, Re>(q) : mk<Re>(Re(0), Re(0));
    });
    if constexpr (SPEC == 2) {
      Plan::template each<RR>(pl.t, [&](auto b, int j) {
        const S* q = reinterpret_cast<const S*>(a.spec_aux) + pl.out0() + j * pl.ps;
#pragma unroll
        for (int r = 0; r < RR; ++r, q += step) ar[b * RR + r] = kvalid ? ld_once<S, Re>(q) : mk<Re>(Re(0), Re(0));
      });
    }
  }
  P.template run<false, false, true>(v, pl, sm, tw);
  if constexpr (SPEC != 0) {
    Plan::template each<RR>(pl.t, [&](auto b, int j) {
      if (!kvalid) return;
      S* q = reinterpret_cast<S*>(a.spec_out) + pl.out0() + j * pl.ps;
      const S* x = reinterpret_cast<const S*>(a.spec_aux) + pl.out0() + j * pl.ps;
#pragma unroll
      for (int r = 0; r < RR; ++r, q += step, x += step) {
        const Cx<Re> f = v[b * RR + r];
        if constexpr (SPEC == 1) {
          Conv<S, Re>::st(q, f);
        } else {
          Cx<Re> g;
          if constexpr (PF) g = ar[b * RR + r];
          else g = Conv<S, Re>::ld(x);
          Conv<S, Re>::st(q, scale(cmulc(g, f), Re(a.spec_scale)));
        }
      }
    });
  }
  Plan::template each<RR>(pl.t, [&](auto b, int j) {
    const S* q = ker + j * pl.ps;
#pragma unroll
    for (int r = 0; r < RR; ++r, q += step) {
      Cx<Re> k;
      // 32 points: no stepping pointer, since a chain of 32 addresses keeps the
      // loads from going out together (64 x 1024 x 512 along axis 1: 260.8 ->
      // 181.7 us; chains of 16 do as well: 64 x 512 x 257 43.4 and 43.7)
      if constexpr (PF) k = kr[b * RR + r];
      else k = kvalid ? ld_once<S, Re>(RR >= 32 ? ker + (j + r * nb) * pl.ps : q) : mk<Re>(Re(0), Re(0));
      v[b * RR + r] = KOP == 0 ? cmulc(v[b * RR + r], k) : cmul(v[b * RR + r], k);
    }
  });
  P.template run<true, true>(v, pl, sm, twr);
  store_output<Plan, true, S, Re>(P, pl, a, v);
}

// The forward spectrum of a runtime plan's multi-kernel convolution, kept at
// the points of its transform: the thread that stored a point reads it back.
template <class Re>
struct KeepOut {
  Cx<Re>* p;  // point 0 of the thread's transform
  int ps;     // slots between points
  template <int R>
  __device__ __forceinline__ void store(const Cx<Re>* v, int j, int nb) const {
    Cx<Re>* q = p + j * ps;
#pragma unroll
    for (int r = 0; r < R; ++r, q += nb * ps) *q = v[r];
  }
};
// the kept spectrum times (the conjugate of) one kernel
template <class K, class Re, int KOP>
struct KeepIn {
  const Cx<Re>* p;
  int ps;
  const K* ker;
  long long kps;
  bool ok;
  template <int R>
  __device__ __forceinline__ void load(Cx<Re>* v, int j, int nb) const {
    const Cx<Re>* q = p + j * ps;
    const K* kq = ker + j * kps;
    const long long step = nb * kps;
#pragma unroll
    for (int r = 0; r < R; ++r, q += nb * ps, kq += step) {
      const Cx<Re> k = ok ? Conv<K, Re>::ld(kq) : mk<Re>(Re(0), Re(0));
      v[r] = KOP == 0 ? cmulc(*q, k) : cmul(*q, k);
    }
  }
};

// Fused multi-kernel convolution (the reference's kernel_num > 1 shader,
// vkdispatch/fft/shader_factories.py:166-193): the signal is read and
// transformed once, then for each kernel k: * K_k (conjugate or plain
// product) -> inverse FFT -> output slice k.  Kernel k is read at
// a.ker + k * kstride and output slice k written at a.out + k * ostride
// (elements).  The forward spectrum waits in a thread-private region at the
// end of the dynamic shared memory (MAXE slots per thread; a runtime plan keeps
// point i of its transforms there, a compile-time plan value i of its thread),
// so only the exchange region is shared between threads.  Runtime plans run the
// self-contained passes, like every other transform (with values held in
// registers across the passes, 3000 x 360 rows of three kernels took 43.2 us,
// 31.4 here; 3000 x 1000 of four 110.8 and 81.1).
template <class Plan, bool STRIDED, class S, class Re, int KOP>
__global__ void __launch_bounds__(Plan::MAXE >= 32 ? 256 : 1024, Plan::MAXE >= 32 ? 2 : 1)
    k_conv_multi(FftArgs a, int K, long long kstride, long long ostride) {
  pdl_enter();
  const Plan P(a.pp);
  constexpr int MAXE = Plan::MAXE;
  const Place<STRIDED, Plan::PAD> pl(a, P.T());
  Cx<Re>* sm = smem_base<Re>();
  const Cx<Re>* tw = reinterpret_cast<const Cx<Re>*>(a.tw);
  const Cx<Re>* twr = reinterpret_cast<const Cx<Re>*>(a.twr);
  unsigned dyn;
  asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
  Cx<Re>* keep = sm + (dyn / sizeof(Cx<Re>) - unsigned(MAXE) * blockDim.x);
  const bool kvalid = pl.tile_full || pl.valid;
  if constexpr (!IsFixPlan<Plan>::value) {
    const int ps = STRIDED ? a.pp.M : 1;
    Cx<Re>* kp = keep + (STRIDED ? pl.m : pl.m * P.n());
    P.template transform<false, false, false>(pl, sm, tw, GlobalIn<S, Re>(a, pl, P.n()), KeepOut<Re>{kp, ps});
    for (int k = 0; k < K; ++k) {
      const S* ker = reinterpret_cast<const S*>(a.ker) + k * kstride + pl.ker0();
      P.inverse_reversed(pl, sm, twr, KeepIn<S, Re, KOP>{kp, ps, ker, pl.ps, kvalid},
                         GlobalOut<S, Re>(a, pl, reinterpret_cast<S*>(a.out) + k * ostride));
    }
  } else {
    Cx<Re> v[MAXE];
    P.assume_t(pl.t);
    const int n = P.n();
    gather_input<Plan, S, Re>(P, pl, a, v);
    P.template run<false, false>(v, pl, sm, tw);
#pragma unroll
    for (int i = 0; i < MAXE; ++i) keep[i * blockDim.x + threadIdx.x] = v[i];
    for (int k = 0; k < K; ++k) {
      if (k > 0) {
#pragma unroll
        for (int i = 0; i < MAXE; ++i) v[i] = keep[i * blockDim.x + threadIdx.x];
      }
      const S* ker = reinterpret_cast<const S*>(a.ker) + k * kstride + pl.ker0();
      P.template last<false>([&](auto rc) {
        constexpr int RR = decltype(rc)::value;
        constexpr int B = MAXE / RR;
        const int nb = n / RR;
#pragma unroll
        for (int b = 0; b < B; ++b) {
          const int j = pl.t + b * P.T();
          if (j < nb) {
#pragma unroll
            for (int r = 0; r < RR; ++r) {
              const int pos = j + r * nb;
              const Cx<Re> kv = kvalid ? Conv<S, Re>::ld(ker + pos * pl.ps) : mk<Re>(Re(0), Re(0));
              v[b * RR + r] = KOP == 0 ? cmulc(v[b * RR + r], kv) : cmul(v[b * RR + r], kv);
            }
          }
        }
      });
      P.template run<true, true>(v, pl, sm, twr);
      store_output<Plan, true, S, Re>(P, pl, a, v, reinterpret_cast<S*>(a.out) + k * ostride);
    }
  }
}

// ---------------------------------------------------------------------------
// Bluestein transform of chirp_n points as one n-point convolution, n >= 2
// chirp_n - 1 (see bluestein.cu): x w zero-padded -> FFT_n -> * conj(ker) ->
// inverse FFT_n -> times w, cropped.  The padding is never stored: points from
// chirp_n up read as zero in the first pass and are dropped in the last, so
// HBM sees each input and output once.  (As three launches over a padded
// workspace, 4096 rows of 1009 points took 32.8 + 42.7 + 19.8 us.)
// ---------------------------------------------------------------------------
template <class S, class Re>
struct ChirpIn {
  const S* p;
  const Cx<Re>* w;
  long long ps;
  int n;
  bool ok;
  template <int R>
  __device__ __forceinline__ void load(Cx<Re>* v, int j, int nb) const {
    const S* q = p + j * ps;
    const long long step = nb * ps;
#pragma unroll
    for (int r = 0; r < R; ++r, q += step) {
      const int pos = j + r * nb;
      v[r] = ok && pos < n ? cmul(Conv<S, Re>::ld(q), ldg(w + pos)) : mk<Re>(Re(0), Re(0));
    }
  }
};
template <class Re>
struct ChirpOp {
  const Cx<Re>* k;
  template <int R>
  __device__ __forceinline__ void apply(Cx<Re>* v, int j, int nb) const {
    const Cx<Re>* q = k + j;
#pragma unroll
    for (int r = 0; r < R; ++r, q += nb) v[r] = cmulc(v[r], ldg(q));
  }
};
template <class S, class Re>
struct ChirpOut {
  S* p;
  const Cx<Re>* w;
  long long ps;
  int n;
  Re s, sc;
  bool ok;
  template <int R>
  __device__ __forceinline__ void store(const Cx<Re>* v, int j, int nb) const {
    if (!ok) return;
    S* q = p + j * ps;
    const long long step = nb * ps;
#pragma unroll
    for (int r = 0; r < R; ++r, q += step) {
      const int pos = j + r * nb;
      if (pos < n) Conv<S, Re>::st(q, scale(cmul(scale(v[r], s), ldg(w + pos)), sc));
    }
  }
};

template <class Plan, bool STRIDED, class S, class Re>
__global__ void __launch_bounds__(Plan::MAXE >= 32 ? 256 : 1024, Plan::MAXE >= 32 ? 2 : 1) k_bluestein(FftArgs a) {
  pdl_enter();
  const Plan P(a.pp);
  const Place<STRIDED, Plan::PAD> pl(a, P.T());
  Cx<Re>* sm = smem_base<Re>();
  P.assume_t(pl.t);
  const Cx<Re>* w = reinterpret_cast<const Cx<Re>*>(a.chirp);
  const bool ok = pl.tile_full || pl.valid;
  P.convolve(pl, sm, reinterpret_cast<const Cx<Re>*>(a.tw), reinterpret_cast<const Cx<Re>*>(a.twr),
             ChirpIn<S, Re>{reinterpret_cast<const S*>(a.in) + pl.in0(), w, pl.ps, a.chirp_n, ok},
             ChirpOp<Re>{reinterpret_cast<const Cx<Re>*>(a.ker)},
             ChirpOut<S, Re>{reinterpret_cast<S*>(a.out) + pl.out0(), w, pl.ps, a.chirp_n, Re(a.scale),
                             Re(a.chirp_scale), ok});
}

// ---------------------------------------------------------------------------
// real-to-complex, even N = 2n, rows of the packed RFFT layout: row pitch
// n+1 complex elements = 2n+2 reals (vkdispatch/base/buffer.py:377-448).
// z[m] = x[2m] + i x[2m+1] -> Z = FFT_n(z) -> with e = (Z[k] + conj Z[n-k])/2
// and o = (Z[k] - conj Z[n-k])/2i:
//   X[k] = e + W_2n^k o,   X[n-k] = conj(e - W_2n^k o),   k = 0..n/2
// One thread forms both bins of a pair, so a pair costs one twiddle product
// and two shared-memory reads.
// ---------------------------------------------------------------------------
// packed real row as complex points; the signal range counts reals
template <class S, class Re>
struct RealIn {
  const S* p;
  int lo, hi;
  bool full, valid;
  template <class PL>
  __device__ __forceinline__ RealIn(const FftArgs& a, const PL& pl, int n)
      : p(reinterpret_cast<const S*>(a.in) + pl.in0()), lo(a.sig_lo), hi(a.sig_hi),
        full(a.sig_lo <= 0 && a.sig_hi >= 2 * n && pl.tile_full), valid(pl.valid) {}
  template <int R>
  __device__ __forceinline__ void load(Cx<Re>* v, int j, int nb) const {
    using SR = typename RealOf<S>::type;
    if (full) {
      const S* q = p + j;
#pragma unroll
      for (int r = 0; r < R; ++r, q += nb) v[r] = Conv<S, Re>::ld(q);
      return;
    }
    const SR* pr = reinterpret_cast<const SR*>(p);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int e = 2 * (j + r * nb), o = e + 1;
      const Re xr = valid && e >= lo && e < hi ? ld_real<Re>(pr + e) : Re(0);
      const Re xi = valid && o >= lo && o < hi ? ld_real<Re>(pr + o) : Re(0);
      v[r] = mk<Re>(xr, xi);
    }
  }
};

template <class Plan, class S, class Re>
__global__ void __launch_bounds__(Plan::MAXE >= 32 ? 256 : 1024, Plan::MAXE >= 32 ? 2 : 1) k_r2c_even(FftArgs a) {
  pdl_enter();
  const Plan P(a.pp);
  const Place<false, Plan::PAD> pl(a, P.T());
  Cx<Re>* sm = smem_base<Re>();
  const Cx<Re>* tw = reinterpret_cast<const Cx<Re>*>(a.tw);
  const Cx<Re>* tw2 = reinterpret_cast<const Cx<Re>*>(a.tw2);
  P.assume_t(pl.t);
  const int n = P.n();
  Cx<Re>* z = sm + pl.sidx_plain(a.pp, 0);
  P.template transform<false, false, true>(pl, sm, tw, RealIn<S, Re>(a, pl, n), SharedOut<Re>{z});
  xsync(warp_sized(P.T()));  // rows: the exchange stays inside the row's warp
  if (!(pl.tile_full || pl.valid)) return;
  S* out = reinterpret_cast<S*>(a.out) + pl.out0();
  const Re half = Re(0.5);
  // n <= T * MAXE for every plan, so MAXE/2 steps cover every pair
#pragma unroll
  for (int u = 0; u <= Plan::MAXE / 2; ++u) {
    const int k = pl.t + u * P.T();
    if (2 * k > n) break;
    const Cx<Re> zk = z[k], zc = conj(z[k == 0 ? 0 : n - k]);
    const Cx<Re> e = scale(zk + zc, half);
    const Cx<Re> d = scale(zk - zc, half);
    const Cx<Re> wo = cmul(ldg(&tw2[k]), mk<Re>(d.y, -d.x));  // d / i
    Conv<S, Re>::st(out + k, e + wo);
    if (k == 0) Conv<S, Re>::st(out + n, mk<Re>(zk.x - zk.y, Re(0)));
    else if (2 * k != n) Conv<S, Re>::st(out + (n - k), conj(e - wo));
  }
}

// ---------------------------------------------------------------------------
// complex-to-real, even N = 2n (Hermitian half X[0..n] -> N reals).  With
// s = X[k] + conj X[n-k] and w = W_2n^{-k} (X[k] - conj X[n-k]):
//   Z[k] = s + i w,   Z[n-k] = conj(s - i w),   k = 0..n/2,
// with the imaginary parts of X[0] and X[n] dropped (the real part of the
// full-length inverse does not depend on them) -> z = IFFT_n(Z) ->
// x[2m] + i x[2m+1] = z[m]
// ---------------------------------------------------------------------------
template <class Plan, class S, class Re>
__global__ void __launch_bounds__(Plan::MAXE >= 32 ? 256 : 1024, Plan::MAXE >= 32 ? 2 : 1) k_c2r_even(FftArgs a) {
  pdl_enter();
  const Plan P(a.pp);
  const Place<false, Plan::PAD> pl(a, P.T());
  Cx<Re>* sm = smem_base<Re>();
  const Cx<Re>* tw = reinterpret_cast<const Cx<Re>*>(a.tw);
  const Cx<Re>* tw2 = reinterpret_cast<const Cx<Re>*>(a.tw2);
  const S* in = reinterpret_cast<const S*>(a.in) + pl.in0();
  P.assume_t(pl.t);
  const int n = P.n();
  Cx<Re>* z = sm + pl.sidx_plain(a.pp, 0);
  if (pl.tile_full || pl.valid) {
    constexpr int U = Plan::MAXE / 2;  // pairs per thread (n <= T * MAXE), the middle bin apart
    Cx<Re> lo[U], hi[U];
    // every load in flight before the first shared-memory store
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = pl.t + u * P.T();
      if (2 * k < n) {
        lo[u] = Conv<S, Re>::ld(in + k);
        hi[u] = Conv<S, Re>::ld(in + (n - k));
      }
    }
    if (n % 2 == 0 && pl.t == 0) {
      const Cx<Re> x = Conv<S, Re>::ld(in + n / 2);
      z[n / 2] = mk<Re>(x.x + x.x, -(x.y + x.y));  // s = 2 Re x, w = -2 Im x
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = pl.t + u * P.T();
      if (2 * k < n) {
        Cx<Re> xk = lo[u], xc = conj(hi[u]);
        if (k == 0) xk.y = xc.y = Re(0);
        const Cx<Re> s = xk + xc;
        const Cx<Re> w = cmulc(xk - xc, ldg(&tw2[k]));  // * W^{-k}
        z[k] = mk<Re>(s.x - w.y, s.y + w.x);
        if (k != 0) z[n - k] = mk<Re>(s.x + w.y, w.x - s.y);
      }
    }
  }
  xsync(warp_sized(P.T()));  // rows: the exchange stays inside the row's warp
  P.template transform<true, true, false>(pl, sm, tw, SharedIn<Re>{z}, GlobalOut<S, Re>(a, pl));
}

// ---------------------------------------------------------------------------
// real transforms of odd length N: full-length complex FFT of the real row
// (imaginary part zero), keeping bins 0..N/2 (forward), or of the
// Hermitian-extended half spectrum, keeping real parts (inverse) -- the
// reference's own R2C I/O rules (vkdispatch/fft/global_memory_iterators.py:
// 85-92, 214-226).  Row pitch N+1 reals = N/2+1 complex.
// ---------------------------------------------------------------------------
template <bool INV, class S, class Re>
struct OddIn {
  const S* p;
  int n, lo, hi;
  bool valid;
  template <int R>
  __device__ __forceinline__ void load(Cx<Re>* v, int j, int nb) const {
    using SR = typename RealOf<S>::type;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int pos = j + r * nb;
      if (!valid) v[r] = mk<Re>(Re(0), Re(0));
      else if (!INV)
        v[r] = mk<Re>(pos >= lo && pos < hi ? ld_real<Re>(reinterpret_cast<const SR*>(p) + pos) : Re(0), Re(0));
      else v[r] = pos <= n / 2 ? Conv<S, Re>::ld(p + pos) : conj(Conv<S, Re>::ld(p + (n - pos)));
    }
  }
};
template <bool INV, class S, class Re>
struct OddOut {
  S* p;
  int n;
  Re s;
  bool valid;
  template <int R>
  __device__ __forceinline__ void store(const Cx<Re>* v, int j, int nb) const {
    using SR = typename RealOf<S>::type;
    if (!valid) return;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int pos = j + r * nb;
      if (INV) st_real<Re>(reinterpret_cast<SR*>(p) + pos, v[r].x * s);
      else if (pos <= n / 2) Conv<S, Re>::st(p + pos, v[r]);
    }
  }
};

// In place, every row is read whole before its first store only because the
// passes exchange through shared memory; a one-pass transform stores after
// its own loads, and one thread holds the whole row.
template <class Plan, bool INV, class S, class Re>
__global__ void __launch_bounds__(1024) k_real_odd(FftArgs a) {
  pdl_enter();
  const Plan P(a.pp);
  const Place<false, Plan::PAD> pl(a, P.T());
  Cx<Re>* sm = smem_base<Re>();
  const Cx<Re>* tw = reinterpret_cast<const Cx<Re>*>(a.tw);
  const int n = P.n();
  P.template transform<INV, false, false>(
      pl, sm, tw, OddIn<INV, S, Re>{reinterpret_cast<const S*>(a.in) + pl.in0(), n, a.sig_lo, a.sig_hi, pl.valid},
      OddOut<INV, S, Re>{reinterpret_cast<S*>(a.out) + pl.out0(), n, Re(a.scale), pl.valid});
}

// ---------------------------------------------------------------------------
// twiddle tables, built in FP64: tab[k] = exp(-2 pi i k / den), k < count
// ---------------------------------------------------------------------------
template <class Re>
__global__ void k_twiddle(Cx<Re>* tab, int count, int den) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  double s, c;
  // 2k/den carries one double rounding (relative 2^-53); no range reduction is
  // needed because k < den
  sincospi(2.0 * double(k) / double(den), &s, &c);
  tab[k] = mk<Re>(Re(c), Re(-s));
}

// Stage-ordered twiddles of a pass list: the pass that runs radix R after
// ns points' worth of earlier radices owns entries [ns, ns R), entry
// k + r ns = W_{ns R}^{k r} = W_n^{k r n/(ns R)} (the same integer exponent,
// hence the same bits, as a natural table).  The ranges of all passes tile
// [1, n); entry 0 is never read.
template <class Re>
__global__ void k_stage_twiddle(Cx<Re>* tab, PassPlan pp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pp.n) return;
  int ns = 1, p = 0;
  while (p + 1 < pp.npass && i >= ns * pp.radix[p]) ns *= pp.radix[p++];
  const int r = i / ns, k = i - r * ns;
  const long long e = (long long)k * r * (pp.n / (ns * pp.radix[p]));
  double s, c;
  sincospi(2.0 * double(e) / double(pp.n), &s, &c);
  tab[i] = mk<Re>(Re(c), Re(-s));
}

// ---------------------------------------------------------------------------
// compile-time plans for power-of-two lengths (radix 16 passes, then the
// leftover power of two); threads per transform = n / 16
// ---------------------------------------------------------------------------
template <int N>
struct Pow2;
template <> struct Pow2<16> { using L = RList<16>; static constexpr int T = 1; };
template <> struct Pow2<32> { using L = RList<16, 2>; static constexpr int T = 2; };
template <> struct Pow2<64> { using L = RList<16, 4>; static constexpr int T = 4; };
template <> struct Pow2<128> { using L = RList<16, 8>; static constexpr int T = 8; };
template <> struct Pow2<256> { using L = RList<16, 16>; static constexpr int T = 16; };
template <> struct Pow2<512> { using L = RList<16, 16, 2>; static constexpr int T = 32; };
template <> struct Pow2<1024> { using L = RList<16, 16, 4>; static constexpr int T = 64; };
template <> struct Pow2<2048> { using L = RList<16, 16, 8>; static constexpr int T = 128; };
template <> struct Pow2<4096> { using L = RList<16, 16, 16>; static constexpr int T = 256; };
template <> struct Pow2<8192> { using L = RList<16, 16, 16, 2>; static constexpr int T = 512; };
template <> struct Pow2<16384> { using L = RList<16, 16, 16, 4>; static constexpr int T = 1024; };

template <int N>
using Pow2Plan = FixPlan<N, Pow2<N>::T, typename Pow2<N>::L>;

// compile-time plans of radix-8 passes, 8 points per thread (n/8 threads per
// transform): half the registers of the radix-16 plans, for the strided
// fused convolution that also holds the kernel spectrum in registers
template <int N>
struct Pow2x8;
template <> struct Pow2x8<512> { using L = RList<8, 8, 8>; static constexpr int T = 64; };

template <int N>
using Pow2x8Plan = FixPlan<N, Pow2x8<N>::T, typename Pow2x8<N>::L, 8>;

// two-pass compile-time plans, 32 points per thread (n/32 threads per
// transform): one shared-memory exchange per FFT instead of two
template <int N>
struct Pow2x32;
template <> struct Pow2x32<512> { using L = RList<32, 16>; static constexpr int T = 16; };
template <> struct Pow2x32<1024> { using L = RList<32, 32>; static constexpr int T = 32; };

template <int N>
using Pow2x32Plan = FixPlan<N, Pow2x32<N>::T, typename Pow2x32<N>::L, 32>;


}  // namespace vdx
