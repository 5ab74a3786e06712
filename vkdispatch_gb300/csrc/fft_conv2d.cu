// One-launch 2-D FFT convolution of real images (the whole convolve2DR):
// rfft of every row -> along each column FFT, * op(K), inverse FFT -> irfft of
// every row, for one image per thread-block cluster.
//
// An H x W image is split into C slabs of H / C rows, one per CTA of the
// cluster.  Each CTA keeps its slab's half spectrum (H / C rows x W/2 + 1
// columns of complex64) in shared memory for the whole launch:
//   phase 1: the CTA reads its rows from HBM and real-FFTs them into the slab;
//   phase 2: the CTA takes column tiles of the image; each column's H points
//            are read from the C slabs through distributed shared memory,
//            transformed, multiplied by the kernel spectrum (read from HBM),
//            transformed back and written back into the slabs;
//   phase 3: the CTA inverse-real-FFTs its slab's rows and writes them to HBM.
// HBM sees the image read once, the kernel spectrum read once and the result
// written once -- against three read/write passes for three separate launches
// (rfft, convolve, irfft).  Cluster barriers separate the phases.
//
// Semantics follow the composed path exactly (vkdispatch/fft/functions.py:
// 614-646): the row transform is unscaled, the column inverse is scaled by
// 1/H and the row inverse by 1/W when normalize is set, the kernel spectrum is
// read at the signal's own batch (or broadcast), and the packed row keeps the
// post-convolution Nyquist bin in its last complex slot, as the in-place
// irfft leaves it.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "fft_kernels.cuh"
#include "vdx_internal.h"

namespace cg = cooperative_groups;

namespace vdx {

namespace {

constexpr int kC2Threads = 512;

template <int H, int W, int C>
struct C2Geo {
  static constexpr int n = W / 2;                          // half-length complex FFT of a row
  static constexpr int COLS = n + 1;                        // spectrum columns
  static constexpr int R = H / C;                           // rows per CTA
  static constexpr int TR = Pow2<n>::T;                     // threads per row transform
  static constexpr int RROWS = kC2Threads / TR;             // rows per round
  static constexpr int NPAD = n + 1 + ((n + 1) >> 4) + 1;   // padded exchange slots per row
  static constexpr int TC = Pow2<H>::T;                     // threads per column transform
  static constexpr int MC = kC2Threads / TC;                // columns per tile
  static constexpr int TILES = (COLS + MC - 1) / MC;
  static constexpr int SLAB = R * COLS;                     // complex elements of the slab
  static constexpr int XCH = RROWS * NPAD > H * MC ? RROWS * NPAD : H * MC;  // exchange elements
  static constexpr size_t SMEM = size_t(SLAB + XCH) * sizeof(Cx<float>);
  static_assert(R % RROWS == 0, "rows per CTA must be a multiple of the rows per round");
};

struct RowPl {  // contiguous rows: t = thread of the row, m = row of the round
  int t, m;
  int npad;
  static constexpr bool kLinear = false;
  __device__ __forceinline__ int sidx(const PassPlan&, int i) const { return m * npad + i + (i >> 4); }
  __device__ __forceinline__ int sidx_plain(int i) const { return m * npad + i; }
};

struct ColPl {  // column tile: m = column of the tile, t = thread of the column
  int t, m, M;
  static constexpr bool kLinear = true;
  __device__ __forceinline__ int sidx(const PassPlan&, int i) const { return i * M + m; }
  __device__ __forceinline__ int pitch(const PassPlan&) const { return M; }
};

template <int H, int W, int C, int KOP>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(kC2Threads, 1) k_conv2d_real(Conv2dArgs a) {
  using G = C2Geo<H, W, C>;
  constexpr int MAXE = 16;
  constexpr int n = G::n, COLS = G::COLS;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const long long img = blockIdx.x / C;
  extern __shared__ __align__(16) unsigned char c2_raw[];
  Cx<float>* slab = reinterpret_cast<Cx<float>*>(c2_raw);
  Cx<float>* xch = slab + G::SLAB;
  const int tid = threadIdx.x;
  const PassPlan pp{};  // the compile-time pass chains take their sizes from the plan types
  Cx<float>* rows = a.data + (img * H + (long long)rank * G::R) * COLS;
  const Cx<float>* twr = a.tw_row;
  const Cx<float>* tw2 = a.tw2;

  // ---- phase 1: rfft of the CTA's rows into the slab
  {
    using P = Pow2Plan<n>;
    const P Pl(pp);
    RowPl pl;
    pl.t = tid % G::TR;
    pl.m = tid / G::TR;
    pl.npad = G::NPAD;
    for (int round = 0; round < G::R / G::RROWS; ++round) {
      const int r = round * G::RROWS + pl.m;
      const Cx<float>* in = rows + (long long)r * COLS;
      Cx<float> v[MAXE];
      Pl.template first<false>([&](auto rc) {
        constexpr int RR = decltype(rc)::value;
        gather<RR, MAXE, float>(v, n / RR, G::TR, pl.t, [&](int pos) { return in[pos]; });
      });
      Pl.template run<false, false>(v, pl, xch, twr);
      __syncthreads();
      Pl.template last<false>([&](auto rc) {
        constexpr int RR = decltype(rc)::value;
        each_natural<RR, MAXE, float>(v, n / RR, G::TR, pl.t,
                                      [&](int pos, Cx<float> val) { xch[pl.sidx_plain(pos)] = val; });
      });
      __syncthreads();
      Cx<float>* srow = slab + r * COLS;
      Pl.template last<false>([&](auto rc) {
        constexpr int RR = decltype(rc)::value;
        each_natural<RR, MAXE, float>(v, n / RR, G::TR, pl.t, [&](int k, Cx<float> zk) {
          const int kc = k == 0 ? 0 : n - k;
          const Cx<float> zc = conj(xch[pl.sidx_plain(kc)]);
          const Cx<float> e = scale(zk + zc, 0.5f);
          const Cx<float> d = scale(zk - zc, 0.5f);
          const Cx<float> o = mk<float>(d.y, -d.x);  // d / i
          srow[k] = e + cmul(ldg(&tw2[k]), o);
        });
      });
      if (pl.t == 0) {
        const Cx<float> z0 = xch[pl.sidx_plain(0)];
        srow[n] = mk<float>(z0.x - z0.y, 0.f);
      }
    }
  }
  cluster.sync();

  // ---- phase 2: column tiles through distributed shared memory
  {
    using P = Pow2Plan<H>;
    const P Pl(pp);
    ColPl pl;
    pl.M = G::MC;
    pl.m = tid % G::MC;
    pl.t = tid / G::MC;
    const Cx<float>* ker = a.ker + (a.ker_bs ? img * a.ker_bs : 0);
    const Cx<float>* twc = a.tw_col;
    const Cx<float>* twcr = a.tw_colr;
    const float cs = a.col_scale;
    for (int g = rank; g < G::TILES; g += C) {
      const int c = g * G::MC + pl.m;
      const bool valid = c < COLS;
      const int cc = valid ? c : 0;
      Cx<float> v[MAXE];
      Pl.template first<false>([&](auto rc) {
        constexpr int RR = decltype(rc)::value;
        gather<RR, MAXE, float>(v, H / RR, G::TC, pl.t, [&](int pos) {
          const int owner = pos / G::R, lr = pos - owner * G::R;
          const Cx<float>* src = cluster.map_shared_rank(slab + lr * COLS + cc, owner);
          return valid ? *src : mk<float>(0.f, 0.f);
        });
      });
      Pl.template run<false, false>(v, pl, xch, twc);
      Pl.template last<false>([&](auto rc) {
        constexpr int RR = decltype(rc)::value;
        constexpr int B = MAXE / RR;
        constexpr int nb = H / RR;
#pragma unroll
        for (int b = 0; b < B; ++b) {
          const int j = pl.t + b * G::TC;
          if (j < nb) {
#pragma unroll
            for (int r = 0; r < RR; ++r) {
              const int pos = j + r * nb;
              const Cx<float> kv = valid ? ker[(long long)pos * COLS + cc] : mk<float>(0.f, 0.f);
              v[b * RR + r] = KOP == 0 ? cmulc(v[b * RR + r], kv) : cmul(v[b * RR + r], kv);
            }
          }
        }
      });
      Pl.template run<true, true>(v, pl, xch, twcr);
      Pl.template last<true>([&](auto rc) {
        constexpr int RR = decltype(rc)::value;
        each_natural<RR, MAXE, float>(v, H / RR, G::TC, pl.t, [&](int pos, Cx<float> val) {
          if (!valid) return;
          const int owner = pos / G::R, lr = pos - owner * G::R;
          Cx<float>* dst = cluster.map_shared_rank(slab + lr * COLS + c, owner);
          *dst = scale(val, cs);
        });
      });
    }
  }
  cluster.sync();

  // ---- phase 3: irfft of the CTA's rows from the slab to HBM
  {
    using P = Pow2Plan<n>;
    const P Pl(pp);
    RowPl pl;
    pl.t = tid % G::TR;
    pl.m = tid / G::TR;
    pl.npad = G::NPAD;
    const float rs = a.row_scale;
    for (int round = 0; round < G::R / G::RROWS; ++round) {
      const int r = round * G::RROWS + pl.m;
      const Cx<float>* X = slab + r * COLS;
      Cx<float>* out = rows + (long long)r * COLS;
      Cx<float> v[MAXE];
      Pl.template first<false>([&](auto rc) {
        constexpr int RR = decltype(rc)::value;
        gather<RR, MAXE, float>(v, n / RR, G::TR, pl.t, [&](int k) {
          Cx<float> xk = X[k];
          Cx<float> xn = X[n - k];
          if (k == 0) {  // the imaginary parts of bins 0 and n do not enter a real inverse
            xk.y = 0.f;
            xn.y = 0.f;
          }
          const Cx<float> xc = conj(xn);
          const Cx<float> s = xk + xc;
          const Cx<float> d = xk - xc;
          const Cx<float> wd = cmulc(d, ldg(&tw2[k]));  // d * W^{-k}
          return mk<float>(s.x - wd.y, s.y + wd.x);      // s + i*wd
        });
      });
      Pl.template run<true, false>(v, pl, xch, twr);
      Pl.template last<false>([&](auto rc) {
        constexpr int RR = decltype(rc)::value;
        each_natural<RR, MAXE, float>(v, n / RR, G::TR, pl.t,
                                      [&](int pos, Cx<float> val) { out[pos] = scale(val, rs); });
      });
      if (pl.t == 0) out[n] = X[n];
    }
  }
}

template <int H, int W, int C>
cudaError_t launch_hw(const Conv2dArgs& a, long long images, int kop, cudaStream_t s) {
  Launch l;
  l.grid = dim3((unsigned)(images * C));
  l.block = dim3(kC2Threads);
  l.smem = C2Geo<H, W, C>::SMEM;
  l.stream = s;
  return kop == 0 ? enqueue(k_conv2d_real<H, W, C, 0>, l, a) : enqueue(k_conv2d_real<H, W, C, 1>, l, a);
}

template <int H, int W, int C>
cudaError_t clusters_hw(int* count) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C * 64);
  cfg.blockDim = dim3(kC2Threads);
  cfg.dynamicSmemBytes = C2Geo<H, W, C>::SMEM;
  cudaError_t e = cudaFuncSetAttribute(k_conv2d_real<H, W, C, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)C2Geo<H, W, C>::SMEM);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_conv2d_real<H, W, C, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)C2Geo<H, W, C>::SMEM);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = C;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaOccupancyMaxActiveClusters(count, k_conv2d_real<H, W, C, 0>, &cfg);
}

}  // namespace

bool conv2d_real_supported(int H, int W) { return H == 512 && W == 512; }

cudaError_t conv2d_real_max_clusters(int H, int W, int* count) {
  *count = 0;
  if (H == 512 && W == 512) return clusters_hw<512, 512, 8>(count);
  return cudaErrorInvalidValue;
}

cudaError_t launch_conv2d_real(const Conv2dArgs& a, int H, int W, long long images, int kop, cudaStream_t s) {
  if (H == 512 && W == 512) return launch_hw<512, 512, 8>(a, images, kop, s);
  return cudaErrorInvalidValue;
}

}  // namespace vdx
