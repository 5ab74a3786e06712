// Long axes as a four-step pair of launches (complex-to-complex, fp32 compute).
//
// An axis of length N = N1 * N0 is indexed n = b1 * N0 + b0 and k = k1 + N1 * k2.
//   pass A: for every b0, the N1-point transform over b1, times W_N^{b0 k1},
//           into a workspace;
//   pass B: for every k1, the N0-point transform over b0, written to
//           X[k1 + N1 k2].
// Both passes are tiles of M adjacent columns and one short transform per
// column (n = N1 or N0, a few hundred points at most), so each CTA is small,
// several run on an SM at once and their loads overlap the other CTAs'
// butterflies -- which a single CTA holding a whole 16384-point transform
// (one per SM, all 64K registers) cannot do.  The price is a second trip
// through HBM for the intermediate; the host can walk the array in chunks
// whose workspace fits in L2 instead (VDX_FOURSTEP_WS_MB).
//
// The reference has no multi-kernel transform: its planner rejects axes
// above 16384 points (vkdispatch/fft/config.py:185-190) and runs every axis
// inside one workgroup (vkdispatch/fft/shader_factories.py:11-60).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "fft_large.cuh"

namespace vdx {

namespace {

// cuTensorMapEncodeTiled, fetched once from the driver without linking libcuda
PFN_cuTensorMapEncodeTiled_v12000 encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    cudaGetLastError();
  });
  return fn;
}

size_t store_size(int store) { return store == ST_C64 ? 8 : 4; }

// The pass input as a tensor: element (c, pos, br, bq) at
// base + bq * in_bs1 + br * in_bs2 + pos * in_ps + c; dimensions of extent 1
// are dropped and the rest ordered by stride.
bool encode_tile_map(const FsArgs& a, int store, CUtensorMap* map, TmaTile* tt) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = encoder();
  if (!enc) return false;
  const long long es = (long long)store_size(store);
  const int M = a.pp.M, n = a.pp.n;
  struct D {
    long long extent, stride;
    int which;  // 0 = pos, 1 = br, 2 = bq
  };
  D d[3];
  int k = 0;
  d[k++] = D{n, a.in_ps, 0};
  if (a.split > 1) d[k++] = D{a.split, a.in_bs2, 1};
  const long long bq_count = (a.nbatch + a.split - 1) / a.split;
  if (bq_count > 1) d[k++] = D{bq_count, a.in_bs1, 2};
  std::sort(d, d + k, [](const D& x, const D& y) { return x.stride < y.stride; });
  cuuint64_t dims[5], strides[4];
  cuuint32_t box[5], estr[5];
  dims[0] = (cuuint64_t)a.ncols;
  box[0] = (cuuint32_t)M;
  estr[0] = 1;
  tt->rank = 1 + k;
  tt->row_dim = tt->br_dim = tt->bq_dim = -1;
  for (int i = 0; i < k; ++i) {
    dims[i + 1] = (cuuint64_t)d[i].extent;
    strides[i] = (cuuint64_t)(d[i].stride * es);
    box[i + 1] = d[i].which == 0 ? (cuuint32_t)n : 1;
    estr[i + 1] = 1;
    if (d[i].which == 0) tt->row_dim = i + 1;
    if (d[i].which == 1) tt->br_dim = i + 1;
    if (d[i].which == 2) tt->bq_dim = i + 1;
    if (strides[i] % 16 != 0 || strides[i] >= (1ull << 40)) return false;
  }
  // box extents of 1 add no stride, so the staged tile is [row][column] wherever the rows sit
  if (tt->rank < 2 || tt->rank > 4 || tt->row_dim < 1) return false;
  const CUtensorMapDataType ty = store == ST_C64 ? CU_TENSOR_MAP_DATA_TYPE_UINT64 : CU_TENSOR_MAP_DATA_TYPE_UINT32;
  const CUresult r = enc(map, ty, (cuuint32_t)tt->rank, const_cast<void*>(a.in), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

}  // namespace

// Staged passes are used where they measured faster: 4-byte storage (bf16 or
// fp16 pairs) on strided axes, whose rows are 128-byte segments far apart
// (16384^2 bf16 strided axis: 1.295 -> 1.131 ms).  For complex64 and for the
// contiguous-axis passes the staging tile's shared memory costs more
// occupancy than the bulk copy saves (1.40 -> 1.53 ms, 1.56 -> 2.04 ms).
bool fourstep_tma_ok(const FsArgs& a, int store) {
  const long long es = (long long)store_size(store);
  const int n = a.pp.n, M = a.pp.M;
  if (store != ST_C32 && store != ST_BF16) return false;
  if (n != 128) return false;  // one box of 128 rows, the compile-time 128-point plan
  if ((M * es) % 16 != 0) return false;
  if (reinterpret_cast<uintptr_t>(a.in) % 16 != 0) return false;
  return encoder() != nullptr;
}

cudaError_t launch_fourstep_pass(const FsArgs& a, const Launch& l, int store, bool inv, int mode, bool tma) {
  CUtensorMap map;
  std::memset(&map, 0, sizeof(map));
  TmaTile tt{0, -1, -1, -1};
  Launch lt = l;
  if (tma && fourstep_tma_ok(a, store) && encode_tile_map(a, store, &map, &tt)) {
    lt.smem = std::max(l.smem, size_t(a.pp.n + 1) * a.pp.M * 8) + size_t(a.pp.n) * a.pp.M * store_size(store) + 128;
  } else {
    tt.rank = 0;
  }
  switch (store) {
    case ST_C64: return launch_fs_c64(map, a, tt, lt, inv, mode);
    case ST_C32: return launch_fs_c32(map, a, tt, lt, inv, mode);
    case ST_BF16: return launch_fs_bf16(map, a, tt, lt, inv, mode);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace vdx
