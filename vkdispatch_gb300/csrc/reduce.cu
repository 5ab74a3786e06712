// Batched map-reduce kernels.
//
// Same two-stage shape as the reference (vkdispatch/reduce/stage.py:31-145:
// grid-stride accumulate -> shared-memory tree -> subgroup butterfly; stage 2
// folds the per-workgroup partials), re-designed: one to eight warps fold a
// part of a row, loads of a whole block in flight, a tree of slots and lanes
// whose order depends on n alone; partials go to a caller-provided workspace
// rather than the output buffer, and stage 2 folds the partials of a row in a
// fixed order, so results never depend on scheduling.
#include "vdx_internal.h"
#include "vdx.h"

#include <math_constants.h>

#include <cstdio>
#include <limits>
#include <map>
#include <mutex>
#include <utility>

namespace vdx {

namespace {

template <class T, int OP>
__device__ __forceinline__ T identity() {
  if constexpr (OP == VDX_RED_ADD || OP == VDX_RED_OR || OP == VDX_RED_XOR) return T(0);
  else if constexpr (OP == VDX_RED_MUL) return T(1);
  else if constexpr (OP == VDX_RED_AND) return T(~0ull);
  else if constexpr (std::is_floating_point<T>::value) {
    if (OP == VDX_RED_MIN) return T(CUDART_INF);
    return T(-CUDART_INF);
  } else {
    if (OP == VDX_RED_MIN) return std::numeric_limits<T>::max();
    return std::numeric_limits<T>::lowest();
  }
}

template <class T, int OP>
__device__ __forceinline__ T combine(T a, T b) {
  if constexpr (OP == VDX_RED_ADD) return a + b;
  else if constexpr (OP == VDX_RED_MUL) return a * b;
  else if constexpr (OP == VDX_RED_MIN) return a < b ? a : b;
  else if constexpr (OP == VDX_RED_MAX) return a > b ? a : b;
  else if constexpr (std::is_integral<T>::value) {
    if constexpr (OP == VDX_RED_AND) return a & b;
    else if constexpr (OP == VDX_RED_OR) return a | b;
    else return a ^ b;
  } else {
    return a;
  }
}

// map of one input element to the accumulation type
template <class In, class T, int MAP>
__device__ __forceinline__ T apply_map(In x) {
  if constexpr (std::is_same<In, Cx<float>>::value) {
    if constexpr (MAP == VDX_MAP_ABS) return T(sqrtf(x.x * x.x + x.y * x.y));
    else if constexpr (MAP == VDX_MAP_SQUARE) return T(x.x * x.x + x.y * x.y);
    else if constexpr (MAP == VDX_MAP_IMAG) return T(x.y);
    else return T(x.x);
  } else {
    if constexpr (MAP == VDX_MAP_ABS) return x < In(0) ? T(-x) : T(x);
    else if constexpr (MAP == VDX_MAP_SQUARE) return T(x) * T(x);
    else if constexpr (MAP == VDX_MAP_SIN) {
      if constexpr (std::is_same<In, double>::value) return T(sin(x));
      else return T(sinf(float(x)));
    } else return T(x);
  }
}

template <class T>
__device__ __forceinline__ T shfl_down(T v, int d) {
  return __shfl_down_sync(0xffffffffu, v, d);
}

template <class T, int OP>
__device__ __forceinline__ T block_reduce(T v, T* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v = combine<T, OP>(v, shfl_down(v, d));
  if (lane == 0) sh[w] = v;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  if (w == 0) {
    v = lane < nw ? sh[lane] : identity<T, OP>();
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v = combine<T, OP>(v, shfl_down(v, d));
  }
  return v;
}

// Stage 1: part p of row b covers elements [p*chunk, min(n, (p+1)*chunk)), in
// blocks of 512 elements, 16 per lane of a warp.  Block k belongs to slot k % 8;
// a lane folds the blocks of its slots, the slots are folded as a tree, and the
// lanes last.  W warps (1 to 8) share a part's slots, and a CTA of eight warps
// holds 8 / W parts: of its row, or, where more than one in 16 would stay empty
// that way, numbered over all rows (16384 x 4096 floats, one part a row: 81.6 us
// by rows, 45.3; 65000 x 512 97.2 and 43.3; 20000 x 18000 complex, five parts,
// 457 and 414; but 148 x 21716 complex, no place empty, 8.3 by rows and 9.2 over
// all).  The order depends on n alone, whatever W is, so results do too, and W
// follows the amount of work: two warps per 4096 elements where the parts fill
// the chip (one 512-thread CTA per part spent 16 instructions per element, most
// of them on the fold: 1024 x 65536 floats took 54.9 us against a copy rate of
// 39.5), eight where they do not (262144 complex magnitudes on two warps a part
// took 11.4 us, their loads one after another).
//
// A lane's elements of a block are neighbours in fours where n is a multiple of
// four, in 16-byte loads if the part starts on such a boundary; rows of another
// n start at any element, so there each load of a warp is of neighbours (33 rows
// of 1710185 complex elements: 94 us; 104 us in fours).
constexpr int kWarps = 8;
constexpr int kVec = 4;
constexpr int kStep = 32 * kVec;   // elements of a warp per step
constexpr int kBlock = 4 * kStep;  // elements of a block
constexpr long long kFullWarps = 152 * 32;  // warps that fill the chip

inline int part_warps(long long chunk, long long parts) {
  int w = 1;
  while (w < kWarps && chunk > 64ll * 32 * w) w <<= 1;
  while (w < kWarps && (long long)kBlock * w < chunk && parts * w < kFullWarps) w <<= 1;
  return w;
}

template <class In>
struct alignas(sizeof(In) * kVec <= 16 ? sizeof(In) * kVec : 16) Pack {
  In v[kVec];
};

template <class T, int OP>
__device__ __forceinline__ T warp_reduce(T v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v = combine<T, OP>(v, shfl_down(v, d));
  return v;
}

// A lane's fold of step k of a block; the first `left` elements count (all of
// them if WHOLE).  pack: fours of neighbours; vec: q is aligned for 16-byte loads.
template <class In, bool WHOLE>
__device__ __forceinline__ void load_step(In (&x)[kVec], const In* __restrict__ q, int k, int left, bool pack, bool vec,
                                          int lane) {
  const int first = k * kStep + (pack ? lane * kVec : lane), de = pack ? 1 : 32;
  if (vec) {
    Pack<In> p4{};
    if (WHOLE || first < left) p4 = *reinterpret_cast<const Pack<In>*>(q + first);
#pragma unroll
    for (int i = 0; i < kVec; ++i) x[i] = p4.v[i];
  } else {
#pragma unroll
    for (int i = 0; i < kVec; ++i) x[i] = WHOLE || first + i * de < left ? q[first + i * de] : In{};
  }
}

template <class In, class T, int OP, int MAP, bool WHOLE>
__device__ __forceinline__ T fold_step(const In (&x)[kVec], int k, int left, bool pack, int lane) {
  const int first = k * kStep + (pack ? lane * kVec : lane), de = pack ? 1 : 32;
  T m[kVec];
#pragma unroll
  for (int i = 0; i < kVec; ++i)
    m[i] = WHOLE || first + i * de < left ? apply_map<In, T, MAP>(x[i]) : identity<T, OP>();
  return combine<T, OP>(combine<T, OP>(m[0], m[1]), combine<T, OP>(m[2], m[3]));
}

// A lane's fold of a block: the loads of all four steps first where the block is
// whole; a part's last block goes step by step and stops with its elements.
template <class In, class T, int OP, int MAP>
__device__ __forceinline__ T fold_block(const In* __restrict__ q, long long len, bool pack, bool vec, int lane) {
  if (len >= kBlock) {
    In x[4][kVec];
    if (vec) {
#pragma unroll
      for (int k = 0; k < 4; ++k) load_step<In, true>(x[k], q, k, kBlock, pack, true, lane);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) load_step<In, true>(x[k], q, k, kBlock, pack, false, lane);
    }
    T r[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) r[k] = fold_step<In, T, OP, MAP, true>(x[k], k, kBlock, pack, lane);
    return combine<T, OP>(combine<T, OP>(r[0], r[1]), combine<T, OP>(r[2], r[3]));
  }
  const int left = (int)len;
  T lower = identity<T, OP>(), pair = lower, r = lower;
#pragma unroll 1
  for (int k = 0; k * kStep < left; ++k) {
    In x[kVec];
    load_step<In, false>(x, q, k, left, pack, vec, lane);
    r = fold_step<In, T, OP, MAP, false>(x, k, left, pack, lane);
    if (k & 1) {
      r = combine<T, OP>(pair, r);
      if (k == 1) lower = r;
      pair = identity<T, OP>();
    } else {
      pair = r;
    }
    if (k != 1) r = combine<T, OP>(lower, r);
  }
  return r;
}

template <class In, class T, int OP, int MAP>
__global__ void __launch_bounds__(32 * kWarps) k_reduce_partial(const In* __restrict__ in, long long n, long long chunk,
                                                                T* __restrict__ part, unsigned nparts, unsigned total,
                                                                int W) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __shared__ T sh[kWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = warp & (W - 1);  // warp of its part; W is a power of two
  const unsigned u = blockIdx.x * unsigned(kWarps / W) + unsigned(warp / W);
  unsigned b, p, g;
  bool live;
  if (total) {  // parts numbered over all rows
    g = u;
    b = g / nparts;
    p = g - b * nparts;
    live = g < total;
  } else {
    b = blockIdx.y;
    p = u;
    g = b * nparts + p;
    live = p < nparts;
  }
  const long long lo = (long long)p * chunk;
  const long long len = (lo + chunk < n ? lo + chunk : n) - lo;
  T acc = identity<T, OP>();
  if (live && len > 0) {
    const In* q = in + (long long)b * n + lo;
    const bool pack = n % kVec == 0;
    const bool vec = pack && reinterpret_cast<unsigned long long>(q) % alignof(Pack<In>) == 0;
    const int slots = kWarps / W;
    T h1 = acc, h2 = acc, h4 = acc;  // finished lower halves of the slots' tree
    for (int j = 0; j < slots; ++j) {
      T v = identity<T, OP>();
      for (long long e = (long long)(w * slots + j) * kBlock; e < len; e += kWarps * kBlock)
        v = combine<T, OP>(v, fold_block<In, T, OP, MAP>(q + e, len - e, pack, vec, lane));
      if (slots == 1) acc = v;
      else if (!(j & 1)) h1 = v;
      else {
        v = combine<T, OP>(h1, v);
        if (slots == 2) acc = v;
        else if (!(j & 2)) h2 = v;
        else {
          v = combine<T, OP>(h2, v);
          if (slots == 4) acc = v;
          else if (!(j & 4)) h4 = v;
          else acc = combine<T, OP>(h4, v);
        }
      }
    }
  }
  for (int d = 1; d < W; d <<= 1) {  // the upper levels of the slots' tree, across the part's warps
    sh[warp][lane] = acc;
    __syncthreads();
    if ((w & (2 * d - 1)) == 0) acc = combine<T, OP>(acc, sh[warp + d][lane]);
    __syncthreads();
  }
  if (w != 0) return;
  acc = warp_reduce<T, OP>(acc);
  if (lane == 0 && live) part[g] = acc;
}

// Stage 2 folds the partials of a row in a fixed order: one warp per row for
// up to 32 partials, else one CTA per row.  It is launched to start while
// stage 1 drains and waits for stage 1's partials here.
constexpr int kThreads = 512;
template <class T, int OP>
__global__ void __launch_bounds__(kThreads) k_reduce_final(const T* __restrict__ part, int nparts, long long rows,
                                                           T* __restrict__ out) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (nparts <= 32) {
    const long long b = (long long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    T acc = b < rows && lane < nparts ? part[b * nparts + lane] : identity<T, OP>();
    acc = warp_reduce<T, OP>(acc);
    if (lane == 0 && b < rows) out[b] = acc;
    return;
  }
  __shared__ T sh[32];
  const long long b = blockIdx.x;
  T acc = identity<T, OP>();
  for (int i = threadIdx.x; i < nparts; i += kThreads) acc = combine<T, OP>(acc, part[b * nparts + i]);
  acc = block_reduce<T, OP>(acc, sh);
  if (threadIdx.x == 0) out[b] = acc;
}

template <class In, class T, int OP, int MAP>
cudaError_t run(const void* in, long long n, long long batch, void* out, void* partials, int nparts, cudaStream_t s) {
  // parts start on 16-byte steps of the row
  const long long chunk = ((n + nparts - 1) / nparts + 3) & ~3ll;
  const long long total = nparts * batch;  // at most 1024 parts of 65535 rows
  const int W = part_warps(chunk, total), G = kWarps / W;
  const int per_row = (nparts + G - 1) / G;
  const bool flat = (per_row * G - nparts) * 16 > nparts;
  const dim3 grid = flat ? dim3((unsigned)((total + G - 1) / G)) : dim3((unsigned)per_row, (unsigned)batch);
  const Launch l1{grid, dim3(32 * kWarps), 0, s};
  const In* src = reinterpret_cast<const In*>(in);
  T* part = reinterpret_cast<T*>(partials);
  cudaError_t e = enqueue(k_reduce_partial<In, T, OP, MAP>, l1, src, n, chunk, part, (unsigned)nparts,
                          flat ? (unsigned)total : 0u, W);
  if (e != cudaSuccess) return e;
  Launch l2{dim3((unsigned)batch), dim3(kThreads), 0, s};
  if (nparts <= 32) {
    l2.block = dim3(batch == 1 ? 32 : 128);
    l2.grid = dim3((unsigned)((batch + l2.block.x / 32 - 1) / (l2.block.x / 32)));
  }
  const T* cpart = part;
  return enqueue_pdl(k_reduce_final<T, OP>, l2, cpart, nparts, batch, reinterpret_cast<T*>(out));
}

template <class In, class T, int OP>
cudaError_t by_map(int map, const void* in, long long n, long long batch, void* out, void* partials, int nparts,
                   cudaStream_t s) {
  switch (map) {
    case VDX_MAP_IDENTITY: return run<In, T, OP, VDX_MAP_IDENTITY>(in, n, batch, out, partials, nparts, s);
    case VDX_MAP_ABS: return run<In, T, OP, VDX_MAP_ABS>(in, n, batch, out, partials, nparts, s);
    case VDX_MAP_SQUARE: return run<In, T, OP, VDX_MAP_SQUARE>(in, n, batch, out, partials, nparts, s);
    case VDX_MAP_REAL: return run<In, T, OP, VDX_MAP_REAL>(in, n, batch, out, partials, nparts, s);
    case VDX_MAP_IMAG: return run<In, T, OP, VDX_MAP_IMAG>(in, n, batch, out, partials, nparts, s);
    case VDX_MAP_SIN: return run<In, T, OP, VDX_MAP_SIN>(in, n, batch, out, partials, nparts, s);
    default: return cudaErrorInvalidValue;
  }
}

template <class In, class T>
cudaError_t by_op_arith(int op, int map, const void* in, long long n, long long batch, void* out, void* partials,
                        int nparts, cudaStream_t s) {
  switch (op) {
    case VDX_RED_ADD: return by_map<In, T, VDX_RED_ADD>(map, in, n, batch, out, partials, nparts, s);
    case VDX_RED_MUL: return by_map<In, T, VDX_RED_MUL>(map, in, n, batch, out, partials, nparts, s);
    case VDX_RED_MIN: return by_map<In, T, VDX_RED_MIN>(map, in, n, batch, out, partials, nparts, s);
    case VDX_RED_MAX: return by_map<In, T, VDX_RED_MAX>(map, in, n, batch, out, partials, nparts, s);
    default: return cudaErrorInvalidValue;
  }
}

template <class In, class T>
cudaError_t by_op_int(int op, int map, const void* in, long long n, long long batch, void* out, void* partials,
                      int nparts, cudaStream_t s) {
  switch (op) {
    case VDX_RED_AND: return run<In, T, VDX_RED_AND, VDX_MAP_IDENTITY>(in, n, batch, out, partials, nparts, s);
    case VDX_RED_OR: return run<In, T, VDX_RED_OR, VDX_MAP_IDENTITY>(in, n, batch, out, partials, nparts, s);
    case VDX_RED_XOR: return run<In, T, VDX_RED_XOR, VDX_MAP_IDENTITY>(in, n, batch, out, partials, nparts, s);
    default: return by_op_arith<In, T>(op, map, in, n, batch, out, partials, nparts, s);
  }
}

}  // namespace

cudaError_t launch_reduce(int op, int map, int in_type, const void* in, long long n, long long batch, void* out,
                          void* partials, int nparts, cudaStream_t s) {
  switch (in_type) {
    case VDX_F32: return by_op_arith<float, float>(op, map, in, n, batch, out, partials, nparts, s);
    case VDX_F64: return by_op_arith<double, double>(op, map, in, n, batch, out, partials, nparts, s);
    case VDX_C64: return by_op_arith<Cx<float>, float>(op, map, in, n, batch, out, partials, nparts, s);
    case VDX_I32: return by_op_int<int, int>(op, map, in, n, batch, out, partials, nparts, s);
    case VDX_U32: return by_op_int<unsigned, unsigned>(op, map, in, n, batch, out, partials, nparts, s);
    default: return cudaErrorInvalidValue;
  }
}

// ---------------------------------------------------------------------------
// Allocation-free reduction: the stage-1 partials live in a fixed device
// array instead of a caller-provided workspace.  Every GPU that loads libvdx
// holds VDX_REDUCE_NOALLOC_SCRATCH_BYTES of it until the process exits.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_reduce_scratch[VDX_REDUCE_NOALLOC_SCRATCH_BYTES];

namespace {

std::mutex g_scratch_mu;
// (device ordinal, CUDA context) -> device address of g_reduce_scratch.  The
// context is part of the key because a device reset (cudaDeviceReset, or a
// primary-context release and re-create) reloads the module, after which an
// address resolved in the old context is stale.
std::map<std::pair<int, void*>, void*> g_scratch_addr;

typedef int (*CtxGetCurrentFn)(void**);  // CUresult cuCtxGetCurrent(CUcontext*)

// cuCtxGetCurrent, fetched once from the driver without linking libcuda.
CtxGetCurrentFn ctx_get_current() {
  static CtxGetCurrentFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<CtxGetCurrentFn>(p);
  });
  return fn;
}

// Host code only sees a host-side stand-in under the name g_reduce_scratch;
// its device address comes from cudaGetSymbolAddress, resolved once per
// device and context with that device current (the caller's current device).
cudaError_t scratch_for_current_device(void** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  // Before this thread's first runtime call no context may be current yet;
  // cudaGetSymbolAddress below makes the primary context current, and the
  // context is read again after it.
  void* ctx = nullptr;
  CtxGetCurrentFn get = ctx_get_current();
  if (get) get(&ctx);
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (ctx) {
    auto it = g_scratch_addr.find({dev, ctx});
    if (it != g_scratch_addr.end()) {
      *out = it->second;
      return cudaSuccess;
    }
  }
  void* p = nullptr;
  e = cudaGetSymbolAddress(&p, g_reduce_scratch);
  if (e != cudaSuccess) return e;
  if (!ctx && get) get(&ctx);  // the lookup made the primary context current
  if (ctx) g_scratch_addr[{dev, ctx}] = p;
  *out = p;
  return cudaSuccess;
}

}  // namespace

}  // namespace vdx

extern "C" int vdx_reduce_noalloc(int op, int map, int in_type, const void* in, int64_t n, int64_t batch, void* out,
                                  void* stream) {
  using namespace vdx;
  int rc = check_reduce_args(op, map, in_type, in, n, batch, out);
  if (rc != VDX_OK) return rc;
  int64_t parts = 0;
  rc = vdx_reduce_partial_count(n, &parts);
  if (rc != VDX_OK) return rc;
  const long long need = (long long)parts * batch * reduce_out_bytes(in_type);
  if (need > (long long)VDX_REDUCE_NOALLOC_SCRATCH_BYTES) {
    char msg[256];
    std::snprintf(msg, sizeof(msg),
                  "vdx_reduce_noalloc: %lld rows of %lld elements need %lld bytes of partials, above the %d-byte "
                  "static scratch; use vdx_reduce with a workspace",
                  (long long)batch, (long long)n, need, (int)VDX_REDUCE_NOALLOC_SCRATCH_BYTES);
    return set_error(VDX_ERR_UNSUPPORTED, msg);
  }
  void* scratch = nullptr;
  cudaError_t e = scratch_for_current_device(&scratch);
  if (e != cudaSuccess) {
    char msg[256];
    std::snprintf(msg, sizeof(msg), "vdx_reduce_noalloc: cudaGetSymbolAddress of the scratch array failed: %s",
                  cudaGetErrorString(e));
    return set_error(VDX_ERR_CUDA, msg);
  }
  e = launch_reduce(op, map, in_type, in, n, batch, out, scratch, (int)parts, reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) {
    char msg[256];
    std::snprintf(msg, sizeof(msg), "vdx_reduce_noalloc launch: %s", cudaGetErrorString(e));
    return set_error(VDX_ERR_CUDA, msg);
  }
  return VDX_OK;
}
