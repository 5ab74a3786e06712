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
#include <cuda_runtime.h>

#include "fft_large.cuh"

namespace vdx {

int fourstep_pitch(const PassPlan& pp) { return fs_pitch(pp.M, pp.T); }

cudaError_t launch_fourstep_pass(const FsArgs& a, const Launch& l, int store, bool inv, int mode, bool few) {
  few = few && !fourstep_fixed(a.pp);
  switch (store) {
    case ST_C64: return few ? launch_fs_few_c64(a, l, inv, mode) : launch_fs_c64(a, l, inv, mode);
    case ST_C32: return few ? launch_fs_few_c32(a, l, inv, mode) : launch_fs_c32(a, l, inv, mode);
    case ST_BF16: return few ? launch_fs_few_bf16(a, l, inv, mode) : launch_fs_bf16(a, l, inv, mode);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace vdx
