// Template launcher shared by the per-storage-type translation units.
#pragma once

#include <cstdlib>

#include "vdx_internal.h"

namespace vdx {

// Compile-time convolutions of <= 256-thread CTAs load the kernel spectrum
// before the forward FFT (k_conv_pf) unless VDX_CONV_PREFETCH=0.
inline bool conv_prefetch() {
  static const bool on = [] {
    const char* e = std::getenv("VDX_CONV_PREFETCH");
    return !(e && e[0] == '0');
  }();
  return on;
}


// C2C with an optional fused element-wise operation (complex64 only):
// variant 0 = none, 1 = input weight, 2 = weighted |out|^2 partials
template <class Plan, bool INV, bool STRIDED, class S, class Re>
cudaError_t launch_c2c_layout(const FftArgs& a, const Launch& l, int variant) {
  if constexpr (std::is_same<S, Cx<float>>::value) {
    if (variant == 1) return enqueue_pdl(k_c2c<Plan, INV, STRIDED, S, Re, 1, 0>, l, a);
    if (variant == 2) return enqueue_pdl(k_c2c<Plan, INV, STRIDED, S, Re, 0, 1>, l, a);
  }
  if (variant != 0) return cudaErrorInvalidValue;
  return enqueue_pdl(k_c2c<Plan, INV, STRIDED, S, Re>, l, a);
}

template <class Plan, bool INV, class S, class Re>
cudaError_t launch_c2c(const FftArgs& a, const Launch& l, bool strided, int variant) {
  if (strided) return launch_c2c_layout<Plan, INV, true, S, Re>(a, l, variant);
  return launch_c2c_layout<Plan, INV, false, S, Re>(a, l, variant);
}

// convolution with optional spectrum output (complex64 only): variant 0 =
// none, 1 = write S (used with the conjugate product of a forward
// convolution), 2 = write aux * conj(S) * scale (used with the plain product
// of its adjoint); the plain product (KOP 1) exists for complex64 only
template <class Plan, int KOP, bool STRIDED, class S, class Re>
cudaError_t launch_conv_layout(const FftArgs& a, const Launch& l, int variant) {
  constexpr bool C64 = std::is_same<S, Cx<float>>::value;
  if constexpr (C64 && IsFixPlan<Plan>::value) {
    // 32-point plans have no registers for early loads, so for them k_conv_pf only
    // differs in reading the spectrum evict-first: right for one that each image
    // has of its own (64 x 512 x 512 images: 83.9 -> 81.9 us; 16 x 1024 x 513 along
    // axis 1: 74.1 -> 48.8), wrong for one that all share and L2 should keep
    // (40 x 1024 x 256: 75.8 -> 81.9), and at 1024 points wrong where the forward
    // spectrum is written too (64 x 1024 x 33: 24.2 -> 45.5).
    // Plans of up to 16 points gain by the early loads either way and read every
    // spectrum evict-first: for shared ones that costs 0 to 5 % (65536 x 256 rows
    // 48.0 us, 45.5 with plain loads; 16384 x 1024 66.0 and 65.4), and choosing the
    // policy at run time costs own ones as much (16384 x 1024 70.4 -> 73.6).
    const bool early = Plan::MAXE <= 16 || (a.ker_bs != 0 && (variant == 0 || a.pp.n < 1024));
    if (l.block.x <= 256 && early && conv_prefetch()) {
      if (variant == 0) return enqueue_pdl(k_conv_pf<Plan, STRIDED, S, Re, KOP>, l, a);
      if constexpr (KOP == 0) {
        if (variant == 1) return enqueue_pdl(k_conv_pf<Plan, STRIDED, S, Re, 0, 1>, l, a);
      } else {
        if (variant == 2) return enqueue_pdl(k_conv_pf<Plan, STRIDED, S, Re, 1, 2>, l, a);
      }
    }
  }
  if constexpr (C64 && KOP == 0) {
    if (variant == 1) return enqueue_pdl(k_conv<Plan, STRIDED, S, S, Re, 0, 1>, l, a);
  }
  if constexpr (C64 && KOP == 1) {
    if (variant == 2) return enqueue_pdl(k_conv<Plan, STRIDED, S, S, Re, 1, 2>, l, a);
  }
  if (variant != 0) return cudaErrorInvalidValue;
  if constexpr (KOP == 1 && !C64) return cudaErrorInvalidValue;
  else return enqueue_pdl(k_conv<Plan, STRIDED, S, S, Re, KOP>, l, a);
}

template <class Plan, int KOP, class S, class Re>
cudaError_t launch_conv(const FftArgs& a, const Launch& l, bool strided, int variant) {
  if (strided) return launch_conv_layout<Plan, KOP, true, S, Re>(a, l, variant);
  return launch_conv_layout<Plan, KOP, false, S, Re>(a, l, variant);
}

// Launches `op` with plan policy Plan (DynPlan or a compile-time FixPlan).
template <class Plan, class S, class Re>
cudaError_t launch_real(const FftArgs& a, const Launch& l, int op, bool with_odd) {
  switch (op) {
    case OP_R2C_EVEN:
      return enqueue_pdl(k_r2c_even<Plan, S, Re>, l, a);
    case OP_C2R_EVEN:
      return enqueue_pdl(k_c2r_even<Plan, S, Re>, l, a);
    case OP_R2C_ODD:
      if (with_odd) return enqueue_pdl(k_real_odd<Plan, false, S, Re>, l, a);
      return cudaErrorInvalidValue;
    case OP_C2R_ODD:
      if (with_odd) return enqueue_pdl(k_real_odd<Plan, true, S, Re>, l, a);
      return cudaErrorInvalidValue;
    default:
      return cudaErrorInvalidValue;
  }
}

template <class Plan, class S, class Re>
cudaError_t launch_c2c_any(const FftArgs& a, const Launch& l, int op, bool strided, int variant) {
  if (op == OP_C2C_FWD) return launch_c2c<Plan, false, S, Re>(a, l, strided, variant);
  return launch_c2c<Plan, true, S, Re>(a, l, strided, variant);
}

template <class Plan, class S, class Re>
cudaError_t launch_conv_any(const FftArgs& a, const Launch& l, bool strided, int kop, int variant) {
  if (kop == 0) return launch_conv<Plan, 0, S, Re>(a, l, strided, variant);
  return launch_conv<Plan, 1, S, Re>(a, l, strided, variant);
}

// The runtime-plan kernels of one storage type are split over three
// translation units (C2C, convolution, real) so they compile in parallel.
template <class S, class Re>
cudaError_t launch_dyn_c2c(const FftArgs& a, const Launch& l, int op, bool strided, int variant);
template <class S, class Re, bool STRIDED>
cudaError_t launch_dyn_c2c_layout(const FftArgs& a, const Launch& l, int op, int variant);
template <class S, class Re>
cudaError_t launch_dyn_conv(const FftArgs& a, const Launch& l, bool strided, int kop, int variant);
template <class S, class Re, bool STRIDED>
cudaError_t launch_dyn_conv_layout(const FftArgs& a, const Launch& l, int kop, int variant);
template <class S, class Re>
cudaError_t launch_dyn_real(const FftArgs& a, const Launch& l, int op);

// fp64 Bluestein transforms are bound by the few fp64 units of an SM, so the
// CTAs' spread over the SMs counts: a launch that starts while another drains
// (enqueue_pdl) finds some SMs fuller than others and keeps that imbalance (one
// after another, 500 x 509: 152.3 us, 94.3 with plain launches; 4000 x 121 146.2
// and 131.1, 300 x 1009 145.8 and 101.4).
template <class Plan, class S, class Re>
cudaError_t launch_bluestein(const FftArgs& a, const Launch& l, bool strided) {
  if constexpr (Same<Re, double>::value) {
    if (strided) return enqueue(k_bluestein<Plan, true, S, Re>, l, a);
    return enqueue(k_bluestein<Plan, false, S, Re>, l, a);
  } else {
    if (strided) return enqueue_pdl(k_bluestein<Plan, true, S, Re>, l, a);
    return enqueue_pdl(k_bluestein<Plan, false, S, Re>, l, a);
  }
}
template <class S, class Re>
cudaError_t launch_dyn_bluestein(const FftArgs& a, const Launch& l, bool strided);

template <class Plan, class S, class Re, bool WITH_ODD>
cudaError_t launch_with_plan(const FftArgs& a, const Launch& l, int op, bool strided, int kop, int variant) {
  if (variant != 0 && op != OP_C2C_FWD && op != OP_C2C_INV && op != OP_CONV) return cudaErrorInvalidValue;
  switch (op) {
    case OP_C2C_FWD:
    case OP_C2C_INV:
      return launch_c2c_any<Plan, S, Re>(a, l, op, strided, variant);
    case OP_CONV:
      return launch_conv_any<Plan, S, Re>(a, l, strided, kop, variant);
    case OP_BLUESTEIN:
      return launch_bluestein<Plan, S, Re>(a, l, strided);
    default:
      return launch_real<Plan, S, Re>(a, l, op, WITH_ODD);
  }
}

template <class S, class Re>
cudaError_t launch_fft(const FftArgs& a, const Launch& l, int op, bool strided, int kop, int variant) {
  // radix_dispatch ends at 16: a pass of a larger radix would do nothing
  for (int q = 0; q < a.pp.npass; ++q)
    if (a.pp.radix[q] > 16) return cudaErrorInvalidValue;
  if (variant != 0 && op != OP_C2C_FWD && op != OP_C2C_INV && op != OP_CONV) return cudaErrorInvalidValue;
  switch (op) {
    case OP_C2C_FWD:
    case OP_C2C_INV:
      return launch_dyn_c2c<S, Re>(a, l, op, strided, variant);
    case OP_CONV:
      return launch_dyn_conv<S, Re>(a, l, strided, kop, variant);
    case OP_BLUESTEIN:
      return launch_dyn_bluestein<S, Re>(a, l, strided);
    default:
      return launch_dyn_real<S, Re>(a, l, op);
  }
}

template <int N>
cudaError_t launch_fixed_c64(const FftArgs& a, const Launch& l, int op, bool strided, int kop, int variant) {
  return launch_with_plan<Pow2Plan<N>, Cx<float>, float, false>(a, l, op, strided, kop, variant);
}

// strided complex64 convolution with the 8- or 32-points-per-thread plan
template <int N>
cudaError_t launch_fixedpts_conv_c64(int pts, const FftArgs& a, const Launch& l, int kop, int variant) {
  if (pts == 8) {
    if (kop == 0) return launch_conv_layout<Pow2x8Plan<N>, 0, true, Cx<float>, float>(a, l, variant);
    return launch_conv_layout<Pow2x8Plan<N>, 1, true, Cx<float>, float>(a, l, variant);
  }
  if (kop == 0) return launch_conv_layout<Pow2x32Plan<N>, 0, true, Cx<float>, float>(a, l, variant);
  return launch_conv_layout<Pow2x32Plan<N>, 1, true, Cx<float>, float>(a, l, variant);
}

// every complex64 operation (C2C, convolution, even-length real transforms;
// either layout) on the 32-points-per-thread plan
template <int N>
cudaError_t launch_fixed32_c64(const FftArgs& a, const Launch& l, int op, bool strided, int kop, int variant) {
  return launch_with_plan<Pow2x32Plan<N>, Cx<float>, float, false>(a, l, op, strided, kop, variant);
}

}  // namespace vdx
