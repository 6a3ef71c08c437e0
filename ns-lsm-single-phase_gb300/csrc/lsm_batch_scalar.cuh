// lsm_batch_scalar.cuh -- scalar device functions of the batched path
// (lsm_batch.cu), compiled for the host too by the tests: roots, quotients and
// conversions, the WENO3 reconstruction, the FP64 combination of an FP32 stage.
#pragma once

#include <cuda_runtime.h>

#include "lsm_soft64.cuh"

namespace lsm {
namespace batch {
namespace {

// ------------------------------------------------------------ scalar helpers
// 1 / (a sum of smoothness weights, at least 3e-12): FP32 by the hardware's
// approximation without the general quotient's care for subnormal divisors,
// FP64 on the integer pipes
template <typename T> __device__ __forceinline__ T wrcp(T b) { return sdiv(1.0, b); }
template <> __device__ __forceinline__ float wrcp<float>(float b) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    return r;
#else
    return 1.0f / b;
#endif
}
// a weight over such a sum: FP32 by that reciprocal, FP64 rounded once
template <typename T> __device__ __forceinline__ T wquo(T a, T b) { return sdiv(a, b); }
template <> __device__ __forceinline__ float wquo<float>(float a, float b) { return a * wrcp(b); }
template <typename T> __device__ __forceinline__ T vfma(T a, T b, T c) { return fma(a, b, c); }
template <> __device__ __forceinline__ float vfma<float>(float a, float b, float c) { return fmaf(a, b, c); }
// (FP64 on the integer pipes: the same bits)
template <typename T> __device__ __forceinline__ T vsqrt(T a) { return ssqrt(a); }
template <> __device__ __forceinline__ float vsqrt<float>(float a) { return sqrtf(a); }
template <typename T> __device__ __forceinline__ T vrsqrt(T a) { return sdiv(1.0, ssqrt(a)); }
template <> __device__ __forceinline__ float vrsqrt<float>(float a) { return rsqrtf(a); }
template <typename T> __device__ __forceinline__ T vsin(T a) { return sin(a); }
template <> __device__ __forceinline__ float vsin<float>(float a) { return sinf(a); }
template <typename T> __device__ __forceinline__ bool vfinite(T a) { return isfinite(a); }
// ------------------------------------------------------------ WENO3
// GetWENO3Reconstruction (src/AdvectionMethods.F90:195-245) on an oriented
// stencil (fL, fC, fR): weights 2/3, 1/3 over (beta + 1e-6)^2, rearranged to
// one division: w0 = 2 t1^2 / (2 t1^2 + t0^2), Phi = u1 + w0 (u0 - u1).
// Every operation's rounding is fixed here: all forms of a stage agree.
template <typename T>
__device__ __forceinline__ T rec3_value(T fL, T fC, T g, T w0) {
    return vfma(w0, g, vfma(T(1.5), fC, T(-0.5) * fL));
}
template <typename T>
__device__ __forceinline__ T rec3(T fL, T fC, T fR) {
    const T eL = fL - fC, eR = fC - fR;
    const T t0 = vfma(eR, eR, T(1.0e-6)), t1 = vfma(eL, eL, T(1.0e-6));
    const T a0 = (t1 + t1) * t1;
    return rec3_value(fL, fC, vfma(T(0.5), fL + fR, -fC), wquo(a0, vfma(t0, t0, a0)));
}

// Phi_{+1/2} - Phi_{-1/2} along one axis for the node with stencil
// (m2, m1, c, p1, p2); lo/hi force the reference's one-sided stencils on
// the first / last interior node (calc_RH_AD_WENO3.F90:201-245).
template <typename T>
__device__ __forceinline__ T weno_diff(T m2, T m1, T c, T p1, T p2, T w, bool lo, bool hi) {
    // the stencils are selected first so that each face costs one
    // reconstruction (no evaluation of the branch not taken)
    const bool up = w > T(0);
    const bool P = up || hi, M = up && !lo;
    const T fp = rec3(P ? m1 : p2, P ? c : p1, P ? p1 : c);
    const T fm = rec3(M ? m2 : p1, M ? m1 : c, M ? c : m1);
    return fp - fm;
}

// sgn(w) (Phi_{+1/2} - Phi_{-1/2}), weno_diff's bits: q0, q1, q3 are the
// neighbours two and one against the wind and one along it.  The faces share
// a difference and its smoothness.  `edge`: the first (wind up) or last (wind
// down) interior node, whose upwind face takes the stencil (q3, c, q1) instead
// of (q0, q1, c).
template <typename T>
__device__ __forceinline__ T weno_wind(T q0, T q1, T c, T q3, bool edge) {
    const T fL = edge ? q3 : q0, fC = edge ? c : q1, fR = edge ? q1 : c;
    const T e0 = fL - fC, e1 = q1 - c, e2 = c - q3;   // (fC - fR)^2 is e1^2
    const T t0 = vfma(e0, e0, T(1.0e-6)), t1 = vfma(e1, e1, T(1.0e-6)), t2 = vfma(e2, e2, T(1.0e-6));
    const T au = (t0 + t0) * t0, ad = (t1 + t1) * t1;
    const T wu = wquo(au, vfma(t1, t1, au)), wd = wquo(ad, vfma(t2, t2, ad));
    return rec3_value(q1, c, vfma(T(0.5), q1 + q3, -c), wd) - rec3_value(fL, fC, vfma(T(0.5), fL + fR, -fC), wu);
}

// (double)f and (float)d on the integer pipes (a conversion takes the FP64
// pipe as long as a product): exact / rounded to nearest even for 0 and
// normal values whose result is 0 or normal; `ok` is cleared otherwise
__device__ __forceinline__ double widen(float f, bool& ok) {
    const unsigned u = __float_as_uint(f), m = u & 0x7FFFFFFFu;
    ok = ok && (m - 0x00800000u < 0x7F000000u || m == 0u);
    return __hiloint2double((int)((u & 0x80000000u) | (m ? (m >> 3) + 0x38000000u : 0u)), (int)(u << 29));
}
__device__ __forceinline__ float narrow(double d, bool& ok) {
    const unsigned h = (unsigned)__double2hiint(d), l = (unsigned)__double2loint(d), m = h & 0x7FFFFFFFu;
    const unsigned q = ((m - 0x38000000u) << 3) | (l >> 29), r = l << 3;   // truncated, rest
    ok = ok && m - 0x38100000u < 0x0FD00000u;
    return __uint_as_float((h & 0x80000000u) | (q + ((r > 0x80000000u || (r == 0x80000000u && (q & 1u))) ? 1u : 0u)));
}
__device__ __noinline__ float stage_band_any(double W0, double W1, double W2, float D0, float D1, float D2, float c1,
                                             float c2, float c3, float pn, float w2) {
    const double r = W0 * (double)D0 + W1 * (double)D1 + W2 * (double)D2;
    return (float)((double)c1 * (double)pn + (double)c2 * (double)w2 - (double)c3 * r);
}
// The stage in FP64 over the FP32 differences: six operations of the FP64
// pipe instead of fifteen.  A call, so that only the warps with such a node
// pay for it (inlined, its operations were predicated, and predicated-off
// operations occupy the FP64 pipe of every warp: 56 % of the stage's time on
// 64 grids of 32..96 nodes an axis).
__device__ __noinline__ float stage_band(double W0, double W1, double W2, float D0, float D1, float D2, float c1,
                                         float c2, float c3, float pn, float w2) {
    bool ok = true;
    const double d0 = widen(D0, ok), d1 = widen(D1, ok), d2 = widen(D2, ok);
    const double p = widen(pn, ok), w = widen(w2, ok), a = widen(c1, ok), b = widen(c2, ok), c = widen(c3, ok);
    const double r = W0 * d0 + W1 * d1 + W2 * d2;
    const float v = narrow(a * p + b * w - c * r, ok);
    return ok ? v : stage_band_any(W0, W1, W2, D0, D1, D2, c1, c2, c3, pn, w2);
}

}  // namespace
}  // namespace batch
}  // namespace lsm
