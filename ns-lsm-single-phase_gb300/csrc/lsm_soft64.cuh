// lsm_soft64.cuh -- FP64 division, square root and comparisons on the
// integer pipes, bit for bit the IEEE 754 results (round to nearest even).
//
// What bounds the FP64 kernels on GB300 is the FP64 pipe: a multiply or add
// takes it 16 clocks per warp and SM by its two lanes (19 measured with 32
// warps per SM), and a division or square root through CUDA's operators 143
// (measured), while an integer
// multiply-add with a 64-bit result takes its pipe 1.3 and a shift, add or
// logical operation 0.3-0.5.  So quotients and roots are formed here in
// 64-bit fixed point, beside the FP64 pipe's work.
//
// Method (Newton-Raphson on the reciprocal, then the exact remainder:
// Muller et al., Handbook of Floating-Point Arithmetic, 2nd ed., sections
// 4.7 and 5.3): a 23-bit seed from the FP32 reciprocal or reciprocal root,
// one Newton step in fixed point to 44 bits, the truncated quotient
// Q0 = A R, its exact remainder A 2^k - Q0 B (64 bits suffice: Q0 is at most
// 2^9 short), one more digit from the remainder, and the rounding decided
// by the final remainder.  A quotient or root of two 53-bit significands
// never lies half-way between two 53-bit numbers, so the comparison is
// strict.  Operands or results outside the normal range (zeros, subnormals,
// infinities, NaN) take CUDA's operator.
//
// The seeds may be two units in the last place from the correctly rounded
// ones (with three some roots come out wrong, with four some quotients): the
// tests move them by as many on the CPU and compare every argument that they
// can get on the device.
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#include <cuda_runtime.h>
#define LSM_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define LSM_HD inline
#endif

namespace lsm {

using u32 = std::uint32_t;
using u64 = std::uint64_t;
using i64 = std::int64_t;

// (on the device as a move that the optimiser does not see through: it would
// turn tests of the bits into comparisons on the FP64 pipe)
LSM_HD u64 d2u(double x) {
#if defined(__CUDA_ARCH__)
    u64 u;
    asm("mov.b64 %0, %1;" : "=l"(u) : "d"(x));
    return u;
#else
    u64 u;
    std::memcpy(&u, &x, 8);
    return u;
#endif
}
LSM_HD double u2d(u64 u) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double x;
    std::memcpy(&x, &u, 8);
    return x;
#endif
}
LSM_HD u64 mulhi64(u64 a, u64 b) {
#if defined(__CUDA_ARCH__)
    return __umul64hi(a, b);
#else
    return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}
LSM_HD u32 mulhi32(u32 a, u32 b) {
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return (u32)(((u64)a * b) >> 32);
#endif
}

// FP32 seeds.  On the host `soft64_seed_ulps` moves them by that many units
// in the last place (the tests' stand-in for the approximate instructions).
#if !defined(__CUDA_ARCH__)
inline int& soft64_seed_ulps() {
    static thread_local int u = 0;
    return u;
}
#endif
LSM_HD u32 rcp_bits(u32 fbits) {
#if defined(__CUDA_ARCH__)
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(fbits)));
    return __float_as_uint(y);
#else
    float x, y;
    std::memcpy(&x, &fbits, 4);
    y = 1.0f / x;
    u32 r;
    std::memcpy(&r, &y, 4);
    return r + (u32)soft64_seed_ulps();
#endif
}
LSM_HD u32 rsqrt_bits(u32 fbits) {
#if defined(__CUDA_ARCH__)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(fbits)));
    return __float_as_uint(y);
#else
    float x, y;
    std::memcpy(&x, &fbits, 4);
    y = (float)(1.0 / std::sqrt((double)x));
    u32 r;
    std::memcpy(&r, &y, 4);
    return r + (u32)soft64_seed_ulps();
#endif
}

// the FP32 number with the bits y, taken into [1/2, 1), times 2^32
LSM_HD u32 seed_fix(u32 y) {
    y = y < 0x3F7FFFFFu ? y : 0x3F7FFFFFu;
    return (y > 0x3F000000u ? y << 8 : 0u) | 0x80000000u;
}

constexpr u64 kFrac = 0x000FFFFFFFFFFFFFull, kOne52 = 0x0010000000000000ull;

LSM_HD u32 biased_exp(double x) { return (u32)(d2u(x) >> 52) & 0x7FFu; }
// finite, and neither zero nor subnormal
LSM_HD bool is_normal(u32 e) { return e - 1u < 0x7FEu; }

// x > 0 and x < 0 (false for NaN)
LSM_HD bool gt0(double x) { return d2u(x) - 1u < 0x7FF0000000000000ull; }
LSM_HD bool lt0(double x) { return d2u(x) - 0x8000000000000001ull < 0x7FF0000000000000ull; }
// |x| as an integer in the order of the magnitudes
LSM_HD u64 mag(double x) { return d2u(x) & 0x7FFFFFFFFFFFFFFFull; }
LSM_HD bool finite64(double x) { return mag(x) < 0x7FF0000000000000ull; }
// 0.5 x
LSM_HD double half_of(double x) {
    const u32 e = biased_exp(x);
    if (e - 2u < 0x7FDu) return u2d(d2u(x) - kOne52);
    return 0.5 * x;
}
LSM_HD u64 sig53(u64 u) { return (u & kFrac) | kOne52; }

// Rounds hi 2^64 + lo (51 or 52 fraction bits in hi, the rest in lo) to 53
// bits, to nearest even; e is the biased exponent of hi = 2^51, sign the
// sign bit in place
LSM_HD double round_product(unsigned __int128 p, u32 e, u64 sign) {
    u64 hi = (u64)(p >> 64), lo = (u64)p;
    const u32 s = hi < kOne52 ? 1u : 0u;
    if (s) {
        hi = hi << 1 | lo >> 63;
        lo <<= 1;
    }
    const u32 lh = (u32)(lo >> 32);
    const u64 up = (lh >> 31) && ((lh << 1) | (u32)lo | ((u32)hi & 1u)) ? 1u : 0u;
    return u2d(sign | (((u64)(e - s) << 52) + hi + up));
}

// a b for normal a and b whose product stays inside the normal range: the
// exact 106-bit product rounded once
LSM_HD double umul(double a, double b) {
    const u64 ua = d2u(a), ub = d2u(b);
    const unsigned __int128 p = (unsigned __int128)(sig53(ua) << 11) * sig53(ub);
    return round_product(p, biased_exp(a) + biased_exp(b) - 1023u, (ua ^ ub) & (1ull << 63));
}
// the same where a or b may also be a zero
LSM_HD double umul0(double a, double b) {
    const double p = umul(a, b);
    return mag(a) == 0u || mag(b) == 0u ? u2d((d2u(a) ^ d2u(b)) & (1ull << 63)) : p;
}
// a a for 2^-500 <= |a| < 2^500; smaller |a| give 0
LSM_HD double usqr(double a) {
    const u32 e = biased_exp(a);
    const u64 m = sig53(d2u(a));
    const double p = round_product((unsigned __int128)(m << 11) * m, 2u * e - 1023u, 0u);
    return e < 523u ? 0.0 : p;
}

// Reciprocal of a significand mb (2^52 <= mb < 2^53) in fixed point: the
// returned R satisfies R <= 2^64 / b and R >= 2^64 / b (1 - 2^-44), b = mb /
// 2^52 in [1, 2).
LSM_HD u64 recip_fix(u64 mb) {
    const u64 B = mb << 11;
    const u32 Bh = (u32)(B >> 32), Bl = (u32)B;
    // b rounded to 24 bits as FP32 (2.0 when it rounds up to it)
    const u32 y = rcp_bits((Bh >> 8) + ((Bh >> 7) & 1u) + 0x3F000000u);
    // 2^32 / b in 32 bits
    const u32 R0 = seed_fix(y);
    // E / 2^63 = 1 - b r0, |E| < 2^42
    const i64 E = (i64)((1ull << 63) - ((u64)R0 * Bh + (((u64)R0 * Bl) >> 32)));
    // r0 (1 + E / 2^63) on 64 bits (R0 is even: half of it is a signed factor)
    const i64 c = ((i64)(std::int32_t)(R0 >> 1) * (std::int32_t)(E >> 11)) >> 19;
    return ((u64)R0 << 32) + (u64)c - 2u;
}

// RN(ma / mb) with R = recip_fix(mb); `e` is the biased exponent difference
// ea - eb + 1023, `sign` the sign bit in place
LSM_HD double quotient(u64 ma, u64 mb, u64 R, u32 e, u64 sign) {
    const u32 s = ma < mb ? 1u : 0u;              // quotient in [2^52, 2^53) after a shift by 52 + s
    const u64 A = ma << s;
    const u64 Q0 = mulhi64(A << 10, R) >> 10;     // at most 2^9 below floor(A 2^52 / mb)
    const u64 rem = (A << 52) - Q0 * mb;          // exact: 0 <= rem < 2^62
    const u32 d = mulhi32((u32)(rem >> 32), (u32)(R >> 32)) >> 20;
    const u64 r = 2u * (rem - (u64)d * mb);       // twice the remainder of Q0 + d, below 4 mb
    const u64 Q = Q0 + d + (r > mb ? 1u : 0u) + (r > 3u * mb ? 1u : 0u);
    return u2d(sign | (((u64)(e - s - 1u) << 52) + Q));
}

// a / b for normal a and b with a normal quotient
LSM_HD double udiv(double a, double b) {
    const u64 ua = d2u(a), ub = d2u(b), mb = sig53(ub);
    return quotient(sig53(ua), mb, recip_fix(mb), biased_exp(a) - biased_exp(b) + 1023u, (ua ^ ub) & (1ull << 63));
}
// a / b
LSM_HD double sdiv(double a, double b) {
    const u32 ea = biased_exp(a), eb = biased_exp(b);
    if (!(is_normal(ea) && is_normal(eb) && ea - eb + 1021u < 2043u)) return a / b;
    return udiv(a, b);
}
// a / c and b / c, as udiv
LSM_HD void udiv2(double a, double b, double c, double* qa, double* qb) {
    const u64 ua = d2u(a), ub = d2u(b), uc = d2u(c), mc = sig53(uc), R = recip_fix(mc);
    const u32 ec = 1023u - biased_exp(c);
    *qa = quotient(sig53(ua), mc, R, biased_exp(a) + ec, (ua ^ uc) & (1ull << 63));
    *qb = quotient(sig53(ub), mc, R, biased_exp(b) + ec, (ub ^ uc) & (1ull << 63));
}

// sqrt(a)
LSM_HD double ssqrt(double a) {
    const u64 ua = d2u(a);
    const u32 ea = (u32)(ua >> 52);   // with the sign: negative numbers are not normal here
    if (!is_normal(ea)) return ua << 1 == 0u ? a : sqrt(a);
    // a = m 2^(2 h), m in [1, 4): M = m 2^62 on 64 bits
    const u32 odd = (ea & 1u) ^ 1u;   // biased 1023 is even an exponent of 0
    const u64 sig = (ua & kFrac) | kOne52;
    const u64 M = sig << (10u + odd);
    // m rounded to 24 bits as FP32: [1, 2) has the exponent field 127, [2, 4) 128
    const u32 t = (u32)(sig >> 28);
    const u32 fb = (t >> 1) + (t & 1u) + (odd ? 0x3F800000u : 0x3F000000u);
    // 2^32 / sqrt(m)
    const u32 R0 = seed_fix(rsqrt_bits(fb));
    // E / 2^63 = 1 - m r0^2, |E| < 2^43
    const u64 P = (u64)R0 * R0;                                   // r0^2 2^64
    const u64 G = mulhi64(M, P);                                  // m r0^2 2^62
    const i64 E = (i64)((1ull << 62) - G) * 2;
    // r1 = r0 (1 + (e + 3/4 e^2) / 2) for e = E / 2^63 = Eh / 2^51
    const std::int32_t Eh = (std::int32_t)(E >> 12);
    const std::int32_t e2 = (std::int32_t)(((i64)Eh * Eh) >> 32);
    const i64 c = ((i64)(std::int32_t)(R0 >> 1) * (Eh + ((3 * e2) >> 21))) >> 19;
    const u64 R = ((u64)R0 << 32) + (u64)c - 4096u;               // <= 2^64 / sqrt(m)
    // S0 <= floor(sqrt(m) 2^52), at most 2^4 below
    const u64 S0 = mulhi64(M, R) >> 10;
    const u64 rem = (M << 42) - S0 * S0;                          // exact: 0 <= rem < 2^58
    // the next digit: rem / (2 S0)
    const u32 d = mulhi32((u32)(rem >> 32), (u32)(R >> 32)) >> 21;
    const u64 r = rem - (u64)d * (2u * S0 + d);
    const u64 S = S0 + d;                                         // S^2 + r = m 2^104, r < 4 S + 4
    // rounds up when r > S (sqrt above S + 1/2), by two when above S + 3/2
    const u64 Sr = S + (r > S ? 1u : 0u) + (r > 3u * S + 2u ? 1u : 0u);
    const u32 h = (ea + 1023u - odd) >> 1;                        // (ea - 1023 - odd) / 2 + 1023
    return u2d(((u64)(h - 1u) << 52) + Sr);
}

}  // namespace lsm
