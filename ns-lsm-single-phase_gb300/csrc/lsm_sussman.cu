// lsm_sussman.cu -- the reference's live reinitialisation,
// reinitialisation_test2 (src/reinitialisation_test2.F90:1-221), and its
// gradient norm calc_NormGrad_d (src/calc_NormGrad_d.F90:1-2448), in FP64
// with the reference's operation order (built with --fmad=false).
//
// calc_NormGrad_d's 27 blocks (interior, 6 faces, 12 edges, 8 corners)
// reduce to one choice per direction and node: a one-sided BiasedDerivative
// (src/AdvectionMethods.F90:248-302, ENO2Boundary :654-707) along a
// direction whose face is physical at the node, GetENO2Reconstruction
// (src/AdvectionMethods.F90:63-191) otherwise, with the stencil clipped on
// the node next to a physical face.  One thread per node; ghost nodes get 0.
//
// Bound by the FP64 pipe: comparisons, products and the root run on the
// integer pipes (lsm_soft64.cuh), bit for bit; what an inlined FP64 fallback
// would cost by predication goes through calls.
// The two i-face blocks never assign phi0, so their ENO2 stencil choice
// uses phizero at the last node of the interior loop (`stale`).
#include <cuda_runtime.h>

#include "lsm_common.cuh"
#include "lsm_kernels.h"
#include "lsm_soft64.cuh"

namespace lsm {
namespace {

inline unsigned nblocks(long long n, int t) { return (unsigned)((n + t - 1) / t); }

constexpr int BX = 32, BY = 4, BZ = 2;
constexpr u64 kEpsBits = 0x3CB0000000000000ull, kInfBits = 0x7FF0000000000000ull, kSign = 1ull << 63;

// GetENO2Reconstruction, src/AdvectionMethods.F90:63-191
__device__ __noinline__ double eno2_ieee(double f0, double fLL, double fL, double fC, double fR, double fRR, bool lo, bool hi) {
    double a, b, Mf, dp, dm;
    if (lo) {
        a = fR - (2.0 * fC) + fL;
        b = fRR - (2.0 * fR) + fC;
        Mf = a;
        if (fabs(b) < fabs(a)) Mf = b;
        dp = fR - fC - 0.5 * Mf;
        Mf = a;
        dm = fC - fL + 0.5 * Mf;
    } else if (hi) {
        a = fR - (2.0 * fC) + fL;
        Mf = a;
        dp = fR - fC - 0.5 * Mf;
        b = fC - (2.0 * fL) + fLL;
        if (fabs(b) < fabs(a)) Mf = b;
        dm = fC - fL + 0.5 * Mf;
    } else {
        a = fR - (2.0 * fC) + fL;
        b = fRR - (2.0 * fR) + fC;
        Mf = a;
        if (fabs(b) < fabs(a)) Mf = b;
        dp = fR - fC - 0.5 * Mf;
        b = fC - (2.0 * fL) + fLL;
        Mf = a;
        if (fabs(b) < fabs(a)) Mf = b;
        dm = fC - fL + 0.5 * Mf;
    }
    const double sg = fabs(f0) > kEpsSims ? (f0 >= 0.0 ? 1.0 : -1.0) : 0.0;
    if (sg * (fR - fC) < 0.0 && sg * (fC - fL) < -sg * (fR - fC)) return dp;
    if (sg * (fC - fL) > 0.0 && sg * (fR - fC) > -sg * (fC - fL)) return dm;
    return 0.5 * (dp + dm);
}

// ENO2Boundary, src/AdvectionMethods.F90:654-707
__device__ double eno2_boundary(double f0, double f1, double f2, int bias) {
    const double as = (double)bias;
    const double D1 = as * (f1 - f0), D2 = as * (f2 - f1), D3 = as * (f2 - f0) / 2.0;
    if (fabs(D1 - D2) < kEpsSims) return D1;
    if (fabs(D1) < fabs(D2)) return (2.0 * D1 + D2) / 3.0;
    if (fabs(D2) < fabs(D1)) return (D1 + 2.0 * D2) / 3.0;
    if (fabs(D1) == fabs(D2)) return (4.0 * D1 + D2) / 5.0;
    if (fabs(D1) < fabs(D3) && fabs(D2) < fabs(D3)) return (3.0 * D1 + 6.0 * D2 - D3) / 7.0;
    if (fabs(D1) >= fabs(D3) && fabs(D2) >= fabs(D3)) return D3;
    return D1;
}

// BiasedDerivative, src/AdvectionMethods.F90:248-302 (physical faces only)
__device__ __noinline__ double biased(double f0, double f1, double f2, double f3, int order, int bias, bool enobc) {
    const double as = (double)bias;
    if (order == 1) return as * (-1.0 * f0 + 1.0 * f1);
    if (order == 2) {
        if (enobc) return eno2_boundary(f0, f1, f2, bias);
        return as * (-(3.0 * f0) + 4.0 * f1 - 1.0 * f2) / 2.0;
    }
    return as * (-(11.0 * f0) + 18.0 * f1 - 9.0 * f2 + 2.0 * f3) / 6.0;
}

__global__ void sign_phi0_kernel(long long n, const double* __restrict__ phi0, double eps, double* __restrict__ sg) {
    const long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (l >= n) return;
    const double p = phi0[l];
    // GetSignPhi0, src/AdvectionMethods.F90:576-587
    sg[l] = fabs(p) > eps ? (p >= 0.0 ? 1.0 : -1.0) : p / eps - 1.0 / kPi * sin((kPi * p) / eps);
}

// products and sums in calls: rare values in otherwise integer code
__device__ __noinline__ double mul_ieee(double a, double b) { return a * b; }
__device__ __noinline__ double norm_ieee(double c0, double c1, double c2, double c3, double c4, double c5, double c6,
                                         double c7, double c8, double d0, double d1, double d2) {
    const double dx = c0 * d0 + c3 * d1 + c6 * d2;
    const double dy = c1 * d0 + c4 * d1 + c7 * d2;
    const double dz = c2 * d0 + c5 * d1 + c8 * d2;
    return sqrt(dx * dx + dy * dy + dz * dz);
}

// order of finite doubles as signed integers, both zeros equal
__device__ __forceinline__ i64 key(u64 u) {
    return u >> 63 ? (i64)(kSign - u) : (i64)u;
}

// eno2_ieee with its tests on the integer pipes: 11 FP64 operations.  2 f and
// 0.5 M are exact, so fma forms the rounded differences of the written-out
// expression; values of 2^1023 and more and subnormal M take that expression.
__device__ __forceinline__ double eno2(double f0, double fLL, double fL, double fC, double fR, double fRR, bool lo,
                                       bool hi) {
    const double ep = fR - fC, em = fC - fL;
    const double a = fma(-2.0, fC, fR) + fL, b = fma(-2.0, fR, fRR) + fC, c = fma(-2.0, fL, fC) + fLL;
    const double Mp = !hi && mag(b) < mag(a) ? b : a, Mm = !lo && mag(c) < mag(a) ? c : a;
    const u64 big = 0x7FE0000000000000ull;
    auto half_exact = [](double v) { return biased_exp(v) >= 2u || mag(v) == 0u; };
    if (mag(fLL) >= big || mag(fL) >= big || mag(fC) >= big || mag(fR) >= big || mag(fRR) >= big ||
        !half_exact(Mp) || !half_exact(Mm))
        return eno2_ieee(f0, fLL, fL, fC, fR, fRR, lo, hi);
    const double dp = fma(-0.5, Mp, ep), dm = fma(0.5, Mm, em);
    const double avg = half_of(dp + dm);
    // p, q: sg (fR - fC), sg (fC - fL); none for a zero sign
    const u64 sg = d2u(f0) & kSign;
    const bool some = mag(f0) > kEpsBits && mag(f0) <= kInfBits;
    const u64 p = d2u(ep) ^ sg, q = d2u(em) ^ sg;
    if (some && key(p) < 0 && key(q) < key(p ^ kSign)) return dp;
    if (some && key(q) > 0 && key(p) > key(q ^ kSign)) return dm;
    return avg;
}

// |grad phi| of one non-ghost node, src/calc_NormGrad_d.F90
__device__ __forceinline__ double norm_grad(const DevGrid& g, int order, int enobc, const double* __restrict__ phi,
                                            const double* __restrict__ phizero, long long stale,
                                            const double* __restrict__ csi, const double* __restrict__ eta,
                                            const double* __restrict__ zet, long long l, int i, int j, int k) {
    const int c[3] = {i, j, k};
    const int lo[3] = {g.ia, g.ja, g.ka}, hi[3] = {g.ib, g.jb, g.kb};
    const int plo[3] = {g.pb, g.pl, g.pd}, phy[3] = {g.pf, g.pr, g.pu};
    const long long st[3] = {1, g.sj, g.sk};
    const double dd[3] = {g.dc, g.de, g.dz};
    const bool iface = (g.pb && i == g.ia) || (g.pf && i == g.ib);
    const bool jface = (g.pl && j == g.ja) || (g.pr && j == g.jb);
    const bool kface = (g.pd && k == g.ka) || (g.pu && k == g.kb);
    const double phi0 = (iface && !jface && !kface) ? phizero[stale] : phizero[l];
    double d[3];
    const double fc = phi[l];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        const long long s = st[m];
        if (plo[m] && c[m] == lo[m]) {
            d[m] = biased(fc, phi[l + s], phi[l + 2 * s], phi[l + 3 * s], order, 1, enobc != 0);
        } else if (phy[m] && c[m] == hi[m]) {
            d[m] = biased(fc, phi[l - s], phi[l - 2 * s], phi[l - 3 * s], order, -1, enobc != 0);
        } else {
            // the node next to a physical face clips the stencil (the
            // reference passes a dummy zero instead of the node beyond)
            const bool lob = plo[m] && c[m] == lo[m] + 1, hib = phy[m] && c[m] == hi[m] - 1;
            const double fLL = lob ? 0.0 : phi[l - 2 * s], fRR = hib ? 0.0 : phi[l + 2 * s];
            d[m] = eno2(phi0, fLL, phi[l - s], fc, phi[l + s], fRR, lob, hib);
        }
        if (!g.unit) d[m] = mul_ieee(dd[m], d[m]);
    }
    double M[9];
    // (the range as in godunov_norm)
    auto fits = [](double v) { return biased_exp(v) - 823u < 440u || mag(v) == 0u; };
    bool ok = fits(d[0]) && fits(d[1]) && fits(d[2]);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        M[x] = __ldg(csi + 3 * l + x);
        M[3 + x] = __ldg(eta + 3 * l + x);
        M[6 + x] = __ldg(zet + 3 * l + x);
        ok = ok && fits(M[x]) && fits(M[3 + x]) && fits(M[6 + x]);
    }
    if (!ok) return norm_ieee(M[0], M[1], M[2], M[3], M[4], M[5], M[6], M[7], M[8], d[0], d[1], d[2]);
    double w[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) w[x] = usqr(umul0(M[x], d[0]) + umul0(M[3 + x], d[1]) + umul0(M[6 + x], d[2]));
    return ssqrt(w[0] + w[1] + w[2]);
}

__global__ void __launch_bounds__(256, 4) normgrad_d_kernel(DevGrid g, int order, int enobc,
        const double* __restrict__ phi, const double* __restrict__ phizero, long long stale,
        const double* __restrict__ csi, const double* __restrict__ eta, const double* __restrict__ zet,
        double* __restrict__ out) {
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y,
              k = blockIdx.z * BZ + threadIdx.z;
    if (i >= g.ni || j >= g.nj || k >= g.nk) return;
    const long long l = gid(g, i, j, k);
    const bool ghost = i < g.ia || i > g.ib || j < g.ja || j > g.jb || k < g.ka || k > g.kb;
    // ghost node: 0 (NormGrad_RN = zero)
    out[l] = ghost ? 0.0 : norm_grad(g, order, enobc, phi, phizero, stale, csi, eta, zet, l, i, j, k);
}

// The RK update of one moving node (src/reinitialisation_test2.F90:140-168)
// with GetLambdaMassCorrection (src/global_lsm.F90:200-219) and deltaf
// (src/global_lsm.F90:120-133; i2e = 1 / (2 eps)), inside the delta
// function's support or where G is not finite
__device__ __noinline__ double suss_rhs_near(double s, double G, double d1, double eps, double i2e) {
    const double rhs = s * (G - 1.0);
    const double df = fabs(d1) > eps ? 0.0 : i2e * (1.0 + cos(sdiv(kPi * d1, eps)));
    const double num = -df * s * (1.0 - G);
    const double den = (df * df) * G;
    const double lam = fabs(den) < kEpsSims ? 0.0 : sdiv(num, den);
    return rhs - lam * (df * G);
}

// One RK stage of reinitialisation_test2, |grad d| and update fused:
//   stage 1: d = dn; keeps which nodes move (|grad dn| - 1 > epsr); writes A
//   stage 2: d = A; writes B
//   stage 3: d = B; writes dn in place (only a node's own dn is read)
// The reference forms |grad dn| twice per iteration (for the mask and for
// stage 1: the same values) and copies dn1 to dn; with the gradients, the
// updates, the copies and the extrema in passes of their own an iteration
// took nine launches and a wait for the host.  Now it is three launches:
// `mm` (maximum, minimum of |grad d| over all nodes, as integers: the values
// are not negative; exact in any order) of the iteration's start is tested
// by every block, which leaves its output alone once it has converged, and
// stage 3 (and stage 1 of the first iteration) accumulates the next one.
// 192 x 96 x 72 nodes: 1.51 ms an iteration before, 0.45 ms now, the FP64
// pipe busy for 76 % of stage 2's time (27 operations a node).
struct SussArgs {
    const double *dn, *d;
    double* out;
    const double *sg, *phizero, *csi, *eta, *zet;
    unsigned char* move;
    long long stale;
    int order, enobc;
    double eps, i2e, epsr, c1, c2, c3dt;
    const u64* mm;   // extrema that decide whether the iteration runs (nullptr: it runs)
    u64* next;       // extrema to accumulate (nullptr: none)
};

__device__ __forceinline__ bool converged(const u64* mm, double epsr) {
    return fabs(u2d(mm[0]) - 1.0) < epsr && fabs(u2d(mm[1]) - 1.0) < epsr;
}

template <int STAGE>
__global__ void __launch_bounds__(256, 4) sussman_stage_kernel(DevGrid g, SussArgs a) {
    __shared__ int done;
    __shared__ u64 smax[8], smin[8];
    const int t = threadIdx.x + BX * (threadIdx.y + BY * threadIdx.z), lane = t & 31, w = t >> 5;
    if (a.mm) {
        if (t == 0) done = converged(a.mm, a.epsr) ? 1 : 0;
        __syncthreads();
        if (done) {
            // the extrema of a converged iteration stand for the rest
            if (a.next && t == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
                a.next[0] = a.mm[0];
                a.next[1] = a.mm[1];
            }
            return;
        }
    }
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y,
              k = blockIdx.z * BZ + threadIdx.z;
    const bool in = i < g.ni && j < g.nj && k < g.nk;
    u64 hi = 0u, lo = 0x7FE1CCF385EBC8A0ull;   // 0 and 1e308
    if (in) {
        const long long l = gid(g, i, j, k);
        const bool ghost = i < g.ia || i > g.ib || j < g.ja || j > g.jb || k < g.ka || k > g.kb;
        const double d1 = a.d[l];
        double r = d1, G = 0.0;
        bool mv = STAGE > 1 ? a.move[l] != 0 : true;
        if (!ghost && (STAGE != 2 || mv)) {
            G = norm_grad(g, a.order, a.enobc, a.d, a.phizero, a.stale, a.csi, a.eta, a.zet, l, i, j, k);
            const double G1 = G - 1.0;
            if (STAGE == 1) mv = G1 > a.epsr;
            if (mv) {
                const double s = a.sg[l];
                double rhs;
                if (mag(s) == 0x3FF0000000000000ull && mag(d1) > mag(a.eps) && finite64(d1) && finite64(G))
                    rhs = u2d(d2u(G1) ^ (d2u(s) & kSign));
                else
                    rhs = suss_rhs_near(s, G, d1, a.eps, a.i2e);
                // stage 1: 1 dn + 0 d = dn exactly
                if (STAGE == 1 && finite64(d1)) r = d1 - a.c3dt * rhs;
                else r = a.c1 * a.dn[l] + a.c2 * d1 - a.c3dt * rhs;
            }
        }
        if (STAGE == 1) a.move[l] = !ghost && mv ? 1 : 0;
        if (STAGE == 3 ? mv && !ghost : true) a.out[l] = r;
        if (mag(G) <= kInfBits) hi = lo = mag(G);   // NaN: neither
    }
    if (a.next) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const u64 x = __shfl_xor_sync(0xffffffffu, hi, o), y = __shfl_xor_sync(0xffffffffu, lo, o);
            hi = x > hi ? x : hi;
            lo = y < lo ? y : lo;
        }
        if (lane == 0) { smax[w] = hi; smin[w] = lo; }
        __syncthreads();
        if (t == 0) {
            for (int q = 1; q < 8; ++q) {
                hi = smax[q] > hi ? smax[q] : hi;
                lo = smin[q] < lo ? smin[q] : lo;
            }
            atomicMax(reinterpret_cast<unsigned long long*>(a.next), (unsigned long long)hi);
            atomicMin(reinterpret_cast<unsigned long long*>(a.next) + 1, (unsigned long long)lo);
        }
    }
}

// n pairs of extrema: the first as `from` has it, the others of no value yet
__global__ void suss_init_kernel(u64* mm, int n, const u64* from) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) {
        mm[2 * q] = q == 0 && from ? from[0] : 0u;
        mm[2 * q + 1] = q == 0 && from ? from[1] : 0x7FE1CCF385EBC8A0ull;
    }
}

}  // namespace

void launch_sign_phi0(long long n, const double* phi0, double eps, double* sg, cudaStream_t s) {
    ProfScope ps("sign_phi0_kernel", s);
    sign_phi0_kernel<<<nblocks(n, 256), 256, 0, s>>>(n, phi0, eps, sg);
}

void launch_normgrad_d(const DevGrid& g, int order, int enobc, const double* phi, const double* phizero,
                       long long stale, const double* csi, const double* eta, const double* zet, double* out,
                       cudaStream_t s) {
    ProfScope ps("normgrad_d_kernel", s);
    normgrad_d_kernel<<<dim3((g.ni + BX - 1) / BX, (g.nj + BY - 1) / BY, (g.nk + BZ - 1) / BZ), dim3(BX, BY, BZ), 0,
                        s>>>(g, order, enobc, phi, phizero, stale, csi, eta, zet, out);
}

// `iters` iterations of reinitialisation_test2 on d (in place; A, B and move:
// scratch fields); mm: iters + 1 pairs, the extrema at the start of each
// iteration (the host counts those that had not converged).  from: the
// extrema at the start of the first, of iterations run before (nullptr: it is
// the first of all)
void launch_sussman(const DevGrid& g, int order, int enobc, int iters, double* d, double* A, double* B,
                    unsigned char* move, const double* sg, const double* phizero, long long stale, const double* csi,
                    const double* eta, const double* zet, double eps, double epsr, double dt, unsigned long long* mm,
                    const unsigned long long* from, cudaStream_t s) {
    const dim3 grid((g.ni + BX - 1) / BX, (g.nj + BY - 1) / BY, (g.nk + BZ - 1) / BZ), block(BX, BY, BZ);
    const double C[3][3] = {{1.0, 0.0, 1.0}, {3.0 / 4.0, 1.0 / 4.0, 1.0 / 4.0}, {1.0 / 3.0, 2.0 / 3.0, 2.0 / 3.0}};
    u64* m = reinterpret_cast<u64*>(mm);
    {
        ProfScope ps("suss_init_kernel", s);
        suss_init_kernel<<<(iters + 256) / 256, 256, 0, s>>>(m, iters + 1, reinterpret_cast<const u64*>(from));
    }
    for (int it = 0; it < iters; ++it) {
        SussArgs a{d, d, A, sg, phizero, csi, eta, zet, move, stale, order, enobc, eps, 1.0 / (2.0 * eps), epsr, 0.0, 0.0,
                   0.0, nullptr, nullptr};
        auto stage = [&](int q, const double* in, double* out, const u64* mm_in, u64* next) {
            a.d = in;
            a.out = out;
            a.c1 = C[q][0];
            a.c2 = C[q][1];
            a.c3dt = C[q][2] * dt;
            a.mm = mm_in;
            a.next = next;
            ProfScope ps("sussman_stage_kernel", s);
            if (q == 0) sussman_stage_kernel<1><<<grid, block, 0, s>>>(g, a);
            else if (q == 1) sussman_stage_kernel<2><<<grid, block, 0, s>>>(g, a);
            else sussman_stage_kernel<3><<<grid, block, 0, s>>>(g, a);
        };
        // the first iteration's extrema are those of its own stage 1
        const bool own = it == 0 && !from;
        stage(0, d, A, own ? nullptr : m + 2 * it, own ? m : nullptr);
        stage(1, A, B, m + 2 * it, nullptr);
        stage(2, B, d, m + 2 * it, m + 2 * (it + 1));
    }
}

}  // namespace lsm
