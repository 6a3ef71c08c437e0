// lsm_fp64.cu -- FP64 kernels of the level-set transport step that keep the
// reference's arithmetic: every expression is evaluated in the Fortran
// source's association order and this translation unit is compiled with
// --fmad=false, so each multiply and add rounds separately as gfortran's
// x86-64 code does.  Division and square root are IEEE-rounded in CUDA FP64;
// sin/cos are CUDA's (a few ulp from glibc's).
//
// Roofline: these kernels are bound by the FP64 pipe of GB300, not by HBM:
// products, quotients, roots and comparisons therefore run on the integer
// pipes where they are many (lsm_soft64.cuh), bit for bit as CUDA's operators.
#include <cuda_runtime.h>

#include "lsm_common.cuh"
#include "lsm_kernels.h"
#include "lsm_soft64.cuh"

namespace lsm {

namespace {

constexpr int BX = 32, BY = 4, BZ = 2;

inline dim3 box_grid(int ni, int nj, int nk) {
    return dim3((ni + BX - 1) / BX, (nj + BY - 1) / BY, (nk + BZ - 1) / BZ);
}

// a b in a call: an inlined product would be predicated, and predicated-off
// operations occupy the FP64 pipe too
__device__ __noinline__ double product_ieee(double a, double b) { return a * b; }

// GetWENO3Reconstruction, src/AdvectionMethods.F90:195-245, on the stencil
// oriented by the upwind choice
__device__ __noinline__ double weno3_ieee(double fL, double fC, double fR) {
    const double d0 = 2.0 / 3.0, d1 = 1.0 / 3.0, epsw = 0.000001;
    const double b0 = (fC - fR) * (fC - fR);
    const double b1 = (fL - fC) * (fL - fC);
    const double t0 = b0 + epsw, t1 = b1 + epsw;
    const double a0 = d0 / (t0 * t0);
    const double a1 = d1 / (t1 * t1);
    const double w0 = a0 / (a0 + a1), w1 = a1 / (a0 + a1);
    const double u0 = 0.5 * fC + 0.5 * fR;
    const double u1 = -0.5 * fL + 1.5 * fC;
    return u0 * w0 + u1 * w1;
}
// The same value with the products, quotients and halvings on the integer
// pipes, beside the 9 operations left to the FP64 pipe: valid while the
// differences stay below 2^60 (t, a and w then lie in 2^-20 .. 2^121,
// 2^-243 .. 2^40 and 2^-300 .. 1; a square below 2^-1000 does not change
// t) and the two candidates u are normal.
__device__ __forceinline__ double weno3(double fL, double fC, double fR) {
    const double d0 = 2.0 / 3.0, d1 = 1.0 / 3.0, epsw = 0.000001;
    const double eR = fC - fR, eL = fL - fC;
    const double t0 = usqr(eR) + epsw, t1 = usqr(eL) + epsw;
    const double a0 = udiv(d0, usqr(t0));
    const double a1 = udiv(d1, usqr(t1));
    double w0, w1;
    udiv2(a0, a1, a0 + a1, &w0, &w1);
    const double s0 = fC + fR;
    const double u0 = u2d(d2u(s0) - kOne52);   // 0.5 fC + 0.5 fR: halving is exact
    const double u1 = 1.5 * fC - u2d(d2u(fL) - kOne52);
    const bool ok = biased_exp(eR) < 1083u && biased_exp(eL) < 1083u && biased_exp(s0) - 523u < 600u &&
                    biased_exp(u1) - 523u < 600u && biased_exp(fL) - 2u < 1121u;
    if (!ok) return weno3_ieee(fL, fC, fR);
    return umul(u0, w0) + umul(u1, w1);
}

__device__ __forceinline__ bool in_weno_range(const DevGrid& g, int i, int j, int k) {
    return i >= g.ia + g.pb && i <= g.ib - g.pf && j >= g.ja + g.pl && j <= g.jb - g.pr &&
           k >= g.ka + g.pd && k <= g.kb - g.pu;
}

__device__ __forceinline__ bool non_ghost(const DevGrid& g, int i, int j, int k) {
    return i >= g.ia && i <= g.ib && j >= g.ja && j <= g.jb && k >= g.ka && k <= g.kb;
}

// calc_RH_AD (orderAD == 0) for one non-ghost node, src/calc_RH_AD.F90:1-273
__device__ double upwind_rhs_node(const DevGrid& g, const double* __restrict__ phi,
                                  const double* __restrict__ ucn, long long l, int i, int j, int k) {
    const long long st[3] = {1, g.sj, g.sk};
    const double dd[3] = {g.dc, g.de, g.dz};
    const int c[3] = {i, j, k};
    const int plo[3] = {g.pb, g.pl, g.pd}, phs[3] = {g.pf, g.pr, g.pu};
    const int lo[3] = {g.ia, g.ja, g.ka}, hi[3] = {g.ib, g.jb, g.kb};
    double rh = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const long long s = st[d];
        const double U = __ldg(ucn + 3 * l + d);
        const double pc = __ldg(phi + l);
        double val;
        if (plo[d] && c[d] == lo[d]) {
            val = dd[d] * U * (__ldg(phi + l + s) - pc);
        } else if (phs[d] && c[d] == hi[d]) {
            val = dd[d] * U * (pc - __ldg(phi + l - s));
        } else {
            const double ucon = 0.5 * U;
            const double up = ucon + fabs(ucon), um = ucon - fabs(ucon);
            val = dd[d] * (up * (pc - __ldg(phi + l - s)) + um * (__ldg(phi + l + s) - pc));
        }
        rh = d == 0 ? val : val + rh;
    }
    return rh;
}

// ---------------------------------------------------------------- A1 ----
// rhs_contra_j, src/rhs_contra_j.F90:2-53; zero outside the loop range
__global__ void contra_kernel(DevGrid g, const double* __restrict__ q, const double* __restrict__ csi,
                              const double* __restrict__ eta, const double* __restrict__ zet,
                              const double* __restrict__ aj, double* __restrict__ ucn) {
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y,
              k = blockIdx.z * BZ + threadIdx.z;
    if (i >= g.ni || j >= g.nj || k >= g.nk) return;
    const long long l = gid(g, i, j, k);
    const int ista = g.pb ? g.ia : 0, iend = g.pf ? g.ib : g.ni - 1;
    const int jsta = g.pl ? g.ja : 0, jend = g.pr ? g.jb : g.nj - 1;
    const int ksta = g.pd ? g.ka : 0, kend = g.pu ? g.kb : g.nk - 1;
    if (i < ista || i > iend || j < jsta || j > jend || k < ksta || k > kend) {
        ucn[3 * l] = 0.0; ucn[3 * l + 1] = 0.0; ucn[3 * l + 2] = 0.0;
        return;
    }
    const double tmp = sdiv(1.0, aj[l]);
    const double u = q[4 * l + 1], v = q[4 * l + 2], w = q[4 * l + 3];
    ucn[3 * l + 0] = tmp * (csi[3 * l] * u + csi[3 * l + 1] * v + csi[3 * l + 2] * w);
    ucn[3 * l + 1] = tmp * (eta[3 * l] * u + eta[3 * l + 1] * v + eta[3 * l + 2] * w);
    ucn[3 * l + 2] = tmp * (zet[3 * l] * u + zet[3 * l + 1] * v + zet[3 * l + 2] * w);
}

// ------------------------------------------------------------ A2 / A7 ----
__global__ void rh_upwind_kernel(DevGrid g, const double* __restrict__ phi, const double* __restrict__ ucn,
                                 const int* __restrict__ mask, double* __restrict__ rh) {
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y,
              k = blockIdx.z * BZ + threadIdx.z;
    if (i >= g.ni || j >= g.nj || k >= g.nk) return;
    const long long l = gid(g, i, j, k);
    rh[l] = non_ghost(g, i, j, k) && !(mask && mask[l] <= 0) ? upwind_rhs_node(g, phi, ucn, l, i, j, k) : 0.0;
}

// ---------------------------------------------------------------- A4 ----
// One TVD-RK3 stage, src/ad_RKTVD3.F90:53-81, written to `out` (ping-pong):
// out = c1*phin + c2*phi1 - c3*aj*dt*rh on advected non-ghost nodes, phi1
// elsewhere.  rh is 0 on physical-boundary nodes under WENO3.
struct StageArgs {
    const double *phin, *phi1, *ucn, *aj;
    const int* mask;
    double c1, c2, c3, dt;
    int first;   // c1 = 1, c2 = 0, c3 = 1 and phi1 is phin
    double* out;
};

__device__ __forceinline__ double stage_value(const StageArgs& a, long long l, double p1, double rh) {
    // first stage: 1 phin + 0 phi1 = phin and 1 aj = aj, exactly
    if (a.first && finite64(p1)) return p1 - a.aj[l] * a.dt * rh;
    return a.c1 * a.phin[l] + a.c2 * p1 - a.c3 * a.aj[l] * a.dt * rh;
}

__global__ void rk_upwind_kernel(DevGrid g, StageArgs a) {
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y,
              k = blockIdx.z * BZ + threadIdx.z;
    if (i >= g.ni || j >= g.nj || k >= g.nk) return;
    const long long l = gid(g, i, j, k);
    const double p1 = a.phi1[l];
    if (!non_ghost(g, i, j, k) || (a.mask && a.mask[l] <= 0)) { a.out[l] = p1; return; }
    a.out[l] = stage_value(a, l, p1, upwind_rhs_node(g, a.phi1, a.ucn, l, i, j, k));
}

// calc_RH_AD_WENO3 (src/calc_RH_AD_WENO3.F90:132-399) and, with RH false,
// the stage built on it, for the 32 x TY x TZ nodes of a block of NT threads.
//
// The reconstruction of the face between two nodes is the lower node's
// (f+) and the upper node's (f-); both evaluate the same expression on the
// same values whenever they choose the same upwind side.  So a block
// evaluates each face once into shared memory (the choice of the lower
// node where that is advected, else the upper's), then each node takes its
// six faces from there and evaluates for itself only an f- whose stored
// choice is not its own (a sign change of the contravariant velocity).
//
// Bounded by the FP64 pipe (one warp operation in 16 clocks of an SM: 40 of
// them a node, counted on 192 x 96 x 72 nodes; six reconstructions with CUDA's
// divisions took 360) and, nearly as much, by the issue of the integer work
// beside it (62 % and 66 % of the time): 1.81 ms before, 0.33 ms now on 256 x
// 128 x 96 nodes.  A tile of 32 x 8 x 4 evaluates 3.4
// faces a node, 32 x 2 x 2 4.0.
template <int TY, int TZ, int NT, bool RH>
__global__ void __launch_bounds__(NT, 1280 / NT) weno_kernel(DevGrid g, StageArgs a) {
    constexpr int RZ = (TZ + 1) * TY, RY = TZ * (TY + 1), RX = TZ * TY;   // rows of 32 faces per direction
    constexpr int NF = 32 * (RZ + RY + RX) + RX;                          // and the rows' lower x faces
    __shared__ double F[NF];
    __shared__ bool up_of[NF];
    const int t = threadIdx.x, lane = t & 31;
    const int bi = blockIdx.x * 32, bj = blockIdx.y * TY, bk = blockIdx.z * TZ;
    const int c0[3] = {g.ia + g.pb, g.ja + g.pl, g.ka + g.pd}, c1[3] = {g.ib - g.pf, g.jb - g.pr, g.kb - g.pu};
    const int plo[3] = {g.pb, g.pl, g.pd};
    const double* __restrict__ phi = a.phi1;
    const double* __restrict__ ucn = a.ucn;
    const int* __restrict__ mask = a.mask;
    auto advected = [&](int i, int j, int k, long long l) {
        if (!in_weno_range(g, i, j, k)) return false;
        if (!mask) return true;
        const int m = __ldg(mask + l);
        return RH ? m != 0 : m > 0;
    };
    auto rec = [&](long long l, long long s, bool up) {
        return weno3(__ldg(phi + (up ? l - s : l + 2 * s)), __ldg(phi + (up ? l : l + s)),
                     __ldg(phi + (up ? l + s : l)));
    };
    for (int w = t; w < NF; w += NT) {
        int d, i = bi + lane, j = bj, k = bk;   // the face's lower node
        int r = w >> 5;
        if (r < RZ) {
            d = 2; j += r % TY; k += r / TY - 1;
        } else if (r < RZ + RY) {
            r -= RZ; d = 1; j += r % (TY + 1) - 1; k += r / (TY + 1);
        } else if (r < RZ + RY + RX) {
            r -= RZ + RY; d = 0; j += r % TY; k += r / TY;
        } else {
            r = w - 32 * (RZ + RY + RX); d = 0; i = bi - 1; j += r % TY; k += r / TY;
        }
        if (i < 0 || j < 0 || k < 0) continue;
        const long long s = d == 0 ? 1 : (d == 1 ? g.sj : g.sk), l = gid(g, i, j, k);
        const int c = d == 0 ? i : (d == 1 ? j : k);
        const bool last = d == 0 ? g.pf && c == c1[0] : (d == 1 ? g.pr && c == c1[1] : g.pu && c == c1[2]);
        const bool first = d == 0 ? g.pb && c + 1 == c0[0] : (d == 1 ? g.pl && c + 1 == c0[1] : g.pd && c + 1 == c0[2]);
        const bool own = advected(i, j, k, l);
        if (!own && !advected(i + (d == 0), j + (d == 1), k + (d == 2), l + s)) continue;
        const bool pos = gt0(__ldg(ucn + 3 * (own ? l : l + s) + d));
        // the one-sided stencils next to a physical face
        const bool up = own ? pos || last : pos && !first;
        F[w] = rec(l, s, up);
        up_of[w] = up;
    }
    __syncthreads();
    for (int row = t >> 5; row < TY * TZ; row += NT / 32) {
        const int ty = row % TY, tz = row / TY;
        const int i = bi + lane, j = bj + ty, k = bk + tz;
        if (i >= g.ni || j >= g.nj || k >= g.nk) continue;
        const long long l = gid(g, i, j, k);
        double rh = 0.0;
        if (advected(i, j, k, l)) {
            const int xr = 32 * (RZ + RY + row);
            const int lo[3] = {lane ? xr + lane - 1 : 32 * (RZ + RY + RX) + row, 32 * (RZ + tz * (TY + 1) + ty) + lane,
                               32 * row + lane};
            const int hi[3] = {xr + lane, lo[1] + 32, lo[2] + 32 * TY};
            const int c[3] = {i, j, k};
            const long long st[3] = {1, g.sj, g.sk};
            const double dd[3] = {g.dc, g.de, g.dz};
            double L[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double U = __ldg(ucn + 3 * l + d);
                const bool up = gt0(U) && !(plo[d] && c[d] == c0[d]);
                double fm = F[lo[d]];
                if (up_of[lo[d]] != up) fm = rec(l - st[d], st[d], up);
                const double D = F[hi[d]] - fm;
                L[d] = U * (g.unit ? D : product_ieee(dd[d], D));
            }
            rh = L[0] + L[1] + L[2];
        }
        if (RH) {
            a.out[l] = rh;
        } else {
            const double p1 = phi[l];
            a.out[l] = non_ghost(g, i, j, k) && (!mask || mask[l] > 0) ? stage_value(a, l, p1, rh) : p1;
        }
    }
}

// The largest tile that still fills the GPU: 32 x 8 x 4 from one full wave of
// blocks on (5 on each of 152 SMs), 32 x 4 x 2 from two blocks per SM on,
// 32 x 2 x 2 below.  Measured (stage, 8 x 4 / 4 x 2 / 2 x 2, the event timer's
// overhead included): 256 x 128 x 96 nodes 347 / 381 / 399 us, 128^3 250 / 265 /
// 277, 112^3 199 / 205 / 214, 192 x 96 x 72 165 / 168 / 176, 96^3 126 / 120 /
// 125, 88^3 109 / 103 / 107, 64^3 61 / 46 / 47, 48^3 45 / 33 / 32, 32^3 44 / 18 /
// 17, 16^3 42 / 17 / 16: the lines cost 5 % next to them at most.
template <bool RH>
void launch_weno(const DevGrid& g, const StageArgs& a, cudaStream_t s) {
    auto grid = [&](int ty, int tz) { return dim3((g.ni + 31) / 32, (g.nj + ty - 1) / ty, (g.nk + tz - 1) / tz); };
    auto blocks = [](const dim3& d) { return (long long)d.x * d.y * d.z; };
    if (blocks(grid(8, 4)) >= 5 * 152) weno_kernel<8, 4, 256, RH><<<grid(8, 4), 256, 0, s>>>(g, a);
    else if (blocks(grid(4, 2)) >= 2 * 152) weno_kernel<4, 2, 256, RH><<<grid(4, 2), 256, 0, s>>>(g, a);
    else weno_kernel<2, 2, 128, RH><<<grid(2, 2), 128, 0, s>>>(g, a);
}

// ---------------------------------------------------------------- A5 ----
// bcond_lsm, src/bcond_lsm.F90:2-287.  The six faces are applied in the
// order i1, im, j1, jm, k1, km, each reading the two nodes inward of it as
// left by the faces before it.  A boundary node's final value is therefore a
// fixed function of the pre-BC field ("P0"): per axis whose face rule applies
// to the node, the rule on its values at the two nodes inward along that
// axis, i innermost, then j, then k.  Each thread evaluates that chain for
// one boundary node reading P0 only, so the kernel never reads a node that
// another thread writes.  A node of one face reads two values; the loops
// keep the edge's four and the corner's eight out of its way (written out as
// nested calls, a warp walked all 27 evaluations: 22 us on the smallest
// grids, launch and timer included; 8 us so).
//
// One rule: itpa n1 + itpb n2 with itpa = 4/3 + ex (1 - 4/3), itpb = -1/3 +
// ex (0 + 1/3), ex = 1 where |n2| >= BigPhi: 1 and 0 exactly, else 4/3 and
// -1/3.
__device__ __forceinline__ double bc_rule(const DevBC& bc, int face, double n1, double n2) {
    const int type = bc.type[face];
    if (type == 0) return n1;
    const u64 big = d2u(bc.BigPhi) >> 63 ? 0u : d2u(bc.BigPhi);
    const bool first = mag(n2) >= big;
    const double a = type == 2 ? 2.0 : (first ? 1.0 : 4.0 / 3.0);   // type 2: 2 n1 - n2, only on the im face
    const double b = type == 2 ? -1.0 : (first ? 0.0 : -1.0 / 3.0);
    return a * n1 + b * n2;
}

// direction inward and face of the rule that applies at coordinate c (0: none)
__device__ __forceinline__ int bc_dir(const DevBC& bc, int c, int lo, int hi, int plo, int phs, int face, int* f) {
    auto on = [&](int q) { return bc.type[q] == 0 || bc.type[q] == 1 || (bc.type[q] == 2 && q == 1); };
    if (plo && c == lo && on(face)) { *f = face; return 1; }
    if (phs && c == hi && on(face + 1)) { *f = face + 1; return -1; }
    *f = face;
    return 0;
}

template <class P0>
__device__ __forceinline__ double bc_value(const DevGrid& g, const DevBC& bc, const P0& p0, int i, int j, int k) {
    int fi, fj, fk;
    const int di = bc_dir(bc, i, g.ia, g.ib, g.pb, g.pf, 0, &fi), dj = bc_dir(bc, j, g.ja, g.jb, g.pl, g.pr, 2, &fj),
              dk = bc_dir(bc, k, g.ka, g.kb, g.pd, g.pu, 4, &fk);
    if ((di != 0) + (dj != 0) + (dk != 0) == 1) {   // one face: both values in flight at once
        const double n1 = p0(i + di, j + dj, k + dk), n2 = p0(i + 2 * di, j + 2 * dj, k + 2 * dk);
        return bc_rule(bc, di ? fi : dj ? fj : fk, n1, n2);
    }
    double vk = 0.0;
#pragma unroll 1
    for (int a = 0; a < (dk ? 2 : 1); ++a) {
        double vj = 0.0;
#pragma unroll 1
        for (int b = 0; b < (dj ? 2 : 1); ++b) {
            double vi = 0.0;
#pragma unroll 1
            for (int c = 0; c < (di ? 2 : 1); ++c) {
                const double v = p0(di ? i + di * (c + 1) : i, dj ? j + dj * (b + 1) : j, dk ? k + dk * (a + 1) : k);
                if (c == 0) vi = v;
                else vi = bc_rule(bc, fi, vi, v);
            }
            if (b == 0) vj = vi;
            else vj = bc_rule(bc, fj, vj, vi);
        }
        if (a == 0) vk = vj;
        else vk = bc_rule(bc, fk, vk, vj);
    }
    return vk;
}

__device__ __forceinline__ bool on_phys_face(const DevGrid& g, int i, int j, int k) {
    return (g.pb && i == g.ia) || (g.pf && i == g.ib) || (g.pl && j == g.ja) || (g.pr && j == g.jb) ||
           (g.pd && k == g.ka) || (g.pu && k == g.kb);
}

// P0 inside an RK stage: interior nodes from the stage output, physical-
// boundary nodes recomputed pointwise from the stage inputs.
struct P0Stage {
    DevGrid g;
    int orderAD;
    const double *phin, *phi1, *ucn, *aj, *dst;
    const int* mask;
    double c1, c2, c3, dt;
    __device__ double operator()(int i, int j, int k) const {
        const long long l = gid(g, i, j, k);
        if (!on_phys_face(g, i, j, k)) return dst[l];
        const double p1 = phi1[l];
        if (mask && mask[l] <= 0) return p1;
        const double rh = orderAD == 1 ? 0.0 : upwind_rhs_node(g, phi1, ucn, l, i, j, k);
        return c1 * phin[l] + c2 * p1 - c3 * aj[l] * dt * rh;
    }
};

struct P0Field {
    DevGrid g;
    const double* src;
    __device__ double operator()(int i, int j, int k) const { return src[gid(g, i, j, k)]; }
};

// Boundary nodes of the six face planes (edge nodes appear twice and are
// written twice with the same value).
__device__ __forceinline__ bool face_node(const DevGrid& g, unsigned t, int* pi, int* pj, int* pk) {
    const unsigned Ni = g.ib - g.ia + 1, Nj = g.jb - g.ja + 1, Nk = g.kb - g.ka + 1;
    const unsigned nI = Nj * Nk, nJ = Ni * Nk, nK = Ni * Nj;   // below 2^32 in all, as the nodes are
    if (t < 2 * nI) {
        const bool up = t >= nI;
        if (!(up ? g.pf : g.pb)) return false;
        const unsigned r = up ? t - nI : t;
        *pi = up ? g.ib : g.ia; *pj = g.ja + (int)(r % Nj); *pk = g.ka + (int)(r / Nj);
        return true;
    }
    t -= 2 * nI;
    if (t < 2 * nJ) {
        const bool up = t >= nJ;
        if (!(up ? g.pr : g.pl)) return false;
        const unsigned r = up ? t - nJ : t;
        *pj = up ? g.jb : g.ja; *pi = g.ia + (int)(r % Ni); *pk = g.ka + (int)(r / Ni);
        return true;
    }
    t -= 2 * nJ;
    const bool up = t >= nK;
    if (t >= 2 * nK || !(up ? g.pu : g.pd)) return false;
    const unsigned r = up ? t - nK : t;
    *pk = up ? g.kb : g.ka; *pi = g.ia + (int)(r % Ni); *pj = g.ja + (int)(r / Ni);
    return true;
}

__global__ void bc_rk_kernel(DevGrid g, DevBC bc, P0Stage p0, double* __restrict__ dst, long long nface) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= nface) return;
    int i, j, k;
    if (!face_node(g, (unsigned)t, &i, &j, &k)) return;
    dst[gid(g, i, j, k)] = bc_value(g, bc, p0, i, j, k);
}

// dst = bcond_lsm(src) over the full array (ghosts copied); flags non-finite output.
__global__ void bc_full_kernel(DevGrid g, DevBC bc, const double* __restrict__ src, double* __restrict__ dst,
                               unsigned* errflag) {
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y,
              k = blockIdx.z * BZ + threadIdx.z;
    if (i >= g.ni || j >= g.nj || k >= g.nk) return;
    const long long l = gid(g, i, j, k);
    double v;
    if (non_ghost(g, i, j, k) && on_phys_face(g, i, j, k)) {
        P0Field p0{g, src};
        v = bc_value(g, bc, p0, i, j, k);
    } else {
        v = src[l];
    }
    dst[l] = v;
    if (errflag && !finite64(v)) atomicOr(errflag, (unsigned)kErrNonFinite);
}

// ------------------------------------------------------------ R1 / R2 ----
// The Godunov norm of calc_sign_ini.F90:190-242 as written there, from the
// metrics and the backward / forward differences
__device__ __noinline__ double godunov_norm_ieee(bool plus, double m0, double m1, double m2, double m3, double m4,
                                                 double m5, double m6, double m7, double m8, double q0, double q1,
                                                 double q2, double p0, double p1, double p2) {
    const double M[9] = {m0, m1, m2, m3, m4, m5, m6, m7, m8};
    double m[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const double ab = (M[x] * q0 + M[3 + x] * q1 + M[6 + x] * q2) / 2.0;
        const double af = (M[x] * p0 + M[3 + x] * p1 + M[6 + x] * p2) / 2.0;
        const double p = plus ? ab + fabs(ab) : ab - fabs(ab), q = plus ? af - fabs(af) : af + fabs(af);
        m[x] = fmax(p * p, q * q);
    }
    return sqrt(m[0] + m[1] + m[2]);
}

// The norm G+ (plus) or G- of one node: the one-sided differences of
// src/calc_sign_ini.F90:42-176 (= calc_RH_RN.F90:36-170), the gradients on
// them and the Godunov choice.
//
// Of each pair b/2 +- |b/2| one is b and the other 0, and the larger of two
// squares is the square of the larger magnitude: both are chosen on the
// integer pipes, and only the norm that is used is formed, with one square
// per direction.  The products and the root run on the integer pipes too,
// beside the 20 additions left to the FP64 pipe (134 clocked operations
// where both norms were formed with CUDA's root).  Each is exactly the value
// of the written-out expression while every factor is 0 or in 2^-200 .. 2^240
// (products are then multiples of 2^-452, and so is a sum of them that
// cancels: within usqr's range or 0); others take that expression, in a call
// (as in product_ieee).  0.79 ms a pseudo-step before, 0.20 ms now on
// 256 x 128 x 96 nodes; at most 64 registers for four blocks per SM (86 and
// two blocks: 0.27 ms).
__device__ __forceinline__ double godunov_norm(const DevGrid& g, const double* __restrict__ f,
                                               const double* __restrict__ csi, const double* __restrict__ eta,
                                               const double* __restrict__ zet, long long l, int i, int j, int k,
                                               bool plus) {
    const long long st[3] = {1, g.sj, g.sk};
    const double dd[3] = {g.dc, g.de, g.dz};
    const int c[3] = {i, j, k};
    const int plo[3] = {g.pb, g.pl, g.pd}, phs[3] = {g.pf, g.pr, g.pu};
    const int lo[3] = {g.ia, g.ja, g.ka}, hi[3] = {g.ib, g.jb, g.kb};
    double mas[3], men[3], M[9];
    const double fc = __ldg(f + l);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const long long s = st[d];
        const bool first = plo[d] && c[d] == lo[d], last = phs[d] && c[d] == hi[d];
        double p = last ? 0.0 : __ldg(f + l + s) - fc, q = first ? 0.0 : fc - __ldg(f + l - s);
        if (!g.unit) { p = product_ieee(dd[d], p); q = product_ieee(dd[d], q); }
        mas[d] = last ? q : p;
        men[d] = first ? p : q;
    }
    const double* m[3] = {csi + 3 * l, eta + 3 * l, zet + 3 * l};
    auto fits = [](double v) { return biased_exp(v) - 823u < 440u || mag(v) == 0u; };
    bool ok = true;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        M[q] = __ldg(m[q / 3] + q % 3);
        ok = ok && fits(M[q]);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) ok = ok && fits(mas[d]) && fits(men[d]);
    if (!ok)
        return godunov_norm_ieee(plus, M[0], M[1], M[2], M[3], M[4], M[5], M[6], M[7], M[8], men[0], men[1], men[2],
                                 mas[0], mas[1], mas[2]);
    double w[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const double b = umul0(M[x], men[0]) + umul0(M[3 + x], men[1]) + umul0(M[6 + x], men[2]);
        const double e = umul0(M[x], mas[0]) + umul0(M[3 + x], mas[1]) + umul0(M[6 + x], mas[2]);
        const u64 p = ((d2u(b) >> 63) != 0u) != plus ? mag(b) : 0u;   // plus: b > 0, else b < 0
        const u64 q = ((d2u(e) >> 63) != 0u) == plus ? mag(e) : 0u;   // plus: e < 0, else e > 0
        w[x] = usqr(u2d(p > q ? p : q));
    }
    return ssqrt(w[0] + w[1] + w[2]);
}

// deltaf, src/global_lsm.F90:120-133
__device__ __forceinline__ double deltaf(double v, double e) {
    if (fabs(v) > e) return 0.0;
    return 1.0 / (2.0 * e) * (1.0 + cos(kPi * v / e));
}

// calc_sign_ini, src/calc_sign_ini.F90:199-269 (+ deltaf(phi0) for the reinit steps)
__global__ void __launch_bounds__(256, 4) sign_ini_kernel(DevGrid g, const double* __restrict__ phi0, const double* __restrict__ csi,
                                const double* __restrict__ eta, const double* __restrict__ zet, double eps,
                                int M_Sphi0, double* __restrict__ sgn, double* __restrict__ ng,
                                double* __restrict__ delta) {
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y,
              k = blockIdx.z * BZ + threadIdx.z;
    if (i >= g.ni || j >= g.nj || k >= g.nk) return;
    const long long l = gid(g, i, j, k);
    if (!non_ghost(g, i, j, k)) {
        sgn[l] = 0.0; ng[l] = 0.0;
        if (delta) delta[l] = 0.0;
        return;
    }
    const double f = phi0[l];
    const bool pos = gt0(f);
    const double nrm = pos || lt0(f) ? godunov_norm(g, phi0, csi, eta, zet, l, i, j, k, pos) : 1.0;
    double s;
    if (M_Sphi0 == 1) {
        if (f >= eps) s = 1.0;
        else if (f <= (-1.0) * eps) s = -1.0;
        else s = f / eps - 1.0 / kPi * sin(kPi * f / eps);
    } else {
        s = f / sqrt(f * f + (nrm * eps) * (nrm * eps));
    }
    sgn[l] = s;
    ng[l] = nrm;
    if (delta) delta[l] = deltaf(f, eps);
}

// s (|grad d| - 1), src/calc_RH_RN.F90:185-238; s is +-1 but near the surface,
// where the product is the factor with its sign changed
__device__ __forceinline__ double reinit_rhs(const DevGrid& g, const double* __restrict__ d,
                                             const double* __restrict__ csi, const double* __restrict__ eta,
                                             const double* __restrict__ zet, long long l, int i, int j, int k,
                                             double s) {
    const bool pos = gt0(s);
    const double r = (pos || lt0(s) ? godunov_norm(g, d, csi, eta, zet, l, i, j, k, pos) : 1.0) - 1.0;
    return mag(s) == 0x3FF0000000000000ull ? (pos ? r : -r) : product_ieee(s, r);
}

// calc_RH_RN, src/calc_RH_RN.F90:185-238
__global__ void rh_rn_kernel(DevGrid g, const double* __restrict__ d, const double* __restrict__ sgn,
                             const double* __restrict__ csi, const double* __restrict__ eta,
                             const double* __restrict__ zet, double* __restrict__ rh) {
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y,
              k = blockIdx.z * BZ + threadIdx.z;
    if (i >= g.ni || j >= g.nj || k >= g.nk) return;
    const long long l = gid(g, i, j, k);
    if (!non_ghost(g, i, j, k)) { rh[l] = 0.0; return; }
    const double s = sgn[l];
    rh[l] = reinit_rhs(g, d, csi, eta, zet, l, i, j, k, s);
}

// calc_lambda_RN method 0, src/calc_lambda_RN.F90:42-63 (rdt = 1 / dt)
__device__ __forceinline__ double lambda_node(const DevGrid& g, double del, double rdt, double d, double p0,
                                              double ng) {
    const double Lop = del * (rdt * (d - p0));
    const double num = g.unit ? Lop : g.vc * Lop;
    const double den = (g.unit ? del * del : g.vc * (del * del)) * ng;
    return den == 0.0 ? 0.0 : sdiv(-num, den);
}

__global__ void lambda_rn_kernel(DevGrid g, double eps, const double* __restrict__ phi0,
                                 const double* __restrict__ ng, const double* __restrict__ d, double dt,
                                 double* __restrict__ lam) {
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y,
              k = blockIdx.z * BZ + threadIdx.z;
    if (i >= g.ni || j >= g.nj || k >= g.nk) return;
    const long long l = gid(g, i, j, k);
    if (!non_ghost(g, i, j, k)) { lam[l] = 0.0; return; }
    lam[l] = lambda_node(g, deltaf(phi0[l], eps), 1.0 / dt, d[l], phi0[l], ng[l]);
}

// One pseudo-step of `reinitialization`, src/reinitialization.F90:55-99,
// fused: Godunov RHS -> Euler update -> lambda -> correction.
__global__ void __launch_bounds__(256, 4) reinit_step_kernel(DevGrid g, double dt, double rdt, const double* __restrict__ din,
                                   const double* __restrict__ sgn, const double* __restrict__ ng,
                                   const double* __restrict__ delta, const double* __restrict__ phi0,
                                   const double* __restrict__ csi, const double* __restrict__ eta,
                                   const double* __restrict__ zet, double* __restrict__ dout) {
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y,
              k = blockIdx.z * BZ + threadIdx.z;
    if (i >= g.ni || j >= g.nj || k >= g.nk) return;
    const long long l = gid(g, i, j, k);
    const double dc0 = din[l];
    if (!non_ghost(g, i, j, k)) { dout[l] = dc0; return; }
    const double d1 = dc0 - dt * reinit_rhs(g, din, csi, eta, zet, l, i, j, k, sgn[l]);
    const double del = delta[l], gn = ng[l];
    // away from the surface delta is 0: lambda is 0 and the correction +0
    if (mag(del) == 0u && finite64(gn)) { dout[l] = d2u(d1) == 1ull << 63 ? 0.0 : d1; return; }
    const double lam = lambda_node(g, del, rdt, d1, phi0[l], gn);
    dout[l] = d1 + dt * lam * del * gn;
}

// ---------------------------------------------------------------- N1 ----
// narrowband, src/narrowband.F90:9-19 (every node, ghosts included)
__global__ void narrowband_kernel(long long n, double thr, int isnarrow, const double* __restrict__ phin,
                                  int* __restrict__ nb) {
    const long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (l >= n) return;
    nb[l] = isnarrow == 0 ? 1 : (fabs(phin[l]) < thr ? 1 : 0);
}

// ---------------------------------------------------------------- M0 ----
// mg_metrics on one rank's fine grid, src/mg_metrics.F90:44-264
__global__ void metrics_kernel(DevGrid g, const double* __restrict__ x, const double* __restrict__ y,
                               const double* __restrict__ z, double* __restrict__ csi, double* __restrict__ eta,
                               double* __restrict__ zet, double* __restrict__ aj) {
    const int i = blockIdx.x * BX + threadIdx.x, j = blockIdx.y * BY + threadIdx.y,
              k = blockIdx.z * BZ + threadIdx.z;
    if (i >= g.ni || j >= g.nj || k >= g.nk) return;
    const long long l = gid(g, i, j, k);
    const long long st[3] = {1, g.sj, g.sk};
    const double dd[3] = {g.dc, g.de, g.dz};
    const int c[3] = {i, j, k}, hi[3] = {g.ni - 1, g.nj - 1, g.nk - 1};
    double dx[3], dy[3], dzv[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const long long s = st[d];
        const double dum1 = dd[d], dum = 0.5 * dd[d];
        if (c[d] == 0) {
            dx[d] = dum1 * (x[l + s] - x[l]); dy[d] = dum1 * (y[l + s] - y[l]); dzv[d] = dum1 * (z[l + s] - z[l]);
        } else if (c[d] == hi[d]) {
            dx[d] = dum1 * (x[l] - x[l - s]); dy[d] = dum1 * (y[l] - y[l - s]); dzv[d] = dum1 * (z[l] - z[l - s]);
        } else {
            dx[d] = dum * (x[l + s] - x[l - s]); dy[d] = dum * (y[l + s] - y[l - s]);
            dzv[d] = dum * (z[l + s] - z[l - s]);
        }
    }
    const double xc = dx[0], yc = dy[0], zc = dzv[0], xe = dx[1], ye = dy[1], ze = dzv[1];
    const double xz = dx[2], yz = dy[2], zz = dzv[2];
    const double gj = xc * (ye * zz - yz * ze) + xe * (yz * zc - yc * zz) + xz * (yc * ze - ye * zc);
    const double a = 1.0 / gj;
    aj[l] = a;
    csi[3 * l + 0] = a * (ye * zz - yz * ze);
    csi[3 * l + 1] = a * (xz * ze - xe * zz);
    csi[3 * l + 2] = a * (xe * yz - xz * ye);
    eta[3 * l + 0] = a * (yz * zc - yc * zz);
    eta[3 * l + 1] = a * (xc * zz - xz * zc);
    eta[3 * l + 2] = a * (xz * yc - xc * yz);
    zet[3 * l + 0] = a * (yc * ze - ye * zc);
    zet[3 * l + 1] = a * (xe * zc - xc * ze);
    zet[3 * l + 2] = a * (xc * ye - xe * yc);
}

__global__ void copy_kernel(const double* __restrict__ src, double* __restrict__ dst, long long n) {
    for (long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x; l < n;
         l += (long long)gridDim.x * blockDim.x)
        dst[l] = src[l];
}

}  // namespace

// ---------------------------------------------------------------- launchers
#define LSM_BOX(g) box_grid((g).ni, (g).nj, (g).nk), dim3(BX, BY, BZ), 0, s

void launch_contra(const DevGrid& g, const double* q, const double* csi, const double* eta,
                   const double* zet, const double* aj, double* ucn, cudaStream_t s) {
    ProfScope ps_("contra_kernel", s);
    contra_kernel<<<LSM_BOX(g)>>>(g, q, csi, eta, zet, aj, ucn);
}

void launch_rh_ad(const DevGrid& g, int orderAD, const double* phi, const double* ucn, const int* mask,
                  double* rh, cudaStream_t s) {
    ProfScope ps_("rh_ad_kernel", s);
    if (orderAD == 1) launch_weno<true>(g, StageArgs{nullptr, phi, ucn, nullptr, mask, 0.0, 0.0, 0.0, 0.0, 0, rh}, s);
    else rh_upwind_kernel<<<LSM_BOX(g)>>>(g, phi, ucn, mask, rh);
}

void launch_rk_stage(const DevGrid& g, int orderAD, const double* phin, const double* phi1, const double* ucn,
                     const double* aj, const int* mask, double c1, double c2, double c3, double dt, double* out,
                     cudaStream_t s) {
    ProfScope ps_("rk_stage_kernel", s);
    const int first = c1 == 1.0 && c2 == 0.0 && c3 == 1.0 && phin == phi1;
    const StageArgs a{phin, phi1, ucn, aj, mask, c1, c2, c3, dt, first, out};
    if (orderAD == 1) launch_weno<false>(g, a, s);
    else rk_upwind_kernel<<<LSM_BOX(g)>>>(g, a);
}

void launch_bc_rk(const DevGrid& g, const DevBC& bc, int orderAD, const double* phin, const double* phi1,
                  const double* ucn, const double* aj, const int* mask, double c1, double c2, double c3,
                  double dt, double* dst, cudaStream_t s) {
    const long long Ni = g.ib - g.ia + 1, Nj = g.jb - g.ja + 1, Nk = g.kb - g.ka + 1;
    const long long nface = 2 * (Nj * Nk + Ni * Nk + Ni * Nj);
    P0Stage p0{g, orderAD, phin, phi1, ucn, aj, dst, mask, c1, c2, c3, dt};
    ProfScope ps_("bc_rk_kernel", s);
    bc_rk_kernel<<<(unsigned)((nface + 127) / 128), 128, 0, s>>>(g, bc, p0, dst, nface);
}

void launch_bc_full(const DevGrid& g, const DevBC& bc, const double* src, double* dst, unsigned* errflag,
                    cudaStream_t s) {
    ProfScope ps_("bc_full_kernel", s);
    bc_full_kernel<<<LSM_BOX(g)>>>(g, bc, src, dst, errflag);
}

void launch_sign_ini(const DevGrid& g, const double* phi0, const double* csi, const double* eta,
                     const double* zet, double eps, int M_Sphi0, double* sgn, double* ng, double* delta,
                     cudaStream_t s) {
    ProfScope ps_("sign_ini_kernel", s);
    sign_ini_kernel<<<LSM_BOX(g)>>>(g, phi0, csi, eta, zet, eps, M_Sphi0, sgn, ng, delta);
}

void launch_rh_rn(const DevGrid& g, const double* d, const double* sgn, const double* csi, const double* eta,
                  const double* zet, double* rh, cudaStream_t s) {
    ProfScope ps_("rh_rn_kernel", s);
    rh_rn_kernel<<<LSM_BOX(g)>>>(g, d, sgn, csi, eta, zet, rh);
}

void launch_lambda_rn(const DevGrid& g, double eps, const double* phi0, const double* ng, const double* d,
                      double dt, double* lam, cudaStream_t s) {
    ProfScope ps_("lambda_rn_kernel", s);
    lambda_rn_kernel<<<LSM_BOX(g)>>>(g, eps, phi0, ng, d, dt, lam);
}

void launch_reinit_step(const DevGrid& g, double dt, const double* din, const double* sgn, const double* ng,
                        const double* delta, const double* phi0, const double* csi, const double* eta,
                        const double* zet, double* dout, cudaStream_t s) {
    ProfScope ps_("reinit_step_kernel", s);
    reinit_step_kernel<<<LSM_BOX(g)>>>(g, dt, 1.0 / dt, din, sgn, ng, delta, phi0, csi, eta, zet, dout);
}

void launch_narrowband(const DevGrid& g, double thr, int isnarrow, const double* phin, int* nb, cudaStream_t s) {
    const long long n = (long long)g.ni * g.nj * g.nk;
    ProfScope ps_("narrowband_kernel", s);
    narrowband_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, thr, isnarrow, phin, nb);
}

void launch_metrics(const DevGrid& g, const double* x, const double* y, const double* z, double* csi,
                    double* eta, double* zet, double* aj, cudaStream_t s) {
    ProfScope ps_("metrics_kernel", s);
    metrics_kernel<<<LSM_BOX(g)>>>(g, x, y, z, csi, eta, zet, aj);
}

void launch_copy(const double* src, double* dst, long long n, cudaStream_t s) {
    long long blocks = (n + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (blocks < 1) blocks = 1;
    ProfScope ps_("copy_kernel", s);
    copy_kernel<<<(unsigned)blocks, 256, 0, s>>>(src, dst, n);
}

}  // namespace lsm
