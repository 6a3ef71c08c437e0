// lsm_volume.cu -- total water volume (FP64), the AdvectionNodes band and
// the ghost-fluid node list.  Compiled with --fmad=false: the volumes of the
// interface cells, the per-cell volumes and band membership are bit-identical
// to the reference's arithmetic; the sums are deterministic fixed-order trees
// (a thread's cells, block tree, then one block over the block partials)
// instead of the reference's sequential k-j-i accumulation.
//
// Roofline: the algorithmic traffic is 4 words per node (phi, x, y, z), of
// which x, y, z matter in the water and at the interface; what bounds the
// passes is the FP64 pipe, so comparisons run on the integer pipes.
#include <cuda_runtime.h>

#include "lsm_common.cuh"
#include "lsm_kernels.h"
#include "lsm_soft64.cuh"
#include "lsm_volume_dev.cuh"

namespace lsm {
namespace {

constexpr int VOL_THREADS = 128;
constexpr int VOL_BLOCKS = 152 * 8;

// comparisons with +-epsilon(1d0) and 0 on the bits (false for NaN)
constexpr u64 kEpsBits = 0x3CB0000000000000ull, kInfBits = 0x7FF0000000000000ull, kSign = 1ull << 63;
__device__ __forceinline__ bool above_eps(double v) { return d2u(v) - (kEpsBits + 1u) < kInfBits - kEpsBits; }
__device__ __forceinline__ bool below_eps(double v) { return d2u(v) - (kSign + kEpsBits + 1u) < kInfBits - kEpsBits; }
__device__ __forceinline__ bool near_zero(double v) { return mag(v) < kEpsBits; }
__device__ __forceinline__ bool at_most_eps(double v) { return mag(v) <= kInfBits && !above_eps(v); }
// copysign(1, a) * b < 0
__device__ __forceinline__ bool opposite(double a, double b) {
    return (d2u(a) ^ d2u(b)) >> 63 != 0u && mag(b) - 1u < kInfBits;
}

struct CellBox {
    int i0, j0, k0, Ni, Nj, Nk;       // base cells
    int ista, iend, jsta, jend, ksta, kend;  // clamp range of the band search
};

__host__ __device__ inline CellBox cell_box(const DevGrid& g) {
    CellBox b;
    b.i0 = g.ia; b.j0 = g.ja; b.k0 = g.ka;
    b.Ni = (g.ib - (g.pf ? 1 : 0)) - g.ia + 1;
    b.Nj = (g.jb - (g.pr ? 1 : 0)) - g.ja + 1;
    b.Nk = (g.kb - (g.pu ? 1 : 0)) - g.ka + 1;
    b.ista = g.pb ? g.ia : 0; b.iend = g.pf ? g.ib : g.ni - 1;
    b.jsta = g.pl ? g.ja : 0; b.jend = g.pr ? g.jb : g.nj - 1;
    b.ksta = g.pd ? g.ka : 0; b.kend = g.pu ? g.kb : g.nk - 1;
    return b;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// The water volume of one phase-change tetrahedron, bit for bit
// MarchingTetrahedron + GetWaterVolume (src/TetrahedronMethods.F90:26-954), its cases
// folded into two: one vertex apart from the other three, or two from two.
// Vertices and edges are taken by index (reloads of cached coordinates), so
// the lanes of a warp share the two code paths instead of eight.
//   n: the tetrahedron's nodes, ph its values
struct TetCase {
    signed char kind;        // 1: one apart, 2: two and two
    signed char a, b;        // apart vertex / the listed pair
    signed char e[4];        // edges
    signed char rest;        // the volume is the total less the formula's
};
__constant__ TetCase c_cases[16] = {
    {0, 0, 0, {0, 0, 0, 0}, 0}, {1, 0, 0, {0, 2, 3, 0}, 1}, {1, 1, 0, {0, 1, 4, 0}, 1}, {2, 0, 1, {1, 2, 3, 4}, 1},
    {1, 2, 0, {1, 2, 5, 0}, 1}, {2, 0, 2, {0, 1, 3, 5}, 1}, {2, 1, 2, {0, 2, 4, 5}, 1}, {1, 3, 0, {3, 4, 5, 0}, 0},
    {1, 3, 0, {3, 4, 5, 0}, 1}, {2, 1, 2, {0, 2, 4, 5}, 0}, {2, 0, 2, {0, 1, 3, 5}, 0}, {1, 2, 0, {1, 2, 5, 0}, 0},
    {2, 0, 1, {1, 2, 3, 4}, 0}, {1, 1, 0, {0, 1, 4, 0}, 0}, {1, 0, 0, {0, 2, 3, 0}, 0}, {0, 0, 0, {0, 0, 0, 0}, 0}};

__device__ double tet_water_ref(const double* __restrict__ x, const double* __restrict__ y,
                                const double* __restrict__ z, const double* __restrict__ phi, const long long (&n)[4],
                                const double (&ph)[4], unsigned* err) {
    const u64 tiny = 0x0010000000000000ull;   // tiny(1d0)
    unsigned P = 0, M = 0;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const u64 m = mag(ph[v]);
        const bool big = m > tiny && m <= kInfBits;
        if (big && d2u(ph[v]) >> 63 == 0u) P |= 1u << v;
        if (big && d2u(ph[v]) >> 63 != 0u) M |= 1u << v;
    }
    if (M == 15u) return 0.0;
    const unsigned Z = 15u & ~(P | M);
    int fi = (int)M;
    double TV = 0.0;
    auto load = [&](long long l, double (&V)[3]) {
        V[0] = __ldg(x + l); V[1] = __ldg(y + l); V[2] = __ldg(z + l);
    };
    auto node = [&](int v) { return v == 0 ? n[0] : (v == 1 ? n[1] : (v == 2 ? n[2] : n[3])); };
    bool whole = P == 15u;
    if (Z != 0u && (P == 0u || M == 0u)) {
        // zero vertices on one side: the sign of the reference's chosen
        // vertex; four zero vertices: the whole tetrahedron (FlagIndex 0)
        const int nz = __popc(Z);
        int q;
        if (nz == 1) q = Z == 1u ? 1 : 0;
        else if (nz == 2) q = Z == 3u ? 2 : ((Z == 5u || Z == 9u) ? 1 : 0);
        else q = nz == 3 ? __ffs(15 & ~Z) - 1 : 0;
        whole = nz == 4 || (P >> q & 1u);
        if (!whole) return 0.0;
    }
    {
        double V[4][3];
#pragma unroll
        for (int v = 0; v < 4; ++v) load(n[v], V[v]);
        TV = tetvol_ref(V[0], V[1], V[2], V[3]);
    }
    if (whole) return TV;
    const TetCase C = c_cases[fi];
    if (C.kind == 0) return TV;   // values that compare as neither sign (NaN)
    double E[4][3];
#pragma unroll 1
    for (int e = 0; e < 4; ++e) {
        if (e == 3 && C.kind == 1) break;
        const int g = C.e[e];
        const long long ns = node(c_edge[g][0]), ne = node(c_edge[g][1]);
        const double ps = __ldg(phi + ns), pe = __ldg(phi + ne);
        const double den = pe - ps;
        const double sc = mag(den) < 0x3630000000000000ull ? 0.0 : sdiv(pe, den);   // (2^-52)^3
        double S[3], V[3];
        load(ns, S);
        load(ne, V);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double w = V[c] + sc * (S[c] - V[c]);
            if (e == 0) E[0][c] = w;
            else if (e == 1) E[1][c] = w;
            else if (e == 2) E[2][c] = w;
            else E[3][c] = w;
        }
    }
    double A[3], AV;
    load(node(C.a), A);
    if (C.kind == 1) {
        AV = tetvol_ref(A, E[0], E[1], E[2]);
    } else {
        // cases 4/13: (E2, E3, E4), (E1, E2, E4), (b, E1, E4); the others:
        // (e0, e1, e3), (e0, e2, e3), (b, e1, e3)
        const bool f = C.e[0] == 1;
        double B[3], R[3], S[3];
        load(node(C.b), B);
#pragma unroll
        for (int c = 0; c < 3; ++c) { R[c] = f ? E[1][c] : E[0][c]; S[c] = f ? E[2][c] : E[1][c]; }
        AV = tetvol_ref(A, R, S, E[3]);
#pragma unroll
        for (int c = 0; c < 3; ++c) S[c] = f ? E[1][c] : E[2][c];
        AV = AV + tetvol_ref(A, E[0], S, E[3]);
#pragma unroll
        for (int c = 0; c < 3; ++c) R[c] = f ? E[0][c] : E[1][c];
        AV = AV + tetvol_ref(A, B, R, E[3]);
    }
    const double r = C.rest ? TV - AV : AV;
    if (below_eps(r) && err) atomicOr(err, (unsigned)kErrNegativeVolume);
    return r;
}

// Water volume of the base cells (TotalWaterVolume.F90:136-294) in chunks of
// one cell per thread, block partials (K tetrahedra, second tetrahedra,
// bulk) in a fixed order.
//
// Interface cells: listed per chunk, and their 6 tetrahedra shared out over
// the threads (before, a warp walked the tetrahedra of its few interface
// cells one after the other); each cell's tetrahedra are added in order.
// Bound by the FP64 work of the interface cells (~250 operations a
// tetrahedron) and of the water cells (147 each): the pipe is busy for 77 % of
// the time (192 x 96 x 72 nodes).  (The water cells' total
// from the faces of the water's surface alone takes fewer, but the error of
// such a sum grows with the distance to the point that its terms are taken
// about: 2e-15 where the cells' own volumes give 1e-16.)  256 x 128 x 96
// nodes: 0.87 ms before, 0.52 ms now, at eight blocks per SM as at four
// (0.53 ms, without spills; five and six: 0.56 ms).
__global__ void __launch_bounds__(VOL_THREADS, 8) volume_kernel(DevGrid g, CellBox cb,
        const double* __restrict__ phi, const double* __restrict__ x, const double* __restrict__ y,
        const double* __restrict__ z, double* __restrict__ partials, double* __restrict__ cellvol, unsigned* err) {
    __shared__ double val[6 * VOL_THREADS];
    __shared__ unsigned char kind[6 * VOL_THREADS];   // 1: K tetrahedron, 2: second
    __shared__ int cut[VOL_THREADS];                  // chunk positions of the interface cells
    __shared__ int wcut[VOL_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long ncell = (long long)cb.Ni * cb.Nj * cb.Nk;
    double K = 0.0, S = 0.0, B = 0.0;
    for (long long base = blockIdx.x * (long long)VOL_THREADS; base < ncell;
         base += (long long)gridDim.x * VOL_THREADS) {
        const long long t = base + threadIdx.x;
        bool mine = false;
        long long l = 0;
        if (t < ncell) {
            const int i = cb.i0 + (int)(t % cb.Ni);
            const int j = cb.j0 + (int)((t / cb.Ni) % cb.Nj);
            const int k = cb.k0 + (int)(t / ((long long)cb.Ni * cb.Nj));
            l = gid(g, i, j, k);
            const long long o[8] = {l, l + 1, l + 1 + g.sj, l + g.sj,
                                    l + g.sk, l + 1 + g.sk, l + 1 + g.sj + g.sk, l + g.sj + g.sk};
            bool allw = true, alla = true, zero = false, pos = false, neg = false;
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                const double P = __ldg(phi + o[v]);
                const bool a = above_eps(P), b = below_eps(P);
                allw = allw && a;
                alla = alla && b;
                zero = zero || near_zero(P);
                pos = pos || (d2u(P) - 1u < kInfBits);
                neg = neg || (d2u(P) - (kSign + 1u) < kInfBits);
            }
            double vol = 0.0;
            if (allw) {
                double C[8][3];
#pragma unroll
                for (int v = 0; v < 8; ++v) {
                    C[v][0] = __ldg(x + o[v]); C[v][1] = __ldg(y + o[v]); C[v][2] = __ldg(z + o[v]);
                }
                vol = hex_volume(C);
                B = B + vol;
            } else if (!alla) {
                // CellAnalysis: a vertex within eps of zero or a sign change
                // (seen from vertex 0)
                const double P0 = __ldg(phi + l);
                mine = zero || (d2u(P0) >> 63 != 0u ? pos : neg);
            }
            if (cellvol && !mine) cellvol[l] = vol;
        }
        // the chunk's interface cells in order
        const unsigned m = __ballot_sync(0xffffffffu, mine);
        if (lane == 0) wcut[w] = __popc(m);
        __syncthreads();
        int at = __popc(m & ((1u << lane) - 1u)), ncut = 0;
#pragma unroll
        for (int q = 0; q < VOL_THREADS / 32; ++q) {
            if (q < w) at += wcut[q];
            ncut += wcut[q];
        }
        if (mine) cut[at] = threadIdx.x;
        if (ncut == 0) {   // uniform
            __syncthreads();
            continue;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < 6 * ncut; q += VOL_THREADS) {
            const long long tc = base + cut[q % ncut];
            const int tt = q / ncut;
            const long long lc = gid(g, cb.i0 + (int)(tc % cb.Ni), cb.j0 + (int)((tc / cb.Ni) % cb.Nj),
                                     cb.k0 + (int)(tc / ((long long)cb.Ni * cb.Nj)));
            long long n[4];
            double ph[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int cv = c_tets[tt][v];
                n[v] = lc + (cv == 1 || cv == 2 || cv == 5 || cv == 6 ? 1 : 0) +
                       (cv == 2 || cv == 3 || cv == 6 || cv == 7 ? g.sj : 0) + (cv >= 4 ? g.sk : 0);
                ph[v] = __ldg(phi + n[v]);
            }
            bool pct = near_zero(ph[0]), second = !at_most_eps(ph[0]);
#pragma unroll
            for (int v = 1; v < 4; ++v)
                if (opposite(ph[0], ph[v]) || near_zero(ph[v])) {
                    pct = true;
                    if (at_most_eps(ph[v])) second = false;
                }
            double r = 0.0;
            int kd = 0;
            if (pct) {
                kd = 1;
                r = tet_water_ref(x, y, z, phi, n, ph, err);
            } else if (second) {
                kd = 2;
                double V[4][3];
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    V[v][0] = __ldg(x + n[v]); V[v][1] = __ldg(y + n[v]); V[v][2] = __ldg(z + n[v]);
                }
                r = tetvol_ref(V[0], V[1], V[2], V[3]);
            }
            val[q] = r;
            kind[q] = (unsigned char)kd;
        }
        __syncthreads();
        if (mine) {
            double k = 0.0, s2 = 0.0;
#pragma unroll 1
            for (int tt = 0; tt < 6; ++tt) {
                const int q = tt * ncut + at;
                if (kind[q] == 1) k = k + val[q];
                if (kind[q] == 2) s2 = s2 + val[q];
            }
            K = K + k;
            S = S + s2;
            if (cellvol) cellvol[l] = k + s2 + 0.0;
        }
        __syncthreads();
    }
    // fixed-order block reduction of (K, S, B)
    __shared__ double sh[3][VOL_THREADS / 32];
    K = warp_sum(K); S = warp_sum(S); B = warp_sum(B);
    if (lane == 0) { sh[0][w] = K; sh[1][w] = S; sh[2][w] = B; }
    __syncthreads();
    if (threadIdx.x < 3) {
        double acc = 0.0;
        for (int q = 0; q < VOL_THREADS / 32; ++q) acc = acc + sh[threadIdx.x][q];
        partials[3 * (long long)blockIdx.x + threadIdx.x] = acc;
    }
}

// One block folds the block partials in a fixed order, a group of warps per
// sum; result = (VK, V2, VB, total).
__global__ void __launch_bounds__(384) volume_final_kernel(const double* __restrict__ partials, int nblk,
                                                           double* __restrict__ result) {
    __shared__ double sh[12];
    const int c = threadIdx.x >> 7, t = threadIdx.x & 127;
    double acc = 0.0;
#pragma unroll 4
    for (int b = t; b < nblk; b += 128) acc = acc + partials[3 * (long long)b + c];
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) v[q] = (sh[4 * q] + sh[4 * q + 1]) + (sh[4 * q + 2] + sh[4 * q + 3]);
        result[0] = v[0]; result[1] = v[1]; result[2] = v[2];
        result[3] = v[0] + v[1] + v[2];
    }
}

// Phase-change base nodes (TotalWaterVolume.F90:169-224): a value within eps
// of zero, or one of the other sign, in the node's clamped 3 x 3 x 3 box --
// that is, a value within eps or both signs in the box.
__global__ void phase_change_kernel(DevGrid g, CellBox cb, const double* __restrict__ phi,
                                    unsigned char* __restrict__ pcflag) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)cb.Ni * cb.Nj * cb.Nk) return;
    const int i = cb.i0 + (int)(t % cb.Ni), j = cb.j0 + (int)((t / cb.Ni) % cb.Nj),
              k = cb.k0 + (int)(t / ((long long)cb.Ni * cb.Nj));
    const long long l = gid(g, i, j, k);
    const u64 f = d2u(__ldg(phi + l));
    bool pc = (f & ~kSign) < kEpsBits;
    // clamped offsets repeat a node of the box: the same answer
#pragma unroll
    for (int kk = -1; kk <= 1; ++kk)
#pragma unroll
        for (int jj = -1; jj <= 1; ++jj)
#pragma unroll
            for (int ii = -1; ii <= 1; ++ii) {
                const int a = min(max(i + ii, cb.ista), cb.iend), b = min(max(j + jj, cb.jsta), cb.jend),
                          c = min(max(k + kk, cb.ksta), cb.kend);
                const u64 h = d2u(__ldg(phi + gid(g, a, b, c))), m = h & ~kSign;
                pc = pc || m < kEpsBits || (((f ^ h) >> 63) != 0u && m - 1u < kInfBits);
            }
    pcflag[l] = pc ? 1 : 0;
}

// AdvectionNodes: the clamped 3x3x3 box of every phase-change base node is
// marked (TotalWaterVolume.F90:227-235), evaluated as a gather per node.
__global__ void adv_nodes_kernel(DevGrid g, CellBox cb, const unsigned char* __restrict__ pcflag,
                                 int* __restrict__ adv) {
    const long long n = (long long)g.ni * g.nj * g.nk;
    const long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (l >= n) return;
    const int i = (int)(l % g.ni), j = (int)((l / g.ni) % g.nj), k = (int)(l / ((long long)g.ni * g.nj));
    int a = 0;
    if (i >= cb.ista && i <= cb.iend && j >= cb.jsta && j <= cb.jend && k >= cb.ksta && k <= cb.kend) {
        const int bi0 = max(i - 1, cb.i0), bi1 = min(i + 1, cb.i0 + cb.Ni - 1);
        const int bj0 = max(j - 1, cb.j0), bj1 = min(j + 1, cb.j0 + cb.Nj - 1);
        const int bk0 = max(k - 1, cb.k0), bk1 = min(k + 1, cb.k0 + cb.Nk - 1);
        for (int bk = bk0; bk <= bk1; ++bk)
            for (int bj = bj0; bj <= bj1; ++bj)
                for (int bi = bi0; bi <= bi1; ++bi) a |= pcflag[gid(g, bi, bj, bk)];
    }
    adv[l] = a;
}

// ---------------------------------------------------------------- N3 ----
// get_gfm_list, src/get_gfm_list.F90:1-143: flag -> block counts -> scan ->
// ordered scatter.  The box is walked in Fortran (k, j, i) order, i.e. in
// increasing linear index, so the list order is the reference's.
constexpr int GFM_THREADS = 256;

struct GfmBox { int i0, j0, k0, Ni, Nj, Nk; };

__host__ __device__ inline GfmBox gfm_box(const DevGrid& g) {
    GfmBox b;
    b.i0 = g.ia + g.pb; b.j0 = g.ja + g.pl; b.k0 = g.ka + g.pd;
    b.Ni = (g.ib - g.pf) - b.i0 + 1; b.Nj = (g.jb - g.pr) - b.j0 + 1; b.Nk = (g.kb - g.pu) - b.k0 + 1;
    return b;
}

__device__ __forceinline__ bool gfm_flag(const DevGrid& g, const GfmBox& b, double BigPhi,
                                         const double* __restrict__ phi, long long t, int* pi, int* pj, int* pk) {
    const long long T = (long long)b.Ni * b.Nj * b.Nk;
    if (t >= T) return false;
    const int i = b.i0 + (int)(t % b.Ni), j = b.j0 + (int)((t / b.Ni) % b.Nj),
              k = b.k0 + (int)(t / ((long long)b.Ni * b.Nj));
    *pi = i; *pj = j; *pk = k;
    const double f = phi[gid(g, i, j, k)];
    if (above_eps(f) || fabs(f) > BigPhi) return false;
    bool any = false;
#pragma unroll
    for (int kk = -1; kk <= 1; ++kk)
#pragma unroll
        for (int jj = -1; jj <= 1; ++jj) {
            const double* p = phi + gid(g, i - 1, j + jj, k + kk);
            any = any || above_eps(__ldg(p)) || above_eps(__ldg(p + 1)) || above_eps(__ldg(p + 2));
        }
    return any;
}

__global__ void __launch_bounds__(GFM_THREADS) gfm_count_kernel(DevGrid g, GfmBox b, double BigPhi,
                                                                const double* __restrict__ phi, int* counts) {
    const long long t = blockIdx.x * (long long)GFM_THREADS + threadIdx.x;
    int i, j, k;
    const int f = gfm_flag(g, b, BigPhi, phi, t, &i, &j, &k) ? 1 : 0;
    const int c = __syncthreads_count(f);
    if (threadIdx.x == 0) counts[blockIdx.x] = c;
}

// exclusive scan of the block counts (one block, sequential chunks per thread)
__global__ void __launch_bounds__(1024) gfm_scan_kernel(int* counts, int nblk, int* total) {
    __shared__ int sh[1024];
    const int per = (nblk + 1023) / 1024;
    const int b0 = threadIdx.x * per, b1 = min(b0 + per, nblk);
    int sum = 0;
    for (int b = b0; b < b1; ++b) sum += counts[b];
    sh[threadIdx.x] = sum;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        int v = threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
        __syncthreads();
        sh[threadIdx.x] += v;
        __syncthreads();
    }
    int run = sh[threadIdx.x] - sum;
    for (int b = b0; b < b1; ++b) {
        const int c = counts[b];
        counts[b] = run;
        run += c;
    }
    if (threadIdx.x == 1023) *total = sh[1023];
}

__global__ void __launch_bounds__(GFM_THREADS) gfm_scatter_kernel(DevGrid g, GfmBox b, double BigPhi,
        const double* __restrict__ phi, const int* __restrict__ offsets, int il, int jl, int kl,
        int* __restrict__ list, int ld) {
    const long long t = blockIdx.x * (long long)GFM_THREADS + threadIdx.x;
    int i = 0, j = 0, k = 0;
    const bool f = gfm_flag(g, b, BigPhi, phi, t, &i, &j, &k);
    const unsigned m = __ballot_sync(0xffffffffu, f);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __shared__ int wsum[GFM_THREADS / 32];
    if (lane == 0) wsum[w] = __popc(m);
    __syncthreads();
    int base = offsets[blockIdx.x];
    for (int q = 0; q < w; ++q) base += wsum[q];
    if (f) {
        const int pos = base + __popc(m & ((1u << lane) - 1u));
        if (pos < ld) {
            list[pos] = i + il;
            list[pos + (long long)ld] = j + jl;
            list[pos + 2 * (long long)ld] = k + kl;
        }
    }
}

}  // namespace

int volume_partial_blocks(const DevGrid& g) {
    const CellBox cb = cell_box(g);
    const long long chunks = ((long long)cb.Ni * cb.Nj * cb.Nk + VOL_THREADS - 1) / VOL_THREADS;
    return (int)(chunks < VOL_BLOCKS ? chunks : VOL_BLOCKS);
}

void launch_volume(const DevGrid& g, const double* phi, const double* x, const double* y, const double* z,
                   double* partials, double* result, unsigned char* pcflag, double* cellvol, unsigned* err,
                   cudaStream_t s) {
    const CellBox cb = cell_box(g);
    const int nblk = volume_partial_blocks(g);
    {
        ProfScope ps_("volume_kernel", s);
        volume_kernel<<<nblk, VOL_THREADS, 0, s>>>(g, cb, phi, x, y, z, partials, cellvol, err);
    }
    if (pcflag) {
        const long long ncell = (long long)cb.Ni * cb.Nj * cb.Nk;
        ProfScope ps_("phase_change_kernel", s);
        phase_change_kernel<<<(unsigned)((ncell + 255) / 256), 256, 0, s>>>(g, cb, phi, pcflag);
    }
    ProfScope ps_("volume_final_kernel", s);
    volume_final_kernel<<<1, 384, 0, s>>>(partials, nblk, result);
}

void launch_adv_nodes(const DevGrid& g, const unsigned char* pcflag, int* adv, cudaStream_t s) {
    const long long n = (long long)g.ni * g.nj * g.nk;
    ProfScope ps_("adv_nodes_kernel", s);
    adv_nodes_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(g, cell_box(g), pcflag, adv);
}

long long gfm_scratch_ints(const DevGrid& g) {
    const GfmBox b = gfm_box(g);
    const long long T = (long long)b.Ni * b.Nj * b.Nk;
    return (T + GFM_THREADS - 1) / GFM_THREADS;
}

// Passes 1-2 when list == nullptr (count only), pass 3 otherwise (the caller
// has already run passes 1-2 on the same scratch and checked the capacity).
void launch_gfm_list(const DevGrid& g, double BigPhi, const double* phi, int* scratch, int* count_out, int* list,
                     int ld, int il, int jl, int kl, cudaStream_t s) {
    const GfmBox b = gfm_box(g);
    const int nblk = (int)gfm_scratch_ints(g);
    if (!list) {
        {
            ProfScope ps_("gfm_count_kernel", s);
            gfm_count_kernel<<<nblk, GFM_THREADS, 0, s>>>(g, b, BigPhi, phi, scratch);
        }
        ProfScope ps_("gfm_scan_kernel", s);
        gfm_scan_kernel<<<1, 1024, 0, s>>>(scratch, nblk, count_out);
    } else {
        ProfScope ps_("gfm_scatter_kernel", s);
        gfm_scatter_kernel<<<nblk, GFM_THREADS, 0, s>>>(g, b, BigPhi, phi, scratch, il, jl, kl, list, ld);
    }
}

}  // namespace lsm
