// lsm_geometric_dev.cuh -- device code of the geometric reinitialisation
// (lsm_geometric.cu): lists, marching, distances and the kernels.  Compiled
// with --fmad=false there, and for the host by the tests.
#pragma once

#include <cuda_runtime.h>

#include "lsm_common.cuh"
#include "lsm_soft64.cuh"
#include "lsm_volume_dev.cuh"

// (the host tests count what fails it)
#if !defined(LSM_CHAIN_CHECK)
#define LSM_CHAIN_CHECK(ok) ((void)0)
#endif

namespace lsm {
namespace {

constexpr int kThreads = 256;
constexpr int kTile = 4 * kThreads;  // elements per scan tile

// ------------------------------------------------------------- geometry

// Comparisons on the integer pipe: for non-negative doubles (+0 included)
// the IEEE order is the order of the bit patterns as signed integers, and
// x < 0 holds exactly when the sign bit is set and x is not -0.  GB300's
// FP64 pipe is its scarce resource; these are exact (no NaN reaches them).
__device__ __forceinline__ long long dbits(double x) { return (long long)d2u(x); }
__device__ __forceinline__ bool nn_lt(double a, double b) { return dbits(a) < dbits(b); }   // a, b >= +0
__device__ __forceinline__ bool nn_le(double a, double b) { return dbits(a) <= dbits(b); }  // a, b >= +0
__device__ __forceinline__ bool neg(double x) {
    const long long b = dbits(x);
    return b < 0 && b != (long long)0x8000000000000000ULL;
}
__device__ __forceinline__ bool pos(double x) { return dbits(x) > 0; }  // x > 0
constexpr long long kOneBits = 0x3FF0000000000000LL;                    // 1.0
__device__ __forceinline__ bool lt1(double x) { return dbits(x) < kOneBits; }  // x < 1

// NORM2 of a 3-vector as gfortran expands the intrinsic: a scaled sum of
// squares, zeros skipped, sqrt(sum) * scale.  While the scale is exactly 1
// the divisions ax / 1 and the final * 1 are skipped (both are exact).
__device__ __forceinline__ double norm2v(const double* a) {
    double scale = 1.0, r = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const long long b = dbits(a[c]) & 0x7FFFFFFFFFFFFFFFLL;  // |a[c]|
        if (b != 0) {
            const double ax = __longlong_as_double(b);
            if (dbits(scale) < b) {
                const double v = sdiv(scale, ax);
                r = 1.0 + r * v * v;
                scale = ax;
            } else {
                const double v = dbits(scale) == kOneBits ? ax : sdiv(ax, scale);
                r = r + v * v;
            }
        }
    }
    const double q = ssqrt(r);
    return dbits(scale) == kOneBits ? q : q * scale;
}
__device__ __forceinline__ void sub3(const double* a, const double* b, double* c) {
    c[0] = a[0] - b[0]; c[1] = a[1] - b[1]; c[2] = a[2] - b[2];
}
// (the reference's sum starts from 0, which changes only the sign of a zero
// result: no use below depends on it)
__device__ __forceinline__ double dot3g(const double* a, const double* b) {
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}
__device__ __forceinline__ void cross3g(const double* a, const double* b, double* c) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}
__device__ __forceinline__ double dmin(double a, double b) { return nn_lt(b, a) ? b : a; }  // a, b >= +0
__device__ __forceinline__ double sgn1(double x) { return copysign(1.0, x); }  // sign(one, x)

// GetTriangleArea, src/TetrahedronMethods.F90:691-707
__device__ double tri_area(const double (&T)[3][3]) {
    double u[3], v[3], c[3];
    sub3(T[1], T[0], u); sub3(T[2], T[0], v); cross3g(u, v, c);
    return 0.5 * norm2v(c);
}

// TetrahedronTriangles, src/TetrahedronMethods.F90:86-104 (edges 0..5)
__constant__ signed char c_tet_tris[16][6] = {
    {-1, -1, -1, -1, -1, -1}, {0, 3, 2, -1, -1, -1}, {0, 1, 4, -1, -1, -1}, {1, 4, 2, 2, 4, 3},
    {1, 2, 5, -1, -1, -1},    {0, 3, 5, 0, 5, 1},    {0, 2, 5, 0, 5, 4},    {5, 4, 3, -1, -1, -1},
    {3, 4, 5, -1, -1, -1},    {4, 5, 0, 5, 2, 0},    {1, 5, 0, 5, 3, 0},    {5, 2, 1, -1, -1, -1},
    {3, 4, 2, 2, 4, 1},       {4, 1, 0, -1, -1, -1}, {2, 3, 0, -1, -1, -1}, {-1, -1, -1, -1, -1, -1}};

// MarchingTetrahedron with its triangle and area outputs,
// src/TetrahedronMethods.F90:26-664.  ntri: 1 or 2 triangles, 0 none,
// -1/-2 a vertex/edge on the zero level (no triangle kept by the caller).
struct MT {
    int ntri;
    double tri[2][3][3];
    double area, wv;
};

__device__ void marching_full(const double (&V)[4][3], const double (&ph)[4], MT& o, bool want_tri,
                              unsigned* err) {
    o.ntri = 0; o.area = 0.0; o.wv = 0.0;
    int s[4], nz = 0;
    bool allp = true, alln = true, allge = true, allle = true;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        s[v] = ph[v] > kTinyD ? 1 : (ph[v] < -kTinyD ? -1 : 0);
        allp &= s[v] == 1; alln &= s[v] == -1; nz += s[v] == 0;
        allge &= s[v] >= 0; allle &= s[v] <= 0;
    }
    if (allp) { o.wv = tetvol_ref(V[0], V[1], V[2], V[3]); return; }
    if (alln) return;
    int fi = 0;
    if (nz > 0 && (allge || allle)) {
        if (nz == 1 || nz == 2) {
            o.ntri = -nz;  // a vertex or an edge: no triangle is used downstream
            int water;
            if (nz == 1) {
                water = s[0] == 0 ? s[1] == 1 : s[0] == 1;
            } else {
                if (s[0] == 0 && s[1] == 0) water = s[2] == 1;
                else if (s[1] == 0 && s[2] == 0) water = s[0] == 1;
                else if (s[2] == 0 && s[0] == 0) water = s[1] == 1;
                else if (s[0] == 0 && s[3] == 0) water = s[1] == 1;
                else water = s[0] == 1;
            }
            o.wv = water ? tetvol_ref(V[0], V[1], V[2], V[3]) : 0.0;
            return;
        }
        if (nz == 3) {  // a face: one triangle
            o.ntri = 1;
            int v = 0;
            while (s[v] == 0) ++v;
            int q = 0;
#pragma unroll
            for (int w = 0; w < 4; ++w)
                if (w != v) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) o.tri[0][q][c] = V[w][c];
                    ++q;
                }
            if (want_tri) o.area = tri_area(o.tri[0]);
            o.wv = s[v] == 1 ? tetvol_ref(V[0], V[1], V[2], V[3]) : 0.0;
            return;
        }
        // four zero vertices: FlagIndex stays 0
    } else {
#pragma unroll
        for (int v = 0; v < 4; ++v)
            if (s[v] == -1) fi |= 1 << v;
    }
    if (fi == 0) o.wv = tetvol_ref(V[0], V[1], V[2], V[3]);
    const int ef = c_edge_flags[fi];
    if (ef == 0) return;
    double E[6][3];
#pragma unroll
    for (int e = 0; e < 6; ++e) {
        E[e][0] = E[e][1] = E[e][2] = -9.9;
        if (!(ef >> e & 1)) continue;
        const int sv = c_edge[e][0], ev = c_edge[e][1];
        const double den = ph[ev] - ph[sv];
        const double sc = fabs(den) < kEpsSims * kEpsSims * kEpsSims ? 0.0 : ph[ev] / den;
#pragma unroll
        for (int c = 0; c < 3; ++c) E[e][c] = V[ev][c] + sc * (V[sv][c] - V[ev][c]);
    }
    for (int t = 0; t < 2; ++t) {
        if (c_tet_tris[fi][3 * t] < 0) break;
        o.ntri += 1;
        if (!want_tri) continue;
        for (int v = 0; v < 3; ++v) {
            const int e = c_tet_tris[fi][3 * t + v];
#pragma unroll
            for (int c = 0; c < 3; ++c) o.tri[t][v][c] = E[e][c];
        }
        o.area = o.area + tri_area(o.tri[t]);
    }
    o.wv = water_volume(V, E, fi, err);
}

// norm2v and sdiv as calls: the distance code keeps to a few kB, so that the
// warps of an SM do not wait for instructions
__device__ __noinline__ double norm2c(double x, double y, double z) {
    const double a[3] = {x, y, z};
    return norm2v(a);
}
__device__ __forceinline__ double norm2f(const double* a) { return norm2c(a[0], a[1], a[2]); }
__device__ __noinline__ double quot(double a, double b) { return sdiv(a, b); }

// DistancePointLine, src/TetrahedronMethods.F90:1356-1399, given the
// vectors and norms the caller already has: AP = P - A, BP = P - B,
// AB = B - A and their norms (BA = A - B is -AB exactly)
__device__ __forceinline__ double dist_point_line(const double* AP, const double* BP, const double* AB, double nAP,
                                                  double nBP, double nAB) {
    const double BA[3] = {-AB[0], -AB[1], -AB[2]};
    bool valid = true;
    if (nn_lt(nAB, kEpsSims)) valid = false;
    if (neg(dot3g(AB, AP))) valid = false;
    if (neg(dot3g(BA, BP))) valid = false;
    if (valid) {
        double c[3];
        cross3g(AP, BP, c);
        return quot(norm2f(c), nAB);
    }
    return dmin(nAP, nBP);
}

// What DistancePointTriangle computes from the triangle alone, evaluated
// once per triangle with the same operations: the edge vectors
// AB = B - A, BC = C - B, CA = A - C, their norms, and the projection
// step's normal nv = AB x (C - A) (C - A is -CA exactly) with nv . nv.
struct TriGeo {
    double AB[3], BC[3], CA[3];
    double nAB, nBC, nCA;
    double nv[3], nn;
};

__device__ void tri_geo(const double* T, TriGeo& g) {
    const double* A = T;
    const double* B = T + 3;
    const double* Cv = T + 6;
    sub3(B, A, g.AB); sub3(Cv, B, g.BC); sub3(A, Cv, g.CA);
    g.nAB = norm2v(g.AB); g.nBC = norm2v(g.BC); g.nCA = norm2v(g.CA);
    const double v[3] = {-g.CA[0], -g.CA[1], -g.CA[2]};
    cross3g(g.AB, v, g.nv);
    g.nn = dot3g(g.nv, g.nv);
}

// DistancePointTriangle + CheckProjectionPointOnATriangle3,
// src/TetrahedronMethods.F90:1008-1070,1593-1684.  Each norm the reference
// evaluates more than once on the same vector (|P - A| as a vertex distance
// and inside DistancePointLine, |B - A| twice per edge, |A - B| = |B - A| in
// the degenerate-triangle test) is evaluated once here, and the parts that
// depend on the triangle alone come from TriGeo: same inputs, same value.
// Kept from the reference: the projected point weights P1 by alpha (the
// weight of P3 in the standard barycentric form) and P3 by gamma.
__device__ double dist_point_triangle(const double* T, const TriGeo& g, const double* P) {
    const double* A = T;
    const double* B = T + 3;
    const double* Cv = T + 6;
    double PA[3], PB[3], PC[3];
    sub3(P, A, PA); sub3(P, B, PB); sub3(P, Cv, PC);
    const double nA = norm2f(PA), nB = norm2f(PB), nC = norm2f(PC);
    double m = dmin(dmin(nA, nB), nC);
    m = dmin(m, dist_point_line(PA, PB, g.AB, nA, nB, g.nAB));
    m = dmin(m, dist_point_line(PB, PC, g.BC, nB, nC, g.nBC));
    m = dmin(m, dist_point_line(PC, PA, g.CA, nC, nA, g.nCA));
    if (nn_le(g.nAB, kEpsSims) || nn_le(g.nCA, kEpsSims) || nn_le(g.nBC, kEpsSims)) return m;
    const double v[3] = {-g.CA[0], -g.CA[1], -g.CA[2]};
    double cu[3], cw[3];
    cross3g(g.AB, PA, cu); cross3g(PA, v, cw);
    const double alpha = quot(dot3g(cu, g.nv), g.nn), beta = quot(dot3g(cw, g.nv), g.nn);
    const double gamma = 1.0 - beta - alpha;
    if (pos(alpha) && lt1(alpha) && pos(beta) && lt1(beta) && pos(gamma) && lt1(gamma)) {
        double pp[3], dd[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) pp[c] = alpha * A[c] + beta * B[c] + gamma * Cv[c];
        sub3(P, pp, dd);
        m = dmin(m, norm2f(dd));
    }
    return m;
}

// the reference's running minimum d + exsign (da - d), exsign = (sign(1,
// d - da) + 1) / 2: 1 when da <= d (d - da >= +0), and then d + (da - d);
// 0 otherwise, and then d + 0 = d.  d, da >= +0.
__device__ __forceinline__ double run_min(double d, double da) {
    return nn_le(da, d) ? d + (da - d) : d;
}

// the reference's signed update of a running |value| by a distance dp
// (exsign2 = 1 when |value| >= dp): the new magnitude
__device__ __forceinline__ double mag_step(double a, double dp) {
    return nn_le(dp, a) ? a + (dp - a) : a;
}

// ------------------------------------------------------------ the lists

// cell vertex v at offset (dx, dy, dz): the reference's numbering
// v0 = 000, v1 = 100, v2 = 110, v3 = 010, v4 = 001, v5 = 101, v6 = 111, v7 = 011
__constant__ int c_cell_off[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0},
                                     {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
__constant__ unsigned char c_vert_at[2][2][2] = {{{0, 4}, {3, 7}}, {{1, 5}, {2, 6}}};  // [dx][dy][dz]

// bits 1..6: the tetrahedra of the TriangulationCase-1 split containing vertex v
__host__ __device__ constexpr unsigned tets_of_vertex(int v) {
    constexpr int T[6][4] = {{0, 5, 1, 6}, {0, 1, 2, 6}, {0, 2, 3, 6}, {0, 3, 7, 6}, {0, 7, 4, 6}, {0, 4, 5, 6}};
    unsigned m = 0;
    for (int t = 0; t < 6; ++t)
        for (int q = 0; q < 4; ++q)
            if (T[t][q] == v) m |= 1u << (t + 1);
    return m;
}
__constant__ unsigned char c_vtets[8] = {tets_of_vertex(0), tets_of_vertex(1), tets_of_vertex(2),
                                         tets_of_vertex(3), tets_of_vertex(4), tets_of_vertex(5),
                                         tets_of_vertex(6), tets_of_vertex(7)};

// CellPnodeTetrahedronIdentification, src/TetrahedronMethods.F90:2124-2361:
// bit t (1..6) of *tets marks a phase-change tetrahedron, bit v of *verts a
// vertex of one
__device__ void cell_pnodes(const double (&P)[8], unsigned* verts, unsigned* tets) {
    *verts = 0; *tets = 0;
    bool allw = true, alla = true, anyz = false;
#pragma unroll
    for (int v = 0; v < 8; ++v) {
        allw &= P[v] > kEpsSims; alla &= P[v] < -kEpsSims; anyz |= fabs(P[v]) < kEpsSims;
    }
    if (allw || alla) return;
    bool pc = anyz;
    if (!pc) {
        const double s0 = sgn1(P[0]);
#pragma unroll
        for (int v = 1; v < 8; ++v) pc |= s0 * P[v] < 0.0;
    }
    if (!pc) return;
#pragma unroll
    for (int t = 0; t < 6; ++t) {
        double a = P[c_tets[t][0]];
        bool change = fabs(a) < kEpsSims, second = !(a <= kEpsSims);
        const double sg = sgn1(a);
#pragma unroll
        for (int q = 1; q < 4; ++q) {
            a = P[c_tets[t][q]];
            if (sg * a < 0.0 || fabs(a) < kEpsSims) {
                if (a <= kEpsSims) second = false;
                change = true;
            }
        }
        if (change && !second) {
            *tets |= 1u << (t + 1);
#pragma unroll
            for (int q = 0; q < 4; ++q) *verts |= 1u << c_tets[t][q];
        }
    }
}

__device__ __forceinline__ void node_ijk(const DevGrid& g, long long l, int* i, int* j, int* k) {
    *k = (int)(l / g.sk);
    const long long r = l - (long long)*k * g.sk;
    *j = (int)(r / g.sj);
    *i = (int)(r - (long long)*j * g.sj);
}

// the K tetrahedra with a vertex at node (i, j, k), in the order
// GetTetrahedraList appends them to the node's list
template <class F>
__device__ __forceinline__ void for_each_tet(const DevGrid& g, int i, int j, int k,
                                             const unsigned char* __restrict__ cellbits,
                                             const int* __restrict__ tetbase, F f) {
    for (int dz = 1; dz >= 0; --dz) {
        const int ck = k - dz;
        if (ck < 0 || ck > g.nk - 2) continue;
        for (int dy = 1; dy >= 0; --dy) {
            const int cj = j - dy;
            if (cj < 0 || cj > g.nj - 2) continue;
            for (int dx = 1; dx >= 0; --dx) {
                const int ci = i - dx;
                if (ci < 0 || ci > g.ni - 2) continue;
                const long long lc = gid(g, ci, cj, ck);
                const unsigned bits = cellbits[lc];
                unsigned m = bits & c_vtets[c_vert_at[dx][dy][dz]];
                if (!m) continue;
                const int base = tetbase[lc];
                while (m) {
                    const int t = __ffs(m) - 1;
                    m &= m - 1;
                    f(base + __popc(bits & ((1u << t) - 1u)));
                }
            }
        }
    }
}

// one K tetrahedron: its isosurface triangles (18 doubles) with their
// triangle-only distance terms (TriGeo), area and water volume of the
// linear reconstruction, its four pnode ids (0-based), and per triangle an
// FP32 bounding box (rounded outwards), used only to skip distance
// evaluations that cannot change a running minimum
struct alignas(16) GeoTet {
    double tri[2][9];
    TriGeo tg[2];
    float box[2][6];  // lo x y z, hi x y z
    double area, wv;
    int nis;
    int v[4];
    int pad;
};

// A distance evaluation is skipped only when a lower bound of the exact
// point-triangle distance -- the distance from the point to the triangle's
// bounding box -- exceeds the running minimum d by a margin.  Every candidate
// point of DistancePointTriangle (vertices, feet on the edges, the
// projection step's convex combination of the vertices) lies in the
// triangle, so the computed distance is at least the exact distance less a
// few ulps of the coordinates.  The bound is evaluated in FP32 (the FP64
// units are scarce) on a box rounded outwards: the point and d rounded to
// FP32 and the FP32 norm keep its error below 1e-6 of the sizes involved,
// and the margin is 1e-5 of them.  A skipped triangle therefore leaves
// d + exsign (da - d) = d exactly as the full evaluation would.
__device__ __forceinline__ bool beyond_box(const float* p, float pscale, const float* lo, const float* hi, float d) {
    const float dx = fmaxf(fmaxf(lo[0] - p[0], p[0] - hi[0]), 0.0f);
    const float dy = fmaxf(fmaxf(lo[1] - p[1], p[1] - hi[1]), 0.0f);
    const float dz = fmaxf(fmaxf(lo[2] - p[2], p[2] - hi[2]), 0.0f);
    const float lb = sqrtf(dx * dx + dy * dy + dz * dz);
    return lb > d + 1.0e-5f * (lb + d + pscale);
}

// One triangle in FP32, for tri_interval: vertex A, the edges AB and AC with
// their squared inverse lengths and BC's, the gradients ga and gb of the
// reference's alpha and beta in P - A, 1 / (least height), and a bound of the
// inradius (-1: an edge too short for the enclosure below, whose distance is
// bounded by the bounding box alone).
struct alignas(16) TriF {
    float A[3], rad, AB[3], iAB, AC[3], iAC, ga[3], iBC, gb[3], gmax;
};

__device__ void tri_f32(const double* T, const TriGeo& g, TriF& f) {
    double len = 0.0, scale = 0.0, nga = 0.0, ngb = 0.0, ngc = 0.0;
#pragma unroll
    for (int c = 0; c < 9; ++c) scale = fmax(scale, fabs(T[c]));
    len = fmin(g.nAB, fmin(g.nBC, g.nCA));
    const double AC[3] = {-g.CA[0], -g.CA[1], -g.CA[2]};
    double ga[3], gb[3];
    cross3g(g.nv, g.AB, ga);
    cross3g(AC, g.nv, gb);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        ga[c] = g.nn > 0.0 ? ga[c] / g.nn : 0.0;
        gb[c] = g.nn > 0.0 ? gb[c] / g.nn : 0.0;
        nga += ga[c] * ga[c];
        ngb += gb[c] * gb[c];
        ngc += (ga[c] + gb[c]) * (ga[c] + gb[c]);
        f.A[c] = (float)T[c];
        f.AB[c] = (float)g.AB[c];
        f.AC[c] = (float)AC[c];
        f.ga[c] = (float)ga[c];
        f.gb[c] = (float)gb[c];
    }
    const double gm = sqrt(fmax(nga, fmax(ngb, ngc)));
    f.gmax = g.nn > 0.0 && gm < 1.0e30 ? (float)gm : 3.0e38f;
    // the inradius is at most half the least height
    f.rad = !(len >= 1.0e-6 * (1.0 + scale)) ? -1.0f
                                             : (gm > 0.0 ? __double2float_ru(0.500001 / gm) : __double2float_ru(len));
    f.iAB = (float)(1.0 / (g.nAB * g.nAB));
    f.iAC = (float)(1.0 / (g.nCA * g.nCA));
    f.iBC = (float)(1.0 / (g.nBC * g.nBC));
}

// -------------------------------------------------------------- kernels

// GetTetrahedraList, first loop (src/GetTetrahedraList.F90:205-284)
__global__ void k_geo_cells(DevGrid g, const double* __restrict__ phi, unsigned char* __restrict__ cellbits,
                            int* __restrict__ flags) {
    const long long ncell = (long long)(g.ni - 1) * (g.nj - 1) * (g.nk - 1);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell;
         c += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(c % (g.ni - 1));
        const long long r = c / (g.ni - 1);
        const int j = (int)(r % (g.nj - 1));
        const int k = (int)(r / (g.nj - 1));
        double P[8];
#pragma unroll
        for (int v = 0; v < 8; ++v)
            P[v] = phi[gid(g, i + c_cell_off[v][0], j + c_cell_off[v][1], k + c_cell_off[v][2])];
        unsigned verts, tets;
        cell_pnodes(P, &verts, &tets);
        cellbits[gid(g, i, j, k)] = (unsigned char)tets;
#pragma unroll
        for (int v = 0; v < 8; ++v)
            if (verts >> v & 1) flags[gid(g, i + c_cell_off[v][0], j + c_cell_off[v][1], k + c_cell_off[v][2])] = 1;
    }
}

// block-wide exclusive scan of one value per thread; returns the prefix and
// the block total in *total
__device__ int block_exclusive_scan(int v, int* total) {
    __shared__ int ws[kThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = lane < kThreads / 32 ? ws[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < kThreads / 32) ws[lane] = t;
    }
    __syncthreads();
    const int before = w ? ws[w - 1] : 0;
    *total = ws[kThreads / 32 - 1];
    __syncthreads();
    return before + x - v;
}

// per-element count: mode 0 the pnode flag, mode 1 the number of K tetrahedra of the cell,
// mode 2 the -1 tag, mode 3 the number itself
template <int MODE>
__device__ __forceinline__ int scan_count(const void* src, long long l) {
    if (MODE == 0) return static_cast<const int*>(src)[l] ? 1 : 0;
    if (MODE == 2) return static_cast<const int*>(src)[l] < 0 ? 1 : 0;
    if (MODE == 3) return static_cast<const int*>(src)[l];
    return __popc(static_cast<const unsigned char*>(src)[l]);
}

template <int MODE>
__global__ void __launch_bounds__(kThreads) k_scan_tiles(long long n, const void* __restrict__ src,
                                                         int* __restrict__ tile_sum) {
    const long long base = (long long)blockIdx.x * kTile + 4 * threadIdx.x;
    int s = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (base + q < n) s += scan_count<MODE>(src, base + q);
    int tot;
    block_exclusive_scan(s, &tot);
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = tot;
}

// exclusive scan of the tile sums in place (one block); total -> *total
__global__ void __launch_bounds__(kThreads) k_scan_top(int ntiles, int* __restrict__ tile_sum,
                                                       int* __restrict__ total) {
    int carry = 0;
    for (int b0 = 0; b0 < ntiles; b0 += kThreads) {
        const int b = b0 + threadIdx.x;
        const int v = b < ntiles ? tile_sum[b] : 0;
        int tot;
        const int ex = block_exclusive_scan(v, &tot);
        if (b < ntiles) tile_sum[b] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) *total = carry;
}

// mode 0: ids[l] = pnode id + 1 (0: not a pnode), node_of[id] = l;
// mode 1: tetbase[l] = first K-tetrahedron id of cell l, node_of[id] = 8 l + its number 0..5;
// mode 2: node_of[c] = the c-th node tagged -1;
// mode 3: out[l] = the sum of the numbers before l, out[n] = that of all
template <int MODE>
__global__ void __launch_bounds__(kThreads) k_scan_apply(long long n, const void* __restrict__ src,
                                                         const int* __restrict__ tile_off, int* __restrict__ out,
                                                         long long* __restrict__ node_of) {
    const long long base = (long long)blockIdx.x * kTile + 4 * threadIdx.x;
    int c[4], s = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        c[q] = base + q < n ? scan_count<MODE>(src, base + q) : 0;
        s += c[q];
    }
    int tot;
    int off = tile_off[blockIdx.x] + block_exclusive_scan(s, &tot);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (base + q >= n) break;
        if (MODE == 0) {
            out[base + q] = c[q] ? off + 1 : 0;
            if (c[q]) node_of[off] = base + q;
        } else if (MODE == 1 || MODE == 3) {
            out[base + q] = off;
            if (MODE == 3 && base + q == n - 1) out[n] = off + c[q];
            if (MODE == 1 && c[q]) {
                int id = off;
                for (unsigned m = static_cast<const unsigned char*>(src)[base + q]; m; m &= m - 1)
                    node_of[id++] = 8 * (base + q) + __ffs(m) - 2;
            }
        } else if (c[q]) {
            node_of[off] = base + q;
        }
        off += c[q];
    }
}

// GetTetrahedraList third loop + the marching step of GetIsosurfaceAndDistances
// (src/GetIsosurfaceAndDistances.F90:80-162)
__global__ void k_geo_tets(DevGrid g, const double* __restrict__ phi, const double* __restrict__ x,
                           const double* __restrict__ y, const double* __restrict__ z,
                           int ntet, const long long* __restrict__ tet_of, const int* __restrict__ ids,
                           GeoTet* __restrict__ tets, TriF* __restrict__ trif, unsigned* err) {
    for (int tid = blockIdx.x * blockDim.x + threadIdx.x; tid < ntet; tid += gridDim.x * blockDim.x) {
        const long long lc = tet_of[tid] >> 3;
        const int t = (int)(tet_of[tid] & 7);
        double V[4][3], ph[4];
        GeoTet T;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int cv = c_tets[t][q];
            const long long l = lc + c_cell_off[cv][0] + g.sj * c_cell_off[cv][1] + g.sk * c_cell_off[cv][2];
            V[q][0] = x[l]; V[q][1] = y[l]; V[q][2] = z[l];
            ph[q] = phi[l];
            T.v[q] = ids[l] - 1;
        }
        MT o;
        marching_full(V, ph, o, true, err);
        T.nis = o.ntri > 0 ? o.ntri : 0;
        T.area = o.area;
        T.wv = o.wv;
        T.pad = 0;
        // (one copy of the triangle code for both triangles)
#pragma unroll 1
        for (int q = 0; q < 2; ++q) {
#pragma unroll
            for (int c = 0; c < 9; ++c) T.tri[q][c] = q < T.nis ? o.tri[q][c / 3][c % 3] : 0.0;
            if (q >= T.nis) continue;   // never read
            tri_geo(T.tri[q], T.tg[q]);
            TriF f;
            tri_f32(T.tri[q], T.tg[q], f);
            trif[2 * (long long)tid + q] = f;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double a = T.tri[q][c], b = T.tri[q][3 + c], e = T.tri[q][6 + c];
                T.box[q][c] = __double2float_rd(fmin(a, fmin(b, e)));
                T.box[q][3 + c] = __double2float_ru(fmax(a, fmax(b, e)));
            }
        }
        tets[tid] = T;
    }
}

// nodes within +-4 of a pnode that are not pnodes are tagged -1
// (src/GetIsosurfaceAndDistances.F90:322-328); out starts as a copy of ids
__global__ void k_geo_mark(DevGrid g, int npn, const long long* __restrict__ node_of, const int* __restrict__ ids,
                           int* __restrict__ out) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npn; p += gridDim.x * blockDim.x) {
        int i, j, k;
        node_ijk(g, node_of[p], &i, &j, &k);
        for (int ks = max(k - 4, 0); ks <= min(k + 4, g.nk - 1); ++ks)
            for (int js = max(j - 4, 0); js <= min(j + 4, g.nj - 1); ++js)
                for (int is = max(i - 4, 0); is <= min(i + 4, g.ni - 1); ++is) {
                    const long long l = gid(g, is, js, ks);
                    if (ids[l] == 0) out[l] = -1;
                }
    }
}

// a point in both precisions (the FP32 copy for the culling bounds)
struct Pt {
    double d[3];
    float f[3];
    float scale;
};
__device__ __forceinline__ Pt make_pt(double a, double b, double c) {
    Pt p;
    p.d[0] = a; p.d[1] = b; p.d[2] = c;
    p.f[0] = (float)a; p.f[1] = (float)b; p.f[2] = (float)c;
    p.scale = fmaxf(fabsf(p.f[0]), fmaxf(fabsf(p.f[1]), fabsf(p.f[2])));
    return p;
}

// per pnode: the bounding box of every triangle of its K tetrahedra
// (lo.w = 0: none of them has a triangle) and their number
__global__ void k_geo_prad(DevGrid g, int npn, const long long* __restrict__ node_of,
                           const unsigned char* __restrict__ cellbits, const int* __restrict__ tetbase,
                           const GeoTet* __restrict__ tets, float4* __restrict__ pbox, int* __restrict__ ntri) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npn; p += gridDim.x * blockDim.x) {
        int i, j, k;
        node_ijk(g, node_of[p], &i, &j, &k);
        float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
        float any = 0.0f;
        int nt = 0;
        for_each_tet(g, i, j, k, cellbits, tetbase, [&](int t) {
            const GeoTet& T = tets[t];
            if (T.nis > 0 && T.area > 0.0)
                for (int q = 0; q < T.nis; ++q) {
                    any = 1.0f;
                    ++nt;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        lo[c] = fminf(lo[c], T.box[q][c]);
                        hi[c] = fmaxf(hi[c], T.box[q][3 + c]);
                    }
                }
        });
        pbox[2 * p] = make_float4(lo[0], lo[1], lo[2], any);
        pbox[2 * p + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
        ntri[p] = nt;
    }
}

// The triangles of every pnode in the reference's order, from the entry
// pstart[p] on: 4 (2 tetrahedron + triangle) + min(2, ends of tetrahedra
// between this triangle and the next).  lead[p]: min(2, tetrahedra without
// triangles before the first one).
__global__ void k_geo_fill(DevGrid g, int npn, const long long* __restrict__ node_of,
                           const unsigned char* __restrict__ cellbits, const int* __restrict__ tetbase,
                           const GeoTet* __restrict__ tets, const int* __restrict__ pstart, int* __restrict__ pent,
                           unsigned char* __restrict__ lead) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npn; p += gridDim.x * blockDim.x) {
        int i, j, k;
        node_ijk(g, node_of[p], &i, &j, &k);
        int at = pstart[p] - 1, cur = -1, early = 0;
        for_each_tet(g, i, j, k, cellbits, tetbase, [&](int t) {
            const GeoTet& T = tets[t];
            const int nq = T.nis > 0 && T.area > 0.0 ? T.nis : 0;
            for (int q = 0; q < nq; ++q) {
                if (cur >= 0) pent[at] = cur;
                ++at;
                cur = 4 * (2 * t + q);
            }
            if (cur < 0) early = min(early + 1, 2);
            else if ((cur & 3) < 2) ++cur;
        });
        if (cur >= 0) pent[at] = cur;
        lead[p] = (unsigned char)early;
    }
}

// lower bound of the distance from P to pnode m's triangles (3e38: none)
__device__ __forceinline__ float pnode_bound(int m, const Pt& P, const float4* __restrict__ pbox) {
    const float4 a = pbox[2 * m], b = pbox[2 * m + 1];
    const float dx = fmaxf(fmaxf(a.x - P.f[0], P.f[0] - b.x), 0.0f);
    const float dy = fmaxf(fmaxf(a.y - P.f[1], P.f[1] - b.y), 0.0f);
    const float dz = fmaxf(fmaxf(a.z - P.f[2], P.f[2] - b.z), 0.0f);
    return a.w == 0.0f ? 3.0e38f : sqrtf(dx * dx + dy * dy + dz * dz);
}
// beyond_box for such a bound
__device__ __forceinline__ bool beyond(float lb, float pscale, float d) {
    return lb > d + 1.0e-5f * (lb + d + pscale);
}

// ------------------------------------------------- the distance chains
//
// Both distance loops are chains a <- a + (c - a) where c <= a, over the
// distances c of a node to the triangles of the pnodes in its +-4 box, in
// the reference's order.  Two facts make most of them unnecessary:
//   - a distance that is certainly above the running value changes nothing;
//   - for a/2 <= c <= a the update gives exactly c (c - a is exact), whatever
//     a was: what came before such a c is forgotten.
// A warp encloses the distances of each pnode's triangles in FP32 (one
// triangle per lane) and keeps, as tasks, only the triangles that can still
// decide the final bits: a pnode that certainly falls below everything
// before it, by less than a factor 2, drops all earlier tasks; a pnode
// certainly above adds none; one in between adds its triangles near the
// minimum; one that falls by a factor 2 or more adds all of its triangles.
// The lanes then evaluate the tasks in FP64 together and the chain is
// replayed over them in order.  The FP64 pipe (16 clocks per warp operation
// and SM) evaluated a few hundred distances per node before, of ~150
// operations each; now some ten.
constexpr int kMaxTri = 48;           // triangles of a pnode: two in each of at most 24 tetrahedra
constexpr int kTasks = 2 * kMaxTri + 32, kItems = 32;
constexpr int kChainWarps = 4;
enum : int { kSimple = 0, kReset = 1, kFull = 2 };

struct ChainQueue {
    double d[kTasks];
    int ent[kTasks];                  // entries of pent
    int item[kItems];                 // one per pnode: 4 (tasks before it) + kind
    int aux[kItems];                  // 4 (k_geo_sd: pnode's ordinal in the box; k_geo_neigh: exact_min) + lead
};

// Encloses the reference's distance of P to a triangle (dist_point_triangle).
// The value is the least of the distances to the edges and, inside the
// triangle, of the one to the reference's projection; any point it can take
// lies in the triangle.  E covers the FP32 roundings of an edge's distance,
// tau those of alpha and beta.  With u = 2^-24, p = P - A (n1 its sum of
// magnitudes) and l the longer of AB and AC:
//   P and A rounded, and their difference: 3.5 u scale + 2 u n1;
//   the foot on an edge (a dot product, the inverse length) and the vector to
//   it, for a vector q to the edge's start: 11 u |q|, |q| <= n1 + l;
//   AB and AC rounded, BC's direction and its inverse length from their
//   difference: 22 u l;
//   the square root of the sum of squares: 3 u s
// -- each below its share of E (2e-6 = 33 u).  n1 and l count where the point
// is near the origin of the coordinates and near the surface: scale and s are
// then small beside the triangle.
__device__ __noinline__ float2 tri_interval(const TriF* __restrict__ trif, const GeoTet* __restrict__ tets, int tri,
                                            float x, float y, float z, float scale) {
    float lo, hi;
    const float4* r = reinterpret_cast<const float4*>(trif + tri);
    const float4 a = __ldg(r), b = __ldg(r + 1), c = __ldg(r + 2), u = __ldg(r + 3), v = __ldg(r + 4);
    const float px = x - a.x, py = y - a.y, pz = z - a.z;
    if (a.w < 0.0f) {
        const float* box = tets[tri >> 1].box[tri & 1];
        const float dx = fmaxf(fmaxf(box[0] - x, x - box[3]), 0.0f);
        const float dy = fmaxf(fmaxf(box[1] - y, y - box[4]), 0.0f);
        const float dz = fmaxf(fmaxf(box[2] - z, z - box[5]), 0.0f);
        lo = fmaxf(0.0f, 0.99997f * sqrtf(dx * dx + dy * dy + dz * dz) - 1.1e-5f * scale);
        return make_float2(lo, 3.0e38f);
    }
    auto seg = [](float qx, float qy, float qz, float ex, float ey, float ez, float inv) {
        const float t = fminf(fmaxf((qx * ex + qy * ey + qz * ez) * inv, 0.0f), 1.0f);
        const float rx = qx - t * ex, ry = qy - t * ey, rz = qz - t * ez;
        return rx * rx + ry * ry + rz * rz;
    };
    const float s2 = fminf(fminf(seg(px, py, pz, b.x, b.y, b.z, b.w), seg(px, py, pz, c.x, c.y, c.z, c.w)),
                           seg(px - b.x, py - b.y, pz - b.z, c.x - b.x, c.y - b.y, c.z - b.z, u.w));
    const float n1 = fabsf(px) + fabsf(py) + fabsf(pz), l = rsqrtf(fminf(b.w, c.w));
    const float s = sqrtf(s2), E = 2.0e-6f * (scale + n1 + 2.0f * l + s) + 1.0e-12f;
    hi = s + E;
    lo = s - E;
    const float al = px * u.x + py * u.y + pz * u.z, be = px * v.x + py * v.y + pz * v.z, ga = 1.0f - be - al;
    const float tau = v.w * 1.0e-6f * (scale + n1);
    if (tau < 0.25f) {
        const float m = fminf(al, fminf(be, ga));
        if (m > -2.0f * tau) {
            const float wx = px - be * b.x - ga * c.x, wy = py - be * b.y - ga * c.y, wz = pz - be * b.z - ga * c.z;
            const float d = sqrtf(wx * wx + wy * wy + wz * wz);
            const float e = E + 4.0f * tau * l;
            lo = fminf(lo, d - e);
            if (m > 2.0f * tau) hi = fminf(hi, d + e);
        }
    } else {
        lo -= a.w;   // within the inradius of an edge
    }
    return make_float2(fmaxf(lo, 0.0f), hi);
}

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// FP32 enclosures of up to 48 triangles of a pnode: entry `lane` and `lane +
// 32`, infinite beyond the list
struct Encl {
    int e0, e1;            // entries of pent
    float lo0, hi0, lo1, hi1, lo, hi;   // and the least of each over the warp
};
__device__ __forceinline__ Encl enclose(const TriF* __restrict__ trif, const GeoTet* __restrict__ tets,
                                        const int* __restrict__ pent, int s, int n, const Pt& P, int lane) {
    Encl c;
    c.e0 = c.e1 = 0;
    c.lo0 = c.hi0 = c.lo1 = c.hi1 = 3.0e38f;
    if (lane < n) {
        c.e0 = __ldg(pent + s + lane);
        const float2 r = tri_interval(trif, tets, c.e0 >> 2, P.f[0], P.f[1], P.f[2], P.scale);
        c.lo0 = r.x;
        c.hi0 = r.y;
    }
    if (lane + 32 < n) {
        c.e1 = __ldg(pent + s + 32 + lane);
        const float2 r = tri_interval(trif, tets, c.e1 >> 2, P.f[0], P.f[1], P.f[2], P.scale);
        c.lo1 = r.x;
        c.hi1 = r.y;
    }
    c.lo = warp_min(fminf(c.lo0, c.lo1));
    c.hi = warp_min(fminf(c.hi0, c.hi1));
    return c;
}

// whether a triangle bounded by its box alone can lie below v
__device__ __forceinline__ bool box_only_near(const Encl& c, float v) {
    return __any_sync(0xffffffffu, (c.hi0 > 1.0e38f && c.lo0 <= v) || (c.hi1 > 1.0e38f && c.lo1 <= v));
}

// appends the entries chosen by t0 / t1 in order; returns the new task count
__device__ __forceinline__ int push_tasks(ChainQueue& Q, int nt, const Encl& c, bool t0, bool t1, int lane) {
    const unsigned m0 = __ballot_sync(0xffffffffu, t0), m1 = __ballot_sync(0xffffffffu, t1);
    const unsigned below = (1u << lane) - 1u;
    if (t0) Q.ent[nt + __popc(m0 & below)] = c.e0;
    if (t1) Q.ent[nt + __popc(m0) + __popc(m1 & below)] = c.e1;
    return nt + __popc(m0) + __popc(m1);
}

// (a call: one copy of the distance code for every place that flushes)
__device__ __noinline__ void eval_tasks(ChainQueue* Q, int nt, const GeoTet* __restrict__ tets, double px, double py,
                                        double pz) {
    const double P[3] = {px, py, pz};
    __syncwarp();
    for (int q = threadIdx.x & 31; q < nt; q += 32) {
        const int tri = Q->ent[q] >> 2;
        const GeoTet& T = tets[tri >> 1];
        Q->d[q] = dist_point_triangle(T.tri[tri & 1], T.tg[tri & 1], P);
    }
    __syncwarp();
}

// the +-4 box of a node, walked in k, j, i order 32 positions at a time
struct Box9 {
    int i0, j0, k0, ni, nj, n;
    __device__ __forceinline__ Box9(const DevGrid& g, int i, int j, int k) {
        i0 = max(i - 4, 0); j0 = max(j - 4, 0); k0 = max(k - 4, 0);
        ni = min(i + 4, g.ni - 1) - i0 + 1;
        nj = min(j + 4, g.nj - 1) - j0 + 1;
        n = ni * nj * (min(k + 4, g.nk - 1) - k0 + 1);
    }
    __device__ __forceinline__ long long node(const DevGrid& g, int q) const {
        const int r = q / ni;
        return gid(g, i0 + q - r * ni, j0 + r % nj, k0 + r / nj);
    }
};

// the pnodes' signed distances (src/GetIsosurfaceAndDistances.F90:166-330):
// a running minimum dp (from 10) over the triangles of the box's pnodes and,
// after each tetrahedron, sd <- sd + (dp - sd) where dp <= sd (from 99.9).
// In kSimple and kReset pnodes every update is exact, so dp is the least
// distance and sd follows it.  One more step after a kFull pnode brings sd
// to rest; it is made when another pnode (which has at least one
// tetrahedron) follows.
__global__ void __launch_bounds__(32 * kChainWarps, 8) k_geo_sd(
        DevGrid g, int npn, const long long* __restrict__ node_of, const int* __restrict__ ids,
        const GeoTet* __restrict__ tets, const TriF* __restrict__ trif, const int* __restrict__ pstart,
        const int* __restrict__ pent, const unsigned char* __restrict__ lead, const float4* __restrict__ prad,
        const double* __restrict__ phi, const double* __restrict__ x, const double* __restrict__ y,
        const double* __restrict__ z, double* __restrict__ sd_out) {
    __shared__ ChainQueue qs[kChainWarps];
    ChainQueue& Q = qs[threadIdx.x >> 5];
    const unsigned FM = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    for (int p = blockIdx.x * kChainWarps + (threadIdx.x >> 5); p < npn; p += gridDim.x * kChainWarps) {
        const long long l0 = node_of[p];
        int i, j, k;
        node_ijk(g, l0, &i, &j, &k);
        const Pt P = make_pt(x[l0], y[l0], z[l0]);
        const Box9 box(g, i, j, k);
        double dp = 10.0, sd = 99.9;          // exact state before the first queued pnode (kReset: replaced)
        float slo = 9.9f, shi = 100.0f;       // dp and sd after the last queued one lie between
        float dhi = 10.0f;                    // dp does not exceed
        int nt = 0, nitem = 0, ord = 0;
        int rest = -1;                        // ordinal of a kFull pnode (or the start) after which sd may not rest
        auto flush = [&]() {
            eval_tasks(&Q, nt, tets, P.d[0], P.d[1], P.d[2]);
            for (int it = 0; it < nitem; ++it) {
                const int t0 = Q.item[it] >> 2, kind = Q.item[it] & 3;
                const int t1 = it + 1 < nitem ? Q.item[it + 1] >> 2 : nt;
                const int o = Q.aux[it] >> 2;
                if (kind == kFull) {
                    if (rest > -2 && o - rest > 1) sd = mag_step(sd, dp);
                    if (Q.aux[it] & 3) sd = mag_step(sd, dp);
                    for (int q = t0; q < t1; ++q) {
                        const int e = Q.ent[q];
                        const float* bx = tets[e >> 3].box[(e >> 2) & 1];
                        if (!beyond_box(P.f, P.scale, bx, bx + 3, (float)dp)) dp = run_min(dp, Q.d[q]);
                        for (int st = e & 3; st > 0; --st) sd = mag_step(sd, dp);
                    }
                    rest = o;
                } else {
                    if (rest > -2) sd = mag_step(sd, dp);   // its first tetrahedron, or a pnode between
                    rest = -2;
                    LSM_CHAIN_CHECK(t1 > t0);
                    double m = Q.d[t0];
                    for (int q = t0 + 1; q < t1; ++q) m = dmin(m, Q.d[q]);
                    if (kind == kReset) {
                        dp = sd = m;
                    } else {
                        dp = dmin(dp, m);
                        sd = dmin(sd, dp);
                    }
                }
            }
            nt = nitem = 0;
            slo = 0.999999f * (float)fmin(dp, sd);
            shi = 1.000001f * (float)fmax(dp, sd);
            dhi = 1.000001f * (float)dp;
            __syncwarp();
        };
        for (int q0 = 0; q0 < box.n; q0 += 32) {
            const int q = q0 + lane;
            const int m0 = q < box.n ? ids[box.node(g, q)] - 1 : -1;
            const unsigned all = __ballot_sync(FM, m0 >= 0);
            const float lb = m0 >= 0 ? pnode_bound(m0, P, prad) : 3.0e38f;
            const bool in = !beyond(lb, P.scale, dhi);
            const int s0 = in ? pstart[m0] : 0, n0 = in ? pstart[m0 + 1] - s0 : 0, f0 = in ? lead[m0] : 0;
            unsigned near = __ballot_sync(FM, in);
            while (near) {
                const int b = __ffs(near) - 1;
                near &= near - 1;
                if (beyond(__shfl_sync(FM, lb, b), P.scale, dhi)) continue;
                const int s = __shfl_sync(FM, s0, b), n = __shfl_sync(FM, n0, b), fl = __shfl_sync(FM, f0, b);
                const int o = ord + __popc(all & ((1u << b) - 1u));
                Encl c = enclose(trif, tets, pent, s, n, P, lane);
                if (c.lo > dhi) continue;
                if (nt > kTasks - kMaxTri || nitem == kItems) {
                    flush();
                    if (c.lo > dhi) continue;   // (dhi is tighter now: an item would have no task)
                }
                const bool exact = c.lo >= 0.50001f * shi && !box_only_near(c, dhi);
                const int kind = !exact ? kFull : (c.hi < slo ? kReset : kSimple);
                if (kind == kReset) nt = nitem = 0;
                const float near_min = kind == kFull ? 3.0e38f : fminf(c.hi, dhi);
                if (lane == 0) {
                    Q.item[nitem] = 4 * nt + kind;
                    Q.aux[nitem] = 4 * o + fl;
                }
                ++nitem;
                nt = push_tasks(Q, nt, c, lane < n && c.lo0 <= near_min, lane + 32 < n && c.lo1 <= near_min, lane);
                // (kFull: the roundings of dp = 10 + (c - 10) and of sd stay below 1e-12)
                const bool below = c.hi < slo;
                slo = 0.999999f * (below ? c.lo : fminf(slo, c.lo)) - 1.0e-12f;
                shi = 1.000001f * fminf(shi, c.hi) + 1.0e-12f;
                dhi = 1.000001f * fminf(dhi, c.hi) + 1.0e-12f;
            }
            ord += __popc(all);
        }
        flush();
        if (rest > -2 && ord - 1 > rest) sd = mag_step(sd, dp);
        if (lane == 0) sd_out[p] = copysign(sd, sgn1(phi[l0]));
    }
}

// LocalVolumeVariation, src/TetrahedronMethods.F90:2390-2437
__device__ double local_dv(double eta, const double (&V)[4][3], const double (&ph)[4], double v0, unsigned* err) {
    double a[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] = ph[q] + eta;
    MT o;
    marching_full(V, a, o, false, err);
    return v0 - o.wv;
}

__device__ __forceinline__ void tet_vertices(const GeoTet& T, const long long* __restrict__ node_of,
                                             const double* __restrict__ x, const double* __restrict__ y,
                                             const double* __restrict__ z, double (&V)[4][3]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const long long l = node_of[T.v[q]];
        V[q][0] = x[l]; V[q][1] = y[l]; V[q][2] = z[l];
    }
}

// PiecewiseConstantFunction + SecantMethodLocalCorrection,
// src/PiecewiseConstantFunction.F90:1-102, src/TetrahedronMethods.F90:2439-2588
__global__ void k_geo_secant(int ntet, const GeoTet* __restrict__ tets, const long long* __restrict__ node_of,
                             const double* __restrict__ x, const double* __restrict__ y,
                             const double* __restrict__ z, const double* __restrict__ sd, double tol,
                             double* __restrict__ eta, unsigned* err) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntet; t += gridDim.x * blockDim.x) {
        const GeoTet T = tets[t];
        double V[4][3], ph[4];
        tet_vertices(T, node_of, x, y, z, V);
#pragma unroll
        for (int q = 0; q < 4; ++q) ph[q] = sd[T.v[q]];
        MT o;
        marching_full(V, ph, o, true, err);
        const double vol0 = T.wv, dv0 = vol0 - o.wv;
        double res = 0.0;
        if (!(fabs(dv0) < tol)) {
            double x0 = o.area > kEpsSims ? dv0 / o.area : 0.0;
            double x1 = T.area > kEpsSims ? dv0 / T.area : 0.0;
            double f0 = local_dv(x0, V, ph, vol0, err);
            double f1 = local_dv(x1, V, ph, vol0, err);
            if (fabs(f0) < tol || fabs(f1) < tol) {
                res = fabs(f1) < fabs(f0) ? x1 : x0;
            } else {
                bool conv = false;
                double x2 = 0.0;
                for (int it = 1; it <= 40; ++it) {
                    if (fabs(f1 - f0) < kEpsSims) break;
                    x2 = x1 - f1 * (x1 - x0) / (f1 - f0);
                    x0 = x1; x1 = x2; f0 = f1;
                    f1 = local_dv(x1, V, ph, vol0, err);
                    if (fabs(f1) < tol) { conv = true; break; }
                }
                if (fabs(f1) > dv0) x2 = 0.0;
                res = conv ? x2 : 0.0;
            }
        }
        eta[t] = res;
    }
}

// OrthogonalProjection, src/OrthogonalProjection.F90:1-49
__global__ void k_geo_xi(DevGrid g, int npn, const long long* __restrict__ node_of,
                         const unsigned char* __restrict__ cellbits, const int* __restrict__ tetbase,
                         const double* __restrict__ eta, double* __restrict__ xi) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npn; p += gridDim.x * blockDim.x) {
        int i, j, k;
        node_ijk(g, node_of[p], &i, &j, &k);
        int na = 0;
        for_each_tet(g, i, j, k, cellbits, tetbase, [&](int) { ++na; });
        const double dn = (double)na;
        double s = 0.0;
        for_each_tet(g, i, j, k, cellbits, tetbase, [&](int t) { s = s + eta[t] / dn; });
        xi[p] = s;
    }
}

// funcv's per-tetrahedron volume of phi* + C xi (src/NewtonRaphsonSolver.F90)
// and a per-block partial sum in fixed order
__global__ void __launch_bounds__(kThreads) k_geo_funcv(int ntet, const GeoTet* __restrict__ tets,
                                                        const long long* __restrict__ node_of,
                                                        const double* __restrict__ x, const double* __restrict__ y,
                                                        const double* __restrict__ z,
                                                        const double* __restrict__ sd,
                                                        const double* __restrict__ xi, double C,
                                                        double* __restrict__ part, unsigned* err) {
    __shared__ double red[kThreads];
    double acc = 0.0;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntet; t += gridDim.x * blockDim.x) {
        const GeoTet T = tets[t];
        double V[4][3], a[4];
        tet_vertices(T, node_of, x, y, z, V);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double s = sd[T.v[q]], ca = C * xi[T.v[q]];
            a[q] = s + ca / 2.0 * fabs(sgn1(s) + sgn1(s + ca));
        }
        MT o;
        marching_full(V, a, o, false, err);
        acc += o.wv;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = kThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void __launch_bounds__(kThreads) k_geo_sum(int n, const double* __restrict__ part,
                                                      double* __restrict__ out) {
    __shared__ double red[kThreads];
    double acc = 0.0;
    for (int b = threadIdx.x; b < n; b += kThreads) acc += part[b];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = kThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

// NeighboursPhiCorrection on the pnodes (src/NeighboursPhiCorrection.F90:142-184)
__global__ void k_geo_pnode_phi(int npn, const long long* __restrict__ node_of, const double* __restrict__ sd,
                                const double* __restrict__ xi, double C, double* __restrict__ pc) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npn; p += gridDim.x * blockDim.x) {
        const double s = sd[p], xv = xi[p];
        const double pcf = fabs(sgn1(s) + sgn1(s + C * xv)) / 2.0;
        const double aux = pcf * C * xv;
        pc[node_of[p]] = s + aux;
    }
}

// NeighboursPhiCorrection on the -1 nodes (src/NeighboursPhiCorrection.F90:
// 186-343): per pnode of the box a running minimum dp over its triangles,
// starting at 10 again, and after each of its tetrahedra |v| <- |v| + (dp -
// |v|) where dp <= |v|.  In kSimple and kReset pnodes every update of |v| is
// exact, so |v| becomes the pnode's last dp where that is lower; that is the
// least distance when an earlier triangle lies within a factor 2 of it, and
// follows from the first triangle and those not above it otherwise.
__global__ void __launch_bounds__(32 * kChainWarps, 8) k_geo_neigh(
        DevGrid g, const int* __restrict__ ids, const GeoTet* __restrict__ tets, const TriF* __restrict__ trif,
        const int* __restrict__ pstart, const int* __restrict__ pent, const unsigned char* __restrict__ lead,
        const float4* __restrict__ prad, const double* __restrict__ x, const double* __restrict__ y,
        const double* __restrict__ z, double* __restrict__ pc, int nsec, const long long* __restrict__ second) {
    __shared__ ChainQueue qs[kChainWarps];
    ChainQueue& Q = qs[threadIdx.x >> 5];
    const unsigned FM = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    for (int c0 = blockIdx.x * kChainWarps + (threadIdx.x >> 5); c0 < nsec; c0 += gridDim.x * kChainWarps) {
        const long long l0 = second[c0];
        int i, j, k;
        node_ijk(g, l0, &i, &j, &k);
        const Pt P = make_pt(x[l0], y[l0], z[l0]);
        const Box9 box(g, i, j, k);
        const double v0 = pc[l0];
        double av = fabs(v0);                 // exact |v| before the first queued pnode (kReset: replaced)
        float vlo, vhi;                       // |v| after the last queued one lies between
        int nt = 0, nitem = 0;
        auto bounds = [&]() {
            vlo = 0.999999f * (float)av;
            vhi = 1.000001f * (float)av;
        };
        bounds();
        auto flush = [&]() {
            eval_tasks(&Q, nt, tets, P.d[0], P.d[1], P.d[2]);
            for (int it = 0; it < nitem; ++it) {
                const int t0 = Q.item[it] >> 2, kind = Q.item[it] & 3;
                const int t1 = it + 1 < nitem ? Q.item[it + 1] >> 2 : nt;
                double dp = 10.0;
                if (kind == kFull) {
                    for (int st = Q.aux[it] & 3; st > 0; --st) av = mag_step(av, dp);
                    for (int q = t0; q < t1; ++q) {
                        const int e = Q.ent[q];
                        const float* bx = tets[e >> 3].box[(e >> 2) & 1];
                        if (!beyond_box(P.f, P.scale, bx, bx + 3, (float)dp)) dp = run_min(dp, Q.d[q]);
                        for (int st = e & 3; st > 0; --st) av = mag_step(av, dp);
                    }
                } else {
                    LSM_CHAIN_CHECK(t1 > t0);
                    dp = Q.aux[it] >> 2 ? Q.d[t0] : run_min(dp, Q.d[t0]);
                    for (int q = t0 + 1; q < t1; ++q) dp = run_min(dp, Q.d[q]);   // exact_min: the least
                    av = kind == kReset ? dp : dmin(av, dp);
                }
            }
            nt = nitem = 0;
            bounds();
            __syncwarp();
        };
        for (int q0 = 0; q0 < box.n; q0 += 32) {
            const int q = q0 + lane;
            const int m0 = q < box.n ? ids[box.node(g, q)] - 1 : -1;
            // a |v| of 10 or more follows dp = 10 after any tetrahedron; one that
            // is no number stays so: every test against 9.9999 fails for it
            const float lb = m0 >= 0 ? pnode_bound(m0, P, prad) : 3.0e38f;
            const bool in = m0 >= 0 && (!(vhi < 9.9999f) || !beyond(lb, P.scale, vhi));
            const int s0 = in ? pstart[m0] : 0, n0 = in ? pstart[m0 + 1] - s0 : 0, f0 = in ? lead[m0] : 0;
            unsigned near = __ballot_sync(FM, in);
            while (near) {
                const int b = __ffs(near) - 1;
                near &= near - 1;
                if (vhi < 9.9999f && beyond(__shfl_sync(FM, lb, b), P.scale, vhi)) continue;
                const int s = __shfl_sync(FM, s0, b), n = __shfl_sync(FM, n0, b), fl = __shfl_sync(FM, f0, b);
                Encl c = enclose(trif, tets, pent, s, n, P, lane);
                if (c.lo > vhi && vhi < 9.9999f) continue;
                if (nt > kTasks - kMaxTri || nitem == kItems) flush();
                // the steps with dp = 10 before the first triangle change no |v| below 10
                const bool exact = c.lo >= 0.50001f * vhi && vhi < 9.9999f && !box_only_near(c, vhi);
                const int kind = !exact ? kFull : (c.hi < vlo ? kReset : kSimple);
                if (kind == kReset) nt = nitem = 0;
                bool t0 = lane < n, t1 = lane + 32 < n;
                int exact_min = 0;
                if (kind != kFull) {
                    // the triangles that can be the pnode's least; an earlier
                    // one within a factor 2 of it makes the last dp their least
                    const bool w0 = t0 && c.lo0 <= c.hi, w1 = t1 && c.lo1 <= c.hi;
                    const unsigned b0 = __ballot_sync(FM, w0), b1 = __ballot_sync(FM, w1);
                    const int first = b0 ? __ffs(b0) - 1 : 31 + __ffs(b1);
                    exact_min = __any_sync(FM, (t0 && lane < first && c.hi0 <= 1.9999f * c.lo) ||
                                                   (t1 && lane + 32 < first && c.hi1 <= 1.9999f * c.lo));
                    // (otherwise: the first, and what can fall below it)
                    const float h = exact_min ? c.hi : __shfl_sync(FM, c.hi0, 0);
                    t0 = t0 && (c.lo0 <= h || (!exact_min && lane == 0));
                    t1 = t1 && c.lo1 <= h;
                }
                if (lane == 0) {
                    Q.item[nitem] = 4 * nt + kind;
                    Q.aux[nitem] = 4 * exact_min + fl;
                }
                ++nitem;
                nt = push_tasks(Q, nt, c, t0, t1, lane);
                if (!(vhi < 9.9999f)) {
                    flush();   // exact again at once: rare
                } else {
                    // (kFull: the rounding of dp = 10 + (c - 10) stays below 1e-12)
                    vlo = 0.999999f * (c.hi < vlo ? c.lo : fminf(vlo, c.lo)) - 1.0e-12f;
                    vhi = 1.000001f * fminf(vhi, c.hi) + 1.0e-12f;
                }
            }
        }
        flush();
        if (lane == 0) pc[l0] = copysign(av, v0);
    }
}

// levelsetmethod's phicorrected before the geometric step
// (src/levelsetmethod.F90:303-304): -9.9 where phi < -epsilon, 9.9 where
// phi > epsilon, the value in place elsewhere
__global__ void k_geo_seed(long long n, const double* __restrict__ phi, double* __restrict__ pc) {
    for (long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x; l < n;
         l += (long long)gridDim.x * blockDim.x) {
        const double f = phi[l];
        if (f < -kEpsSims) pc[l] = -9.9;
        if (f > kEpsSims) pc[l] = 9.9;
    }
}

}  // namespace
}  // namespace lsm
