// lsm_geometric.cu -- the hybrid path's geometric reinitialisation
// (src/geometric_reinitialisation.F90:1-94) on one GPU, FP64 with the
// reference's rounding (this unit is built with --fmad=false).
//
// The reference builds two linked structures on the host: a list of pnodes
// (vertices of phase-change tetrahedra, numbered in k, j, i order) and a list
// of K tetrahedra (numbered by cell in k, j, i order, then by tetrahedron
// 1..6 inside the cell), each pnode holding the ids of its K tetrahedra in
// the order they were appended.  Here both lists are dense device arrays
// made by two prefix sums:
//   - pnode ids: an exclusive scan of the per-node pnode flag, in the
//     node array's own (Fortran) order;
//   - K-tetrahedron ids: an exclusive scan of popcount(cell bits) over the
//     cells in the same order, plus the rank of the tetrahedron's bit inside
//     its cell.
// A pnode's tetrahedra are enumerated from the (at most) eight cells around
// the node, in increasing cell index and tetrahedron number, which is exactly
// the order GetTetrahedraList appends them (src/GetTetrahedraList.F90:322-446);
// their triangles are listed per pnode in that order.  The distance loops
// keep the results of the reference's sequential running-minimum updates per
// node (whose rounding depends on the order): one warp per node encloses the
// distances in FP32 and evaluates in FP64, in order, only those that the
// final bits can depend on (k_geo_sd, k_geo_neigh; lsm_geometric_dev.cuh).
#include <cuda_runtime.h>

#include "lsm_common.cuh"
#include "lsm_geometric.h"
#include "lsm_geometric_dev.cuh"
#include "lsm_kernels.h"

namespace lsm {
namespace {

int grid_for(long long n, int bs = kThreads) {
    long long b = (n + bs - 1) / bs;
    return (int)(b < 1 ? 1 : (b > 152LL * 64 ? 152LL * 64 : b));
}

}  // namespace

// ------------------------------------------------------------ host driver

void launch_geo_seed(long long n, const double* phi, double* pc, cudaStream_t s) {
    ProfScope ps("k_geo_seed", s);
    k_geo_seed<<<grid_for(n), kThreads, 0, s>>>(n, phi, pc);
}

#define GEO_CU(call)                                   \
    do {                                               \
        cudaError_t e_ = (call);                       \
        if (e_ != cudaSuccess) return e_;              \
    } while (0)

cudaError_t geo_reinit(const DevGrid& g, const double* phi0, const double* x, const double* y, const double* z,
                       double target, int gmc, double tol, double* pc, int* tag, GeoAlloc alloc, void* actx,
                       unsigned* d_err, int* d_count, GeoInfo* info, cudaStream_t s) {
    const long long n = (long long)g.ni * g.nj * g.nk;
    const int ntiles = (int)((n + kTile - 1) / kTile);
    cudaError_t e = cudaSuccess;
    auto* cellbits = static_cast<unsigned char*>(alloc(actx, "geo_cellbits", (size_t)n, &e));
    GEO_CU(e);
    auto* ids = static_cast<int*>(alloc(actx, "geo_ids", 4 * (size_t)n, &e));
    GEO_CU(e);
    auto* tetbase = static_cast<int*>(alloc(actx, "geo_tetbase", 4 * (size_t)n, &e));
    GEO_CU(e);
    auto* tiles = static_cast<int*>(alloc(actx, "geo_tiles", 4 * (size_t)ntiles + 16, &e));
    GEO_CU(e);
    // 1. cells: K-tetrahedra bits and pnode flags (ids holds the flags first)
    GEO_CU(cudaMemsetAsync(cellbits, 0, (size_t)n, s));
    GEO_CU(cudaMemsetAsync(ids, 0, 4 * (size_t)n, s));
    {
        ProfScope ps("k_geo_cells", s);
        k_geo_cells<<<grid_for(n), kThreads, 0, s>>>(g, phi0, cellbits, ids);
        GEO_CU(cudaGetLastError());
    }
    // 2. pnode ids: the flags -> tag (scratch), scanned back into ids
    GEO_CU(cudaMemcpyAsync(tag, ids, 4 * (size_t)n, cudaMemcpyDeviceToDevice, s));
    int counts[2] = {0, 0};
    {
        ProfScope ps("k_geo_scan", s);
        k_scan_tiles<0><<<ntiles, kThreads, 0, s>>>(n, tag, tiles);
        k_scan_top<<<1, kThreads, 0, s>>>(ntiles, tiles, d_count);
        GEO_CU(cudaGetLastError());
    }
    GEO_CU(cudaMemcpyAsync(&counts[0], d_count, sizeof(int), cudaMemcpyDeviceToHost, s));
    GEO_CU(cudaStreamSynchronize(s));
    const int npn = counts[0];
    auto* node_of = static_cast<long long*>(alloc(actx, "geo_node_of", 8 * (size_t)(npn + 1), &e));
    GEO_CU(e);
    {
        ProfScope ps("k_geo_scan", s);
        k_scan_apply<0><<<ntiles, kThreads, 0, s>>>(n, tag, tiles, ids, node_of);
        // 3. K-tetrahedra ids per cell
        k_scan_tiles<1><<<ntiles, kThreads, 0, s>>>(n, cellbits, tiles);
        k_scan_top<<<1, kThreads, 0, s>>>(ntiles, tiles, d_count + 1);
        GEO_CU(cudaGetLastError());
    }
    GEO_CU(cudaMemcpyAsync(&counts[1], d_count + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
    GEO_CU(cudaStreamSynchronize(s));
    const int ntet = counts[1];
    info->nnodes = npn;
    info->ntetrahedra = ntet;
    info->nsecond = 0;
    info->newton_iterations = 0;
    info->newton_converged = 0;
    info->C = 0.0;
    GEO_CU(cudaMemcpyAsync(tag, ids, 4 * (size_t)n, cudaMemcpyDeviceToDevice, s));
    if (npn == 0) return cudaSuccess;
    auto* tets = static_cast<GeoTet*>(alloc(actx, "geo_tets", sizeof(GeoTet) * (size_t)(ntet + 1), &e));
    GEO_CU(e);
    auto* tet_of = static_cast<long long*>(alloc(actx, "geo_tet_of", 8 * (size_t)(ntet + 1), &e));
    GEO_CU(e);
    auto* sd = static_cast<double*>(alloc(actx, "geo_sd", 8 * (size_t)npn, &e));
    GEO_CU(e);
    auto* xi = static_cast<double*>(alloc(actx, "geo_xi", 8 * (size_t)npn, &e));
    GEO_CU(e);
    auto* prad = static_cast<float4*>(alloc(actx, "geo_prad", 32 * (size_t)npn, &e));
    GEO_CU(e);
    auto* trif = static_cast<TriF*>(alloc(actx, "geo_trif", sizeof(TriF) * 2 * (size_t)(ntet + 1), &e));
    GEO_CU(e);
    // a triangle is listed by the four pnodes of its tetrahedron
    auto* pent = static_cast<int*>(alloc(actx, "geo_pent", 4 * 8 * (size_t)(ntet + 1), &e));
    GEO_CU(e);
    auto* ntri = static_cast<int*>(alloc(actx, "geo_ntri", 4 * (size_t)npn, &e));
    GEO_CU(e);
    auto* pstart = static_cast<int*>(alloc(actx, "geo_pstart", 4 * (size_t)(npn + 1), &e));
    GEO_CU(e);
    auto* lead = static_cast<unsigned char*>(alloc(actx, "geo_lead", (size_t)npn, &e));
    GEO_CU(e);
    {
        ProfScope ps("k_geo_tets", s);
        k_scan_apply<1><<<ntiles, kThreads, 0, s>>>(n, cellbits, tiles, tetbase, tet_of);
        k_geo_tets<<<grid_for(ntet, 64), 64, 0, s>>>(g, phi0, x, y, z, ntet, tet_of, ids, tets, trif, d_err);
        GEO_CU(cudaGetLastError());
    }
    {
        ProfScope ps("k_geo_mark", s);
        k_geo_mark<<<grid_for(npn), kThreads, 0, s>>>(g, npn, node_of, ids, tag);
        GEO_CU(cudaGetLastError());
    }
    {
        ProfScope ps("k_geo_prad", s);
        k_geo_prad<<<grid_for(npn), kThreads, 0, s>>>(g, npn, node_of, cellbits, tetbase, tets, prad, ntri);
        GEO_CU(cudaGetLastError());
    }
    {
        ProfScope ps("k_geo_fill", s);
        const int pt = (npn + kTile - 1) / kTile;
        k_scan_tiles<3><<<pt, kThreads, 0, s>>>(npn, ntri, tiles);
        k_scan_top<<<1, kThreads, 0, s>>>(pt, tiles, d_count + 3);
        k_scan_apply<3><<<pt, kThreads, 0, s>>>(npn, ntri, tiles, pstart, nullptr);
        k_geo_fill<<<grid_for(npn), kThreads, 0, s>>>(g, npn, node_of, cellbits, tetbase, tets, pstart, pent, lead);
        GEO_CU(cudaGetLastError());
    }
    {
        ProfScope ps("k_geo_sd", s);
        k_geo_sd<<<grid_for(npn, kChainWarps), 32 * kChainWarps, 0, s>>>(g, npn, node_of, ids, tets, trif, pstart, pent,
                                                                        lead, prad, phi0, x, y, z, sd);
        GEO_CU(cudaGetLastError());
    }
    GEO_CU(cudaMemsetAsync(xi, 0, 8 * (size_t)npn, s));
    double C = 0.0;
    if (gmc && ntet > 0) {
        auto* eta = static_cast<double*>(alloc(actx, "geo_eta", 8 * (size_t)ntet, &e));
        GEO_CU(e);
        const int nb = grid_for(ntet);
        auto* part = static_cast<double*>(alloc(actx, "geo_part", 8 * (size_t)nb + 64, &e));
        GEO_CU(e);
        {
            ProfScope ps("k_geo_secant", s);
            k_geo_secant<<<nb, kThreads, 0, s>>>(ntet, tets, node_of, x, y, z, sd, tol / 1000.0, eta, d_err);
            GEO_CU(cudaGetLastError());
        }
        {
            ProfScope ps("k_geo_xi", s);
            k_geo_xi<<<grid_for(npn), kThreads, 0, s>>>(g, npn, node_of, cellbits, tetbase, eta, xi);
            GEO_CU(cudaGetLastError());
        }
        double* d_sum = part + nb;
        cudaError_t fe = cudaSuccess;
        auto funcv = [&](double c) -> double {
            double tot = 0.0;
            if (fe != cudaSuccess) return 0.0;
            {
                ProfScope ps("k_geo_funcv", s);
                k_geo_funcv<<<nb, kThreads, 0, s>>>(ntet, tets, node_of, x, y, z, sd, xi, c, part, d_err);
                k_geo_sum<<<1, kThreads, 0, s>>>(nb, part, d_sum);
            }
            fe = cudaGetLastError();
            if (fe == cudaSuccess) fe = cudaMemcpyAsync(&tot, d_sum, sizeof(double), cudaMemcpyDeviceToHost, s);
            if (fe == cudaSuccess) fe = cudaStreamSynchronize(s);
            return target - tot;
        };
        int its = 0;
        bool conv = false;
        C = geo_newton(funcv, tol, &its, &conv);
        GEO_CU(fe);
        info->newton_iterations = its;
        info->newton_converged = conv ? 1 : 0;
        info->C = C;
    }
    {
        ProfScope ps("k_geo_pnode_phi", s);
        k_geo_pnode_phi<<<grid_for(npn), kThreads, 0, s>>>(npn, node_of, sd, xi, C, pc);
        GEO_CU(cudaGetLastError());
    }
    // the nodes tagged -1, listed in order
    {
        ProfScope ps("k_geo_scan", s);
        k_scan_tiles<2><<<ntiles, kThreads, 0, s>>>(n, tag, tiles);
        k_scan_top<<<1, kThreads, 0, s>>>(ntiles, tiles, d_count + 2);
        GEO_CU(cudaGetLastError());
    }
    int ns = 0;
    GEO_CU(cudaMemcpyAsync(&ns, d_count + 2, sizeof(int), cudaMemcpyDeviceToHost, s));
    GEO_CU(cudaStreamSynchronize(s));
    info->nsecond = ns;
    if (ns == 0) return cudaSuccess;
    auto* second = static_cast<long long*>(alloc(actx, "geo_second", 8 * (size_t)ns, &e));
    GEO_CU(e);
    {
        ProfScope ps("k_geo_scan", s);
        k_scan_apply<2><<<ntiles, kThreads, 0, s>>>(n, tag, tiles, nullptr, second);
        GEO_CU(cudaGetLastError());
    }
    {
        ProfScope ps("k_geo_neigh", s);
        k_geo_neigh<<<grid_for(ns, kChainWarps), 32 * kChainWarps, 0, s>>>(g, ids, tets, trif, pstart, pent, lead, prad,
                                                                           x, y, z, pc, ns, second);
        GEO_CU(cudaGetLastError());
    }
    GEO_CU(cudaStreamSynchronize(s));
    return cudaSuccess;
}

}  // namespace lsm
