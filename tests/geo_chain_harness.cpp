// Test harness (built by tests/test_geometric_chain_cpu.py): the device code of
// the geometric distance chains (csrc/lsm_geometric_dev.cuh) on the host's
// warp of fibers (tests/simt), against the sequential loops it stands for.
static long g_empty = 0;   // queued items without tasks
#define LSM_CHAIN_CHECK(ok) ((ok) ? (void)0 : (void)++g_empty)
#include "lsm_geometric_dev.cuh"

using namespace lsm;

namespace {

double sequential_sd(const DevGrid& g, int i, int j, int k, const int* ids, const unsigned char* cellbits,
                     const int* tetbase, const GeoTet* tets, const double* P, double phi) {
    double dp = 10.0, sd = 99.9;
    for (int c = max(k - 4, 0); c <= min(k + 4, g.nk - 1); ++c)
        for (int b = max(j - 4, 0); b <= min(j + 4, g.nj - 1); ++b)
            for (int a = max(i - 4, 0); a <= min(i + 4, g.ni - 1); ++a) {
                if (!ids[gid(g, a, b, c)]) continue;
                for_each_tet(g, a, b, c, cellbits, tetbase, [&](int t) {
                    const GeoTet& T = tets[t];
                    if (T.nis > 0 && T.area > 0.0)
                        for (int q = 0; q < T.nis; ++q)
                            dp = run_min(dp, dist_point_triangle(T.tri[q], T.tg[q], P));
                    sd = mag_step(sd, dp);
                });
            }
    return copysign(sd, sgn1(phi));
}

double sequential_neigh(const DevGrid& g, int i, int j, int k, const int* ids, const unsigned char* cellbits,
                        const int* tetbase, const GeoTet* tets, const double* P, double v) {
    double av = fabs(v);
    for (int c = max(k - 4, 0); c <= min(k + 4, g.nk - 1); ++c)
        for (int b = max(j - 4, 0); b <= min(j + 4, g.nj - 1); ++b)
            for (int a = max(i - 4, 0); a <= min(i + 4, g.ni - 1); ++a) {
                if (!ids[gid(g, a, b, c)]) continue;
                double dp = 10.0;
                for_each_tet(g, a, b, c, cellbits, tetbase, [&](int t) {
                    const GeoTet& T = tets[t];
                    if (T.nis > 0 && T.area > 0.0)
                        for (int q = 0; q < T.nis; ++q)
                            dp = run_min(dp, dist_point_triangle(T.tri[q], T.tg[q], P));
                    av = mag_step(av, dp);
                });
            }
    return copysign(av, v);
}

bool differ(double a, double b) { return !(std::isnan(a) && std::isnan(b)) && d2u(a) != d2u(b); }

}  // namespace

// Both chains at every node within `reach` index steps of (ci, cj, ck) and 9
// of which a pnode lies in the +-4 box; pc: |v| before (k_geo_neigh).
// counts: nodes compared, signed distances and |v| that differ, items without
// tasks, the largest relative difference in units of 1e-16
extern "C" int geo_chains(int ni, int nj, int nk, const double* phi, const double* x, const double* y, const double* z,
                          const double* pc, int ci, int cj, int ck, int reach, double* counts) {
    DevGrid g{};
    g.ni = ni; g.nj = nj; g.nk = nk;
    g.sj = ni; g.sk = (long long)ni * nj;
    g.ia = g.ja = g.ka = 0;
    g.ib = ni - 1; g.jb = nj - 1; g.kb = nk - 1;
    const long long n = (long long)ni * nj * nk;
    std::vector<unsigned char> cellbits(n, 0);
    std::vector<int> flags(n, 0), ids(n, 0), tetbase(n, 0);
    threadIdx = blockIdx = {0, 0, 0};
    blockDim = gridDim = {1, 1, 1};
    k_geo_cells(g, phi, cellbits.data(), flags.data());
    std::vector<long long> node_of, tet_of;
    for (long long l = 0; l < n; ++l) {
        if (flags[l]) { node_of.push_back(l); ids[l] = (int)node_of.size(); }
        tetbase[l] = (int)tet_of.size();
        for (unsigned m = cellbits[l]; m; m &= m - 1) tet_of.push_back(8 * l + __ffs((int)m) - 2);
    }
    const int npn = (int)node_of.size(), ntet = (int)tet_of.size();
    if (!npn) return 0;
    std::vector<GeoTet> tets(ntet + 1);
    std::vector<TriF> trif(2 * ntet + 2);
    std::vector<float4> prad(2 * npn);
    std::vector<int> ntri(npn), pstart(npn + 1, 0), pent(8 * (size_t)ntet + 8);
    std::vector<unsigned char> lead(npn);
    unsigned err = 0;
    k_geo_tets(g, phi, x, y, z, ntet, tet_of.data(), ids.data(), tets.data(), trif.data(), &err);
    k_geo_prad(g, npn, node_of.data(), cellbits.data(), tetbase.data(), tets.data(), prad.data(), ntri.data());
    for (int p = 0; p < npn; ++p) pstart[p + 1] = pstart[p] + ntri[p];
    k_geo_fill(g, npn, node_of.data(), cellbits.data(), tetbase.data(), tets.data(), pstart.data(), pent.data(), lead.data());
    gridDim = {1u << 28, 1, 1};   // a warp takes one node
    std::vector<double> sd(npn, 0.0), v(pc, pc + n);
    std::vector<long long> second;
    auto near = [&](long long l, int d) {
        int i, j, k;
        node_ijk(g, l, &i, &j, &k);
        return std::abs(i - ci) <= d && std::abs(j - cj) <= d && std::abs(k - ck) <= d;
    };
    for (long long l = 0; l < n; ++l)
        if (!flags[l] && near(l, reach)) second.push_back(l);
    g_empty = 0;
    auto note = [&](double got, double want, int c) {
        counts[0] += 1.0;
        if (!differ(got, want)) return;
        counts[c] += 1.0;
        const double r = fabs(got - want) / fabs(want) * 1e16;
        if (!(r <= counts[4])) counts[4] = r;
    };
    for (int p = 0; p < npn; ++p) {
        const long long l = node_of[p];
        if (!near(l, reach)) continue;
        blockIdx.x = p / kChainWarps;
        simt::run(32 * (p % kChainWarps), [&]() {
            k_geo_sd(g, npn, node_of.data(), ids.data(), tets.data(), trif.data(), pstart.data(), pent.data(),
                     lead.data(), prad.data(), phi, x, y, z, sd.data());
        });
        int i, j, k;
        node_ijk(g, l, &i, &j, &k);
        const double P[3] = {x[l], y[l], z[l]};
        note(sd[p], sequential_sd(g, i, j, k, ids.data(), cellbits.data(), tetbase.data(), tets.data(), P, phi[l]), 1);
    }
    const int nsec = (int)second.size();
    for (int s = 0; s < nsec; ++s) {
        const long long l = second[s];
        blockIdx.x = s / kChainWarps;
        simt::run(32 * (s % kChainWarps), [&]() {
            k_geo_neigh(g, ids.data(), tets.data(), trif.data(), pstart.data(), pent.data(), lead.data(), prad.data(),
                        x, y, z, v.data(), nsec, second.data());
        });
        int i, j, k;
        node_ijk(g, l, &i, &j, &k);
        const double P[3] = {x[l], y[l], z[l]};
        note(v[l], sequential_neigh(g, i, j, k, ids.data(), cellbits.data(), tetbase.data(), tets.data(), P, pc[l]), 2);
    }
    counts[3] += (double)g_empty;
    return npn;
}

// The FP32 enclosures of n triangles (9 doubles) seen from n points (3): the
// number that do not hold the FP64 distance; width[0]: the largest (hi - lo)
// in units of the distance + coordinates where both ends are finite
extern "C" long geo_enclosures(long n, const double* T, const double* P, double* width) {
    long missed = 0;
    for (long q = 0; q < n; ++q) {
        GeoTet t{};
        TriF f;
        for (int c = 0; c < 9; ++c) t.tri[0][c] = T[9 * q + c];
        tri_geo(t.tri[0], t.tg[0]);
        tri_f32(t.tri[0], t.tg[0], f);
        for (int c = 0; c < 3; ++c) {
            const double a = t.tri[0][c], b = t.tri[0][3 + c], e = t.tri[0][6 + c];
            t.box[0][c] = __double2float_rd(fmin(a, fmin(b, e)));
            t.box[0][3 + c] = __double2float_ru(fmax(a, fmax(b, e)));
        }
        const Pt p = make_pt(P[3 * q], P[3 * q + 1], P[3 * q + 2]);
        const float2 r = tri_interval(&f, &t, 0, p.f[0], p.f[1], p.f[2], p.scale);
        const double d = dist_point_triangle(t.tri[0], t.tg[0], P + 3 * q);
        if (!((double)r.x <= d && d <= (double)r.y)) ++missed;
        if (r.y < 1e37f) width[0] = fmax(width[0], ((double)r.y - (double)r.x) / (d + (double)p.scale));
    }
    return missed;
}
