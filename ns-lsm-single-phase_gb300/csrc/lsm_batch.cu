// lsm_batch.cu -- batched kernels of the level-set transport step, forward
// and adjoint, templated on the scalar type (FP32 for throughput, FP64 for
// gradient checks).
//
// Every launch covers every instance of the batch with persistent CTAs
// (grid = SMs x resident CTAs) walking a table of tiles, each tile inside
// one instance:
//  - brick tables (TX x TY x TZ nodes, one thread per node; the autotuned
//    forward shape): contra, boundary passes, and the brick variants of the
//    pseudo-step;
//  - flat tiles (columns of an instance in row-major order over the threads,
//    marching in k or j): RK stage, pseudo-steps in pairs, stage adjoint, the
//    reverse pseudo-step from stored coefficients;
//  - adjoint-map tiles (adj_shape): k marches over 32 x 8 columns (single
//    pseudo-steps, volume scan, TMA stage) or an overlapped 32 x kReinRY tile
//    (reverse pseudo-step recomputing its coefficients).
// Per-node algorithmic traffic (FP32 words): contra 15 (u 3, metrics 9;
// W 3), RK stage 5/6/6 (phi_prev, phi^n, W 3; phi), pseudo-step 12 (d, s,
// metrics 9; d; a pair 12 for both) or 18 recorded (+ six adjoint
// coefficients), volume 3 (phi
// + 64-bit fixed-point cell volume).
//
// Arithmetic: the reference's formulas rearranged for the GPU (one division
// per WENO3 reconstruction); the water volume sums FP64 hexahedron volumes
// of the bulk water cells and the interface cells' shares (in the stencil
// precision) with exact 64-bit fixed-point sums.  The reinitialisation uses
// the closed form of the reference's method-0 lambda correction: with
// lambda = -(d1 - phi0) / (dtau delta |grad phi0|) the correction dtau
// lambda delta |grad phi0| returns d to phi0 wherever delta(phi0) |grad
// phi0| != 0, i.e. |phi0| < eps; those nodes are folded into the sign field
// as s = 0 (no update) and a pseudo-step reads only d, s and the metrics.
//
// Adjoint: hand-written reverse kernels gathering (no atomics): bcond_lsm
// faces in reverse order; the WENO3 stage with the upwind side of every
// face frozen from the forward pass and the nonlinear weights
// differentiated; the Godunov pseudo-step with its max / clip selections
// and the sign field frozen (a 7-point stencil on lam with coefficients the
// recorded forward step stored, or recomputed from its input); the
// contravariant-velocity chain rule.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "lsm_batch.cuh"
#include "lsm_batch_scalar.cuh"
#include "lsm_common.cuh"
#include "lsm_kernels.h"
#include "lsm_soft64.cuh"
#include "lsm_volume_dev.cuh"

namespace lsm {
namespace batch {
namespace {

// per-instance parameter in the kernel's precision
template <typename T> __device__ __forceinline__ T ipar(float f, double d);
template <> __device__ __forceinline__ float ipar<float>(float f, double) { return f; }
template <> __device__ __forceinline__ double ipar<double>(float, double d) { return d; }

// element at a byte offset from an array's base (of 32 bits: one instruction,
// the base in a uniform register)
template <typename T, typename O> __device__ __forceinline__ T ldo(const T* p, O o) {
    return __ldg(reinterpret_cast<const T*>(reinterpret_cast<const char*>(p) + o));
}
// the same from an array that the kernel writes
template <typename T, typename O> __device__ __forceinline__ T ldv(const T* p, O o) {
    return *reinterpret_cast<const T*>(reinterpret_cast<const char*>(p) + o);
}
template <typename T, typename O> __device__ __forceinline__ void sto(T* p, O o, T v) {
    *reinterpret_cast<T*>(reinterpret_cast<char*>(p) + o) = v;
}

// ------------------------------------------------------------ node walks
struct Node {
    int inst, i, j, k;
    bool valid;
};

template <int TX, int TY, int TZ>
__device__ __forceinline__ Node brick_node(const Inst* __restrict__ inst, const Brick* __restrict__ bricks, int blk) {
    Node b;
    const int4 bk = __ldg(reinterpret_cast<const int4*>(bricks) + blk);
    b.inst = bk.x;
    const Inst& I = inst[b.inst];
    const int t = threadIdx.x;
    b.i = bk.y * TX + t % TX;
    b.j = bk.z * TY + (t / TX) % TY;
    b.k = bk.w * TZ + t / (TX * TY);
    b.valid = b.i < I.ni && b.j < I.nj && b.k < I.nk;
    return b;
}

// flat walk: node t of the packed arrays -> instance and (i, j, k)
__device__ __forceinline__ bool flat_node(const Flat& fl, long long t, Node* nd) {
    if (t >= fl.n) return false;
    int lo = 0, hi = fl.ninst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (fl.offs[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const Inst& I = fl.inst[lo];
    const long long r = t - I.off;
    nd->inst = lo;
    nd->i = (int)(r % I.ni);
    nd->j = (int)((r / I.ni) % I.nj);
    nd->k = (int)(r / ((long long)I.ni * I.nj));
    nd->valid = true;
    return true;
}

// Brick `blk` of an adjoint map: instance and first node of its tile.
struct ABrick {
    int inst, i0, j0, k0;
};
__device__ __forceinline__ ABrick adj_brick(const Tiles& tl, int blk) {
    const int4 bk = __ldg(reinterpret_cast<const int4*>(tl.b) + blk);
    return ABrick{bk.x, bk.y, bk.z, bk.w};
}

// ------------------------------------------------------------ contra
template <typename T, int TX, int TY, int TZ>
__global__ void __launch_bounds__(TX * TY * TZ) k_contra(const Inst* __restrict__ inst,
        const Brick* __restrict__ bricks, int nbricks, FieldsT<T> f) {
    for (int blk = blockIdx.x; blk < nbricks; blk += gridDim.x) {
        const Node b = brick_node<TX, TY, TZ>(inst, bricks, blk);
        if (!b.valid) continue;
        const Inst& I = inst[b.inst];
        const long long l = I.off + b.i + (long long)I.ni * (b.j + (long long)I.nj * b.k);
        const T u = f.u[0][l], v = f.u[1][l], w = f.u[2][l];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const T c = f.m[3 * m][l] * u + f.m[3 * m + 1][l] * v + f.m[3 * m + 2][l] * w;
            f.W[m][l] = ipar<T>(I.dt, I.dt64) * c;
        }
    }
}

// FP64 contravariant velocity x dt of one instance from the FP64 metrics
// (m64: 9 arrays) and velocity (u64: 3 arrays), the same formula as
// k_contra; packed base arrays, `off` the instance's first node
__global__ void k_w64(long long off, long long n, double dt, const double* const* __restrict__ m64,
                      const double* const* __restrict__ u64, double* const* __restrict__ w64) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const long long l = off + t;
        const double u = u64[0][l], v = u64[1][l], w = u64[2][l];
#pragma unroll
        for (int m = 0; m < 3; ++m) w64[m][l] = dt * (m64[3 * m][l] * u + m64[3 * m + 1][l] * v + m64[3 * m + 2][l] * w);
    }
}

// ------------------------------------------------------------ RK stage

// The stage output c1 phi^n + c2 phi1 - c3 R at node l.  FP32 batches that
// keep the FP64 contravariant velocity combine the nodes within kBand64 eps
// of the interface in FP64: R = sum_m W64_m D_m over the FP32 differences D.
template <typename T>
__device__ __forceinline__ T stage_out(const FieldsT<T>& f, long long l, bool interior, T c1, T c2, T c3, T pn, T w2,
                                       T R, T D0, T D1, T D2, T eps) {
    if constexpr (sizeof(T) == 4) {
        if (interior && f.W64[0] && fabsf(w2) < kBand64 * eps)
            return stage_band(__ldg(f.W64[0] + l), __ldg(f.W64[1] + l), __ldg(f.W64[2] + l), D0, D1, D2, c1, c2, c3, pn,
                              w2);
    }
    return c1 * pn + c2 * w2 - c3 * R;
}

// RK stage: interior nodes out = c1 phi^n + c2 phi1 - c3 sum_m W_m (Phi+ -
// Phi-)_m (calc_RH_AD_WENO3 x aj dt, the x term first), other nodes with a sum
// of 0; their faces come from bcond_lsm afterwards.  On flat tiles: sw x sh
// columns of one instance (Inst; whole rows or parts of them), in row-major
// order over the threads, so that few lanes idle where the instance's width is
// no multiple of 32; each thread marches in k with the z stencil in a register
// window.
// What bounds it is the issue of its instructions, and the warps that wait
// where some hold interface nodes (stage_band).  So a face's operations are
// few (weno_wind), neighbours are loaded by the wind's side, the x and y ones
// plainly: the window has brought their lines to L1 three planes before, and
// no warp waits for another at a barrier.  Offsets are bytes of type O, 32 bits
// where an array has fewer than 2^32 (one instruction per access), and two
// planes per turn of the loop keep a plane's registers in their places.
// Measured against tiles of 32 x 8 staged in shared memory: 64 grids of 32..96
// 242 -> 150 us, 512 x 256 x 256 301 -> 238 us, 128^3 31 -> 18 us, two FP64
// grids of 40^3 60 -> 25 us; six blocks per SM (five: 165 us on the 64 grids,
// seven: 158 us).
template <typename T, typename O>
__global__ void __launch_bounds__(kStageThreads, sizeof(T) == 4 ? kStageBlocks : 2) k_stage(const Inst* __restrict__ inst,
        Tiles tl, FieldsT<T> f, const T* __restrict__ phin, const T* __restrict__ phi1, T* __restrict__ out, T c1, T c2, T c3) {
    struct Pl {
        T W0, W1, W2, pn;
    };
    const int t = threadIdx.x;
    for (int blk = blockIdx.x; blk < tl.n; blk += gridDim.x) {
        const ABrick ab = adj_brick(tl, blk);
        const Inst& I = inst[ab.inst];
        const int ni = I.ni, nj = I.nj, nk = I.nk;
        const int y = t / I.sw, x = t - y * I.sw;
        const int i = ab.i0 + x, j = ab.j0 + y;
        const bool col = y < I.sh && i < ni && j < nj;
        const int k0 = ab.k0, k1 = min(k0 + tl.len, nk);
        constexpr O E = sizeof(T);
        const O sj = E * (O)ni, sk = sj * (O)nj;
        O l = E * (O)I.off + sk * (O)k0 + E * (O)i + sj * (O)j;   // plane k
        const bool ij_int = col && i > 0 && i < ni - 1 && j > 0 && j < nj - 1;
        const bool ilo = i == 1, ihi = i == ni - 2, jlo = j == 1, jhi = j == nj - 2;
        const T eps = ipar<T>(I.eps, I.eps64);
        T w0 = T(0), w1 = T(0), w2 = T(0), w3 = T(0), w4 = T(0);
        Pl a, b;
        auto ld = [&](Pl& p, O l) {
            p.W0 = ldo(f.W[0], l);
            p.W1 = ldo(f.W[1], l);
            p.W2 = ldo(f.W[2], l);
            p.pn = ldo(phin, l);
        };
        if (col) {
            if (k0 > 1) w0 = ldo(phi1, l - 2 * sk);
            if (k0 > 0) w1 = ldo(phi1, l - sk);
            w2 = ldo(phi1, l);
            if (k0 + 1 < nk) w3 = ldo(phi1, l + sk);
            if (k0 + 2 < nk) w4 = ldo(phi1, l + 2 * sk);
            ld(a, l);
        }
        auto plane = [&](int k, const Pl& c, Pl& n) {
            T w5 = T(0);
            if (col && k + 1 < k1) {
                if (k + 3 < nk) w5 = ldo(phi1, l + 3 * sk);
                ld(n, l + sk);
            }
            const bool interior = ij_int && k > 0 && k < nk - 1;
            T R = T(0), D0 = T(0), D1 = T(0), D2 = T(0);
            if (interior) {
                // in the array for every interior node; q0 is not used at an edge
                const bool ux = c.W0 > T(0), uy = c.W1 > T(0), uz = c.W2 > T(0);
                const O ox = ux ? E : O(0) - E, oy = uy ? sj : O(0) - sj;
                const T x0 = ldo(phi1, l - 2 * ox), x1 = ldo(phi1, l - ox), x3 = ldo(phi1, l + ox);
                const T y0 = ldo(phi1, l - 2 * oy), y1 = ldo(phi1, l - oy), y3 = ldo(phi1, l + oy);
                D2 = weno_wind(uz ? w0 : w4, uz ? w1 : w3, w2, uz ? w3 : w1, uz ? k == 1 : k == nk - 2);
                D0 = weno_wind(x0, x1, w2, x3, ux ? ilo : ihi);
                D1 = weno_wind(y0, y1, w2, y3, uy ? jlo : jhi);
                R = fabs(c.W0) * D0;
                R = vfma(fabs(c.W1), D1, R);
                R = vfma(fabs(c.W2), D2, R);
                if (!ux) D0 = -D0;
                if (!uy) D1 = -D1;
                if (!uz) D2 = -D2;
            }
            if (col) sto(out, l, stage_out(f, (long long)(l / E), interior, c1, c2, c3, c.pn, w2, R, D0, D1, D2, eps));
            w0 = w1;
            w1 = w2;
            w2 = w3;
            w3 = w4;
            w4 = w5;
            l += sk;
        };
        for (int k = k0;;) {
            plane(k, a, b);
            if (++k >= k1) break;
            plane(k, b, a);
            if (++k >= k1) break;
        }
    }
}

// ------------------------------------------------------------ TMA staging
// Tensor-memory-accelerator copies of one tile per plane into shared memory
// (cp.async.bulk.tensor), completion tracked by an mbarrier whose phase the
// threads wait on, each wait bounded (kErrTimeout after kTmaSpins polls).
constexpr int kTmaSpins = 1 << 20;
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait for phase `parity` of `bar`; false when it gave up
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
    for (int it = 0; it < kTmaSpins; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// 4-D tiled load (x, y, z, array) of the map's box into dst, completing on bar
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int x, int y, int z, int a,
                                            unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(a), "r"(smem_addr(bar))
        : "memory");
}

// RK stage (FP32) with the plane tiles staged by TMA: the same arithmetic (the
// same bits as k_stage), on the tiles of adjoint map 1 (32 x 8 columns) with
// the z stencil in a register window, for a batch of one instance whose rows
// are whole 16-byte units (ni a multiple of 4).  The z face k - 1/2 is
// carried from the plane below where the upwind choices agree, and a warp
// skips its evaluation where all lanes' do.  The stage input phi1 is
// array `a_in` of the 4-D tensor map `tm` ((ni, nj, nk, arrays), the
// arena's arrays ld apart).  Per plane one thread issues the copy of a 40 x
// 12 box starting at (i0 - 4, j0 - 2): x rounded down to a 16-byte boundary,
// a two-node halo on every side, the out-of-range part zero-filled by the
// copy engine.  Three buffers; the copy of plane k + 2 is issued (after the
// plane barrier that frees its buffer) while plane k is computed.
constexpr int kTmaBX = 40, kTmaBY = 12, kTmaBuf = 3;
__global__ void __launch_bounds__(256) k_stage_tma(const __grid_constant__ CUtensorMap tm, int a_in,
        const Inst* __restrict__ inst, Tiles tl, FieldsT<float> f,
        const float* __restrict__ phin, const float* __restrict__ phi1, float* __restrict__ out, float c1, float c2,
        float c3, unsigned* __restrict__ err) {
    __shared__ __align__(128) float pl[kTmaBuf][kTmaBY][kTmaBX];
    __shared__ __align__(8) unsigned long long bar[kTmaBuf];
    __shared__ int abort_flag;
    const unsigned FM = 0xffffffffu;
    const int t = threadIdx.x, tx = t & 31, ty = t >> 5;
    constexpr unsigned kBytes = kTmaBX * kTmaBY * sizeof(float);
    if (t == 0) {
        for (int b = 0; b < kTmaBuf; ++b) mbar_init(&bar[b], 1);
        abort_flag = 0;
        mbar_fence_init();
    }
    __syncthreads();
    unsigned issued = 0, used = 0;   // copies issued / planes consumed by this CTA (same on every thread)
    const Inst& I = inst[0];
    const int ni = I.ni, nj = I.nj, nk = I.nk;
    const long long sk = (long long)ni * nj;
    auto issue = [&](int i0, int j0, int k) {
        if (t == 0) {
            unsigned long long* b = &bar[issued % kTmaBuf];
            mbar_expect_tx(b, kBytes);
            tma_load_4d(&pl[issued % kTmaBuf][0][0], &tm, i0 - 4, j0 - 2, k, a_in, b);
        }
        ++issued;
    };
    bool aborted = false;
    for (int blk = blockIdx.x; blk < tl.n && !aborted; blk += gridDim.x) {
        const ABrick ab = adj_brick(tl, blk);
        const int i = ab.i0 + tx, j = ab.j0 + ty;
        const int k0 = ab.k0, k1 = min(k0 + tl.len, nk);
        const bool col = i < ni && j < nj;
        const long long cb = i + (long long)ni * j;
        const bool ij_int = i > 0 && i < ni - 1 && j > 0 && j < nj - 1;
        // the first two planes of the tile
        issue(ab.i0, ab.j0, k0);
        if (k0 + 1 < k1) issue(ab.i0, ab.j0, k0 + 1);
        auto own = [&](int k) { return col && k >= 0 && k < nk ? __ldg(phi1 + cb + sk * k) : 0.f; };
        float w0 = own(k0 - 2), w1 = own(k0 - 1), w2 = own(k0), w3 = own(k0 + 1), w4 = own(k0 + 2);
        float W0 = 0.f, W1 = 0.f, W2 = 0.f, pn = 0.f;
        if (col) {
            const long long l = cb + sk * k0;
            W0 = __ldg(f.W[0] + l);
            W1 = __ldg(f.W[1] + l);
            W2 = __ldg(f.W[2] + l);
            pn = __ldg(phin + l);
        }
        float fpz = 0.f;
        bool Pz = false, have = false;
        for (int k = k0; k < k1; ++k) {
            const bool nx = k + 1 < k1;
            const float w5 = nx ? own(k + 3) : 0.f;
            float W0n = 0.f, W1n = 0.f, W2n = 0.f, pnn = 0.f;
            if (col && nx) {
                const long long l = cb + sk * (k + 1);
                W0n = __ldg(f.W[0] + l);
                W1n = __ldg(f.W[1] + l);
                W2n = __ldg(f.W[2] + l);
                pnn = __ldg(phin + l);
            }
            const unsigned slot = used % kTmaBuf, par = (used / kTmaBuf) & 1u;
            // a wait that gave up leaves `used` at the copy still owed
            if (mbar_wait(&bar[slot], par)) ++used;
            else abort_flag = 1;
            const float (*P)[kTmaBX] = pl[slot];
            const bool interior = col && ij_int && k > 0 && k < nk - 1;
            const bool upz = W2 > 0.f;
            const bool Pk = upz || k == nk - 2, Mk = upz && k != 1;
            const bool reuse = !interior || (have && Mk == Pz);
            const bool all_reuse = __all_sync(FM, reuse);
            if (col) {
                float R = 0.f;
                float D0 = 0.f, D1 = 0.f, D2 = 0.f;
                if (interior) {
                    const int x = tx + 4, y = ty + 2;
                    // the outer stencil values are read unconditionally: the
                    // tile always holds them (zero-filled outside the grid),
                    // and weno_diff leaves m2 unused at the first interior node
                    // and p2 at the last
                    D0 = weno_diff(P[y][x - 2], P[y][x - 1], w2, P[y][x + 1], P[y][x + 2], W0, i == 1, i == ni - 2);
                    D1 = weno_diff(P[y - 2][x], P[y - 1][x], w2, P[y + 1][x], P[y + 2][x], W1, j == 1, j == nj - 2);
                    const float p2 = w4;
                    const float fp = rec3(Pk ? w1 : p2, Pk ? w2 : w3, Pk ? w3 : w2);
                    float fm = fpz;
                    if (!all_reuse) {
                        const float g = rec3(Mk ? w0 : w3, Mk ? w1 : w2, Mk ? w2 : w1);
                        if (!reuse) fm = g;
                    }
                    D2 = fp - fm;
                    R = W0 * D0;
                    R = vfma(W1, D1, R);
                    R = vfma(W2, D2, R);
                    fpz = fp;
                    Pz = Pk;
                }
                out[cb + sk * k] = stage_out(f, cb + sk * k, interior, c1, c2, c3, pn, w2, R, D0, D1, D2, I.eps);
            }
            have = interior;
            // every thread is done with this plane's buffer: it takes plane k + 2
            __syncthreads();
            if (abort_flag) {
                aborted = true;
                break;
            }
            if (k + 2 < k1) issue(ab.i0, ab.j0, k + 2);
            w0 = w1;
            w1 = w2;
            w2 = w3;
            w3 = w4;
            w4 = w5;
            W0 = W0n;
            W1 = W1n;
            W2 = W2n;
            pn = pnn;
        }
    }
    if (aborted && t == 0) {
        atomicOr(err, (unsigned)kErrTimeout);
        // let the copies still in flight land before the CTA's shared memory
        // goes away (each wait bounded again)
        while (used < issued) {
            mbar_wait(&bar[used % kTmaBuf], (used / kTmaBuf) & 1u);
            ++used;
        }
    }
}

// ------------------------------------------------------------ bcond_lsm
template <typename T>
__device__ __forceinline__ T bc_rule(int type, T n1, T n2, float BigPhi) {
    if (type == 0) return n1;
    if (type == 1) return fabs(n2) >= T(BigPhi) ? n1 : T(4.0 / 3.0) * n1 - T(1.0 / 3.0) * n2;
    return T(2) * n1 - n2;  // type 2 on the im face
}
__device__ __forceinline__ bool face_on(const BC& bc, int face) {
    const int t = bc.type[face];
    return t == 0 || t == 1 || (t == 2 && face == 1);
}

// Value of node (i, j, k) after the first `axes` axes' faces of bcond_lsm
// (i, then j, then k), from the pre-BC field p0: per axis whose face rule
// applies, the rule on the two nodes inward, eight nodes for a corner and two
// for a node of one face.  ONE: one evaluation of p0 in a loop for a field
// that is costly to evaluate (the last pseudo-step: k_bc_reinit 101 us on 64
// grids of 32..96 with all nested calls inlined, 40 us so); otherwise the
// nodes' loads go out together, those not needed predicated off (k_bc_stage
// 32.7 us, 29.0 us).
template <typename T, bool ONE, class P0>
__device__ __forceinline__ T bc_value(const BC& bc, const P0& p0, int ni, int nj, int nk, int i, int j, int k,
                                      int axes = 3) {
    auto dir = [&](int c, int n, int face) { return c == 0 && face_on(bc, face) ? 1 : (c == n - 1 && face_on(bc, face + 1) ? -1 : 0); };
    const int di = axes > 0 ? dir(i, ni, 0) : 0, dj = axes > 1 ? dir(j, nj, 2) : 0, dk = axes > 2 ? dir(k, nk, 4) : 0;
    const int ti = bc.type[di < 0 ? 1 : 0], tj = bc.type[dj < 0 ? 3 : 2], tk = bc.type[dk < 0 ? 5 : 4];
    if constexpr (ONE) {
        if ((di != 0) + (dj != 0) + (dk != 0) == 1) {   // one face: both values in flight at once
            const T v1 = p0(i + di, j + dj, k + dk), v2 = p0(i + 2 * di, j + 2 * dj, k + 2 * dk);
            return bc_rule<T>(di ? ti : dj ? tj : tk, v1, v2, bc.BigPhi);
        }
        T vk = T(0);
#pragma unroll 1
        for (int a = 0; a < (dk ? 2 : 1); ++a) {
            T vj = T(0);
#pragma unroll 1
            for (int b = 0; b < (dj ? 2 : 1); ++b) {
                T vi = T(0);
#pragma unroll 1
                for (int c = 0; c < (di ? 2 : 1); ++c) {
                    const T v = p0(di ? i + di * (c + 1) : i, dj ? j + dj * (b + 1) : j, dk ? k + dk * (a + 1) : k);
                    vi = c == 0 ? v : bc_rule<T>(ti, vi, v, bc.BigPhi);
                }
                vj = b == 0 ? vi : bc_rule<T>(tj, vj, vi, bc.BigPhi);
            }
            vk = a == 0 ? vj : bc_rule<T>(tk, vk, vj, bc.BigPhi);
        }
        return vk;
    } else {
        T v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int c = q & 1, b = (q >> 1) & 1, a = q >> 2;
            v[q] = T(0);
            if ((!c || di) && (!b || dj) && (!a || dk)) v[q] = p0(i + di * (c + 1), j + dj * (b + 1), k + dk * (a + 1));
        }
#pragma unroll
        for (int q = 0; q < 8; q += 2)
            if (di) v[q] = bc_rule<T>(ti, v[q], v[q + 1], bc.BigPhi);
#pragma unroll
        for (int q = 0; q < 8; q += 4)
            if (dj) v[q] = bc_rule<T>(tj, v[q], v[q + 2], bc.BigPhi);
        return dk ? bc_rule<T>(tk, v[0], v[4], bc.BigPhi) : v[0];
    }
}

template <typename T>
struct P0Stage {
    const T *phin, *phi1, *out;
    long long off, sj, sk;
    int ni, nj, nk;
    T c1, c2;
    __device__ T operator()(int i, int j, int k) const {
        const long long l = off + i + sj * j + sk * k;
        const bool bnd = i == 0 || i == ni - 1 || j == 0 || j == nj - 1 || k == 0 || k == nk - 1;
        return bnd ? c1 * phin[l] + c2 * phi1[l] : out[l];
    }
};
template <typename T>
struct P0Src {
    const T* src;
    long long off, sj, sk;
    __device__ T operator()(int i, int j, int k) const { return src[off + i + sj * j + sk * k]; }
};

__device__ __forceinline__ int face_instance(const Inst* __restrict__ inst, int ninst, long long t) {
    int lo = 0, hi = ninst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (inst[mid].face0 <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ bool face_coords(const Inst& I, unsigned r, int* pi, int* pj, int* pk) {
    // an instance's face nodes number below 2^32, as its nodes do
    const unsigned ni = I.ni, nj = I.nj, nk = I.nk, nI = nj * nk, nJ = ni * nk, nK = ni * nj;
    if (r < 2 * nI) { *pi = r < nI ? 0 : I.ni - 1; r = r < nI ? r : r - nI; *pj = (int)(r % nj); *pk = (int)(r / nj); return true; }
    r -= 2 * nI;
    if (r < 2 * nJ) { *pj = r < nJ ? 0 : I.nj - 1; r = r < nJ ? r : r - nJ; *pi = (int)(r % ni); *pk = (int)(r / ni); return true; }
    r -= 2 * nJ;
    if (r >= 2 * nK) return false;
    *pk = r < nK ? 0 : I.nk - 1; r = r < nK ? r : r - nK; *pi = (int)(r % ni); *pj = (int)(r / ni);
    return true;
}

template <typename T>
__global__ void k_bc_stage(const Inst* __restrict__ inst, int ninst, long long nface, BC bc,
                           const T* __restrict__ phin, const T* __restrict__ phi1, T* out, T c1, T c2) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= nface) return;
    const Inst& I = inst[face_instance(inst, ninst, t)];
    int i, j, k;
    if (!face_coords(I, (unsigned)(t - I.face0), &i, &j, &k)) return;
    P0Stage<T> p0{phin, phi1, out, I.off, I.ni, (long long)I.ni * I.nj, I.ni, I.nj, I.nk, c1, c2};
    out[I.off + i + p0.sj * j + p0.sk * k] = bc_value<T, false>(bc, p0, I.ni, I.nj, I.nk, i, j, k);
}

// bcond_lsm on the faces of dst from the pre-BC field src (interior nodes
// of dst already hold src)
template <typename T>
__global__ void k_bc_faces(const Inst* __restrict__ inst, int ninst, long long nface, BC bc, const T* __restrict__ src,
                           T* __restrict__ dst, unsigned* err) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= nface) return;
    const Inst& I = inst[face_instance(inst, ninst, t)];
    int i, j, k;
    if (!face_coords(I, (unsigned)(t - I.face0), &i, &j, &k)) return;
    const long long sj = I.ni, sk = (long long)I.ni * I.nj;
    P0Src<T> p0{src, I.off, sj, sk};
    const T v = bc_value<T, false>(bc, p0, I.ni, I.nj, I.nk, i, j, k);
    dst[I.off + i + sj * j + sk * k] = v;
    if (err && !vfinite(v)) atomicOr(err, (unsigned)kErrNonFinite);
}

template <typename T, int TX, int TY, int TZ>
__global__ void __launch_bounds__(TX * TY * TZ) k_bc_full(const Inst* __restrict__ inst,
        const Brick* __restrict__ bricks, int nbricks, BC bc, const T* __restrict__ src, T* __restrict__ dst,
        unsigned* err) {
    for (int blk = blockIdx.x; blk < nbricks; blk += gridDim.x) {
        const Node b = brick_node<TX, TY, TZ>(inst, bricks, blk);
        if (!b.valid) continue;
        const Inst& I = inst[b.inst];
        const long long sj = I.ni, sk = (long long)I.ni * I.nj;
        const long long l = I.off + b.i + sj * b.j + sk * b.k;
        const bool bnd = b.i == 0 || b.i == I.ni - 1 || b.j == 0 || b.j == I.nj - 1 || b.k == 0 || b.k == I.nk - 1;
        T v;
        if (bnd) {
            P0Src<T> p0{src, I.off, sj, sk};
            v = bc_value<T, false>(bc, p0, I.ni, I.nj, I.nk, b.i, b.j, b.k);
        } else {
            v = src[l];
        }
        dst[l] = v;
        if (err && !vfinite(v)) atomicOr(err, (unsigned)kErrNonFinite);
    }
}

// ------------------------------------------------------------ Godunov |grad|
// max(a, b) for b >= 0, a NaN a dropped; FP64 on the bit patterns (ordered as
// signed integers against a b >= 0: a comparison takes the FP64 pipe as long as
// an addition)
template <typename T> __device__ __forceinline__ T pmax(T a, T b) {
    const i64 u = (i64)d2u(a);
    return u > (i64)d2u(b) && u <= (i64)0x7FF0000000000000ll ? a : b;
}
template <> __device__ __forceinline__ float pmax<float>(float a, float b) { return fmaxf(a, b); }

// acc + v^2, the square rounded by itself in FP32
template <typename T> __device__ __forceinline__ T add_square(T acc, T v) { return fma(v, v, acc); }
template <> __device__ __forceinline__ float add_square<float>(float acc, float v) {
    return __fadd_rn(acc, __fmul_rn(v, v));
}

// One-sided differences (calc_RH_RN.F90:36-170) along one axis times the
// branch sign sg (+-1: the product with it is exact): mas (forward) and men
// (backward); on a physical face both take the one available difference.
template <typename T>
__device__ __forceinline__ void one_sided(const T* __restrict__ d, long long l, long long s, int c, int n, T sg, T sx,
                                          T* mas, T* men) {
    // both loads unconditional (the node itself past a face): none waits for a branch
    const T a = vfma(sg, __ldg(d + (c < n - 1 ? l + s : l)), -sx), b = vfma(-sg, __ldg(d + (c > 0 ? l - s : l)), sx);
    *mas = c < n - 1 ? a : b;
    *men = c > 0 ? b : a;
}

// Godunov norm squared (calc_RH_RN.F90:190-236) from those differences.
// With P the positive part of the backward and -Q that of the negated forward
// product, max(P^2, Q^2) is the square of the larger.  SEL: the selections
// too, per axis the P taken (e) or the Q taken (g).
template <bool SEL, typename T>
__device__ __forceinline__ T godunov_sel_v(const T (&mas)[3], const T (&men)[3], const T (&M)[9], T (&e)[3],
                                           T (&g)[3]) {
    T acc = T(0);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const T bb = vfma(M[6 + x], men[2], vfma(M[x], men[0], M[3 + x] * men[1]));
        const T ff = vfma(M[6 + x], mas[2], vfma(M[x], mas[0], M[3 + x] * mas[1]));
        // max(P^2, Q^2) is the square of the larger of P and -Q
        const T p = pmax(bb, T(0)), v = pmax(-ff, p);
        acc = add_square(acc, v);
        if (SEL) {
            const bool takeP = p * p >= v * v;
            e[x] = takeP ? p : T(0);
            g[x] = takeP ? T(0) : -v;
        }
    }
    return acc;
}

// Godunov norm chosen by the sign s
template <typename T>
__device__ __forceinline__ T godunov(const FieldsT<T>& f, const T* __restrict__ d, const Inst& I, long long l, int i,
                                     int j, int k, T x, T s) {
    T mas[3], men[3], M[9], e[3], g[3];
#pragma unroll
    for (int c = 0; c < 9; ++c) M[c] = __ldg(f.m[c] + l);
    const T sg = s > T(0) ? T(1) : T(-1), sx = sg * x;
    one_sided(d, l, 1, i, I.ni, sg, sx, &mas[0], &men[0]);
    one_sided(d, l, (long long)I.ni, j, I.nj, sg, sx, &mas[1], &men[1]);
    one_sided(d, l, (long long)I.ni * I.nj, k, I.nk, sg, sx, &mas[2], &men[2]);
    return vsqrt(godunov_sel_v<false>(mas, men, M, e, g));
}

// the pseudo-step's value from the norm G (every kernel's, bit for bit)
template <typename T>
__device__ __forceinline__ T reinit_value(T d, T s, T dtau, T G) {
    return s == T(0) ? d : vfma(-(dtau * s), G - T(1), d);
}

// calc_sign_ini (Kang sign) with the frozen band folded in: s = 0 where
// |phi0| < eps and |grad phi0| > 0 (the lambda correction pins d to phi0);
// g is the Godunov norm of phi0 chosen by sign(phi0).
template <typename T>
__device__ __forceinline__ T sign_of(T p, T g, T eps) {
    if (p >= eps) return T(1);
    if (p <= -eps) return T(-1);
    if (p != T(0) && g > T(0)) return T(0);
    return p / eps - T(1.0 / kPi) * vsin(T(kPi) * p / eps);
}

// one reinitialisation pseudo-step at a node: d - dtau s (|grad d|_G - 1)
template <typename T>
__device__ __forceinline__ T reinit_node(const FieldsT<T>& f, const T* __restrict__ din, const Inst& I, long long l,
                                         int i, int j, int k) {
    // every load is issued before the frozen-node test (one memory round trip)
    const T s = __ldg(f.sgn + l);
    const T d = __ldg(din + l);
    const T g = godunov(f, din, I, l, i, j, k, d, s);
    return reinit_value(d, s, ipar<T>(I.dtau, I.dtau64), g);
}

template <typename T, int TX, int TY, int TZ>
__global__ void __launch_bounds__(TX * TY * TZ) k_reinit(const Inst* __restrict__ inst,
        const Brick* __restrict__ bricks, int nbricks, FieldsT<T> f, const T* __restrict__ din,
        T* __restrict__ dout, unsigned* err) {
    for (int blk = blockIdx.x; blk < nbricks; blk += gridDim.x) {
        const Node b = brick_node<TX, TY, TZ>(inst, bricks, blk);
        if (!b.valid) continue;
        const Inst& I = inst[b.inst];
        const long long l = I.off + b.i + (long long)I.ni * (b.j + (long long)I.nj * b.k);
        const T r = reinit_node(f, din, I, l, b.i, b.j, b.k);
        dout[l] = r;
        if (err && !vfinite(r)) atomicOr(err, (unsigned)kErrNonFinite);
    }
}

// calc_sign_ini fused with the first pseudo-step: both use the Godunov norm
// of the advected field phi0 chosen by sign(phi0) (a node whose s is not 0
// has the sign of phi0: p / eps - sin(pi p / eps) / pi has the sign of p),
// so one evaluation and one read of phi0 and the metrics give s and
// d1 = phi0 - dtau s (|grad phi0|_G - 1).
template <typename T, int TX, int TY, int TZ>
__global__ void __launch_bounds__(TX * TY * TZ) k_sign_reinit(const Inst* __restrict__ inst,
        const Brick* __restrict__ bricks, int nbricks, FieldsT<T> f, const T* __restrict__ phi0,
        T* __restrict__ dout, unsigned* err) {
    for (int blk = blockIdx.x; blk < nbricks; blk += gridDim.x) {
        const Node b = brick_node<TX, TY, TZ>(inst, bricks, blk);
        if (!b.valid) continue;
        const Inst& I = inst[b.inst];
        const long long l = I.off + b.i + (long long)I.ni * (b.j + (long long)I.nj * b.k);
        const T p = __ldg(phi0 + l);
        const T g = godunov(f, phi0, I, l, b.i, b.j, b.k, p, p);
        const T s = sign_of(p, g, ipar<T>(I.eps, I.eps64));
        f.sgn[l] = s;
        const T r = reinit_value(p, s, ipar<T>(I.dtau, I.dtau64), g);
        dout[l] = r;
        if (err && !vfinite(r)) atomicOr(err, (unsigned)kErrNonFinite);
    }
}

// Recorded pseudo-steps also write the adjoint's coefficients, so that the
// reverse sweep is a 7-point stencil on lam.  With the Godunov selections
// of the step (branch sign sel: P = sel max(sel bb, 0), Q = sel min(sel ff,
// 0), the larger square taken), G^2 = acc, and w = dtau |s| / G:
//   A'_m = w sum_x M[m][x] (P taken ? sel P : 0),  B'_m = the same with Q,
// moved to B' on a low face and to A' on a high face (their one difference
// serves both sides), and the pseudo-step's adjoint is
//   lam_out(j) = lam(j) - sum_m [lam(j) (A'_m - B'_m)(j)
//                - lam(j+e_m) A'_m(j+e_m) + lam(j-e_m) B'_m(j-e_m)].
// One reinitialisation pseudo-step on the tiles of adjoint map 1 (32 x 8
// columns marching 32 planes in k): each node loads d (and s) and its
// metrics once, a plane ahead; the z neighbours of d stay in a register
// window, the x neighbours come by warp shuffles (the tile's edge lanes load
// the one outside) and the y neighbours are loaded (L1/L2).
//   SIGN: the first pseudo-step fused with calc_sign_ini: din is phi0, the
//         Godunov branch is chosen by sign(phi0) (a node whose s is not 0
//         has the sign of phi0), s is computed and stored;
//   REC:  the pseudo-step's adjoint coefficients are stored as well.
// dout2 (nullable) receives a second copy of d'.  d' equals reinit_node's
// arithmetic (one_sided, godunov) bit for bit.
template <typename T, bool SIGN, bool REC>
__global__ void __launch_bounds__(256) k_reinit_z(const Inst* __restrict__ inst, Tiles tl, FieldsT<T> f, const T* __restrict__ din, T* __restrict__ dout, T* __restrict__ dout2,
        T* __restrict__ cf, long long ld, unsigned* err) {
    const unsigned FM = 0xffffffffu;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int blk = blockIdx.x; blk < tl.n; blk += gridDim.x) {
        const ABrick ab = adj_brick(tl, blk);
        const Inst& I = inst[ab.inst];
        const int ni = I.ni, nj = I.nj, nk = I.nk;
        const long long sj = ni, sk = (long long)ni * nj;
        const int i = ab.i0 + tx, j = ab.j0 + ty;
        const int k0 = ab.k0, k1 = min(k0 + tl.len, nk);
        const bool col = i < ni && j < nj;
        const long long cb = I.off + i + sj * j;
        const bool xm = i > 0, xp = i < ni - 1, ym = j > 0, yp = j < nj - 1;
        const bool ex = col && ((tx == 0 && xm) || (tx == 31 && xp));
        const int eo = tx == 0 ? -1 : 1;
        const T dtau = ipar<T>(I.dtau, I.dtau64), eps = ipar<T>(I.eps, I.eps64);
        struct Plane {
            T s, M[9], dxe, dym, dyp;
        };
        auto ld_plane = [&](int k, Plane& p) {
            p.s = p.dxe = p.dym = p.dyp = T(0);
#pragma unroll
            for (int c = 0; c < 9; ++c) p.M[c] = T(0);
            if (!col || k < 0 || k >= nk) return;
            const long long l = cb + sk * k;
            if (!SIGN) p.s = __ldg(f.sgn + l);
#pragma unroll
            for (int c = 0; c < 9; ++c) p.M[c] = __ldg(f.m[c] + l);
            if (ex) p.dxe = __ldg(din + l + eo);
            if (ym) p.dym = __ldg(din + l - sj);
            if (yp) p.dyp = __ldg(din + l + sj);
        };
        auto ldd = [&](int k) { return col && k >= 0 && k < nk ? __ldg(din + cb + sk * k) : T(0); };
        T dm = ldd(k0 - 1), dc = ldd(k0), dp = ldd(k0 + 1);
        Plane pc, pn;
        ld_plane(k0, pc);
        for (int k = k0; k < k1; ++k) {
            const T dn = ldd(k + 2);
            if (k + 1 < k1) ld_plane(k + 1, pn);
            const T xl = __shfl_up_sync(FM, dc, 1), xr = __shfl_down_sync(FM, dc, 1);
            if (col) {
                // one-sided differences (calc_RH_RN.F90:36-170), as one_sided()
                const T dxm = tx == 0 ? pc.dxe : xl, dxp = tx == 31 ? pc.dxe : xr;
                const T nbm[3] = {dxm, pc.dym, dm}, nbp[3] = {dxp, pc.dyp, dp};
                const bool lo[3] = {!xm, !ym, k == 0}, hi[3] = {!xp, !yp, k == nk - 1};
                const T sg = (SIGN ? dc : pc.s) > T(0) ? T(1) : T(-1), sc = sg * dc;
                T mas[3], men[3];
#pragma unroll
                for (int m = 0; m < 3; ++m) {
                    const T a = vfma(sg, nbp[m], -sc), b = vfma(-sg, nbm[m], sc);
                    mas[m] = hi[m] ? b : a;
                    men[m] = lo[m] ? a : b;
                }
                T e[3], g[3];
                const long long l = cb + sk * k;
                const T acc = godunov_sel_v<REC>(mas, men, pc.M, e, g);
                T s = pc.s;
                if (SIGN) {
                    s = sign_of(dc, vsqrt(acc), eps);
                    f.sgn[l] = s;
                }
                const T r = reinit_value(dc, s, dtau, vsqrt(acc));
                dout[l] = r;
                if (dout2) dout2[l] = r;
                if (REC) {
                    const T w = s != T(0) && acc > T(0) ? dtau * fabs(s) * vrsqrt(acc) : T(0);
#pragma unroll
                    for (int m = 0; m < 3; ++m) {
                        const T gmen = pc.M[3 * m] * e[0] + pc.M[3 * m + 1] * e[1] + pc.M[3 * m + 2] * e[2];
                        const T gmas = pc.M[3 * m] * g[0] + pc.M[3 * m + 1] * g[1] + pc.M[3 * m + 2] * g[2];
                        cf[m * ld + l] = lo[m] ? T(0) : w * (hi[m] ? gmen + gmas : gmen);
                        cf[(3 + m) * ld + l] = hi[m] ? T(0) : w * (lo[m] ? gmen + gmas : gmas);
                    }
                }
                if (err && !vfinite(r)) atomicOr(err, (unsigned)kErrNonFinite);
            }
            dm = dc;
            dc = dp;
            dp = dn;
            pc = pn;
        }
    }
}

// Two pseudo-steps of the FP32 batch in one pass over the metrics.  A
// pseudo-step is bound by its bytes, twelve words per node, and by the issue
// of its instructions; nine of the words are the metrics, which two steps
// share, and the field between the steps stays on the chip.  Measured on 64
// grids of 32..96: 2 x 170 us -> 246 us (512 threads; 268 with 384).  (With the adjoint coefficients, whose
// twelve words per node and pair are written all the same, the pair was
// slower than two recorded steps: 884 against 790 us on 512 x 256 x 256.)
//
// A tile is rw x rh columns of one instance plus, where it does not span the
// instance, a rim of one column, in row-major order over the threads (Inst's
// rw, rh: whole rows where the instance is narrow, so that few lanes idle).
// The block marches in k.  Iteration k evaluates the first step on plane k at
// every thread, from d in a register window in z and in shared memory in x
// and y (the values just outside the rim come there by one more load of some
// threads), and the second step on plane k - 1 inside the rim, from the first
// step's planes k - 2 .. k.  One barrier per plane: the shared planes rotate
// over three buffers, in step with the three planes' registers, and each is
// written again only after a barrier that follows its last read.  A node's
// loads go out one plane ahead, on byte offsets of type O as in k_stage.  The
// arithmetic is k_reinit_z's.
struct PairPlane {
    float s, M[9], o;   // sign, metrics, the thread's value outside the rim
};
constexpr int kPairSmem = 3 * (kPairThreads + 2);   // (ew + 2) (eh + 2) for ew eh <= kPairThreads
template <typename O>
__global__ void __launch_bounds__(kPairThreads, 2) k_reinit_pair(const Inst* __restrict__ inst, Tiles tl,
        FieldsT<float> f, const float* __restrict__ din, float* __restrict__ dout, float* __restrict__ dout2,
        unsigned* err) {
    __shared__ float sd[3][kPairSmem], se[3][kPairSmem];
    const int t = threadIdx.x;
    for (int blk = blockIdx.x; blk < tl.n; blk += gridDim.x) {
        const ABrick ab = adj_brick(tl, blk);
        const Inst& I = inst[ab.inst];
        const int ni = I.ni, nj = I.nj, nk = I.nk;
        const int ox = I.rw < ni ? 1 : 0, oy = I.rh < nj ? 1 : 0;
        const int ew = I.rw + 2 * ox, eh = I.rh + 2 * oy, pitch = ew + 2;
        const int y = t / ew, x = t - y * ew;
        const int i = ab.i0 + x - ox, j = ab.j0 + y - oy;
        const bool col = y < eh && i >= 0 && i < ni && j >= 0 && j < nj;
        const bool core = col && x >= ox && x < I.rw + ox && y >= oy && y < I.rh + oy;
        const int k0 = ab.k0, k1 = min(k0 + tl.len, nk);
        const O sk = O(4) * (O)ni * (O)nj;
        const O base = O(4) * (O)I.off;
        const O cb = base + O(4) * (O)i + O(4) * (O)ni * (O)j;
        const bool xm = i == 0, xp = i == ni - 1, ym = j == 0, yp = j == nj - 1;
        // slot in the shared planes, and the value outside the rim that this
        // thread brings there: rows -1 and eh, then columns -1 and ew
        const int me = min(y + 1, eh) * pitch + x + 1;
        int hx = -1, hy = -1;
        if (t < 2 * ew) { hx = t < ew ? t : t - ew; hy = t < ew ? -1 : eh; }
        else if (t < 2 * (ew + eh)) { const int r = t - 2 * ew; hy = r < eh ? r : r - eh; hx = r < eh ? -1 : ew; }
        const int hi_ = ab.i0 + hx - ox, hj = ab.j0 + hy - oy;
        const bool hok = t < 2 * (ew + eh) && hi_ >= 0 && hi_ < ni && hj >= 0 && hj < nj;
        const int hs = (hy + 1) * pitch + hx + 1;
        const O hb = base + O(4) * (O)hi_ + O(4) * (O)ni * (O)hj;
        const float dtau = I.dtau;
        auto ldd = [&](int k) { return col && k >= 0 && k < nk ? ldo(din, cb + sk * (O)k) : 0.f; };
        auto ld_plane = [&](int k, PairPlane& p) {
            if (k >= nk) return;
            if (hok) p.o = ldo(din, hb + sk * (O)k);
            if (!col) return;
            const O l = cb + sk * (O)k;
            p.s = ldo(f.sgn, l);
#pragma unroll
            for (int c = 0; c < 9; ++c) p.M[c] = ldo(f.m[c], l);
        };
        // one pseudo-step at a node of plane k from its neighbours' values
        auto step = [&](float dc, const float* P, float zl, float zr, int k, const PairPlane& p) {
            const float nbm[3] = {P[me - 1], P[me - pitch], zl}, nbp[3] = {P[me + 1], P[me + pitch], zr};
            const bool lo[3] = {xm, ym, k == 0}, hi[3] = {xp, yp, k == nk - 1};
            const float sg = p.s > 0.f ? 1.f : -1.f, sc = sg * dc;
            float mas[3], men[3], e[3], g[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const float a = fmaf(sg, nbp[m], -sc), b = fmaf(-sg, nbm[m], sc);
                mas[m] = hi[m] ? b : a;
                men[m] = lo[m] ? a : b;
            }
            return reinit_value(dc, p.s, dtau, vsqrt(godunov_sel_v<false>(mas, men, p.M, e, g)));
        };
        const int ks = max(k0 - 1, 0);
        float dm = ldd(ks - 1), dc = ldd(ks), dp = ldd(ks + 1);
        float em = 0.f, ec = 0.f;   // the first step's values at planes k - 2, k - 1
        PairPlane p0, p1, p2;
        ld_plane(ks, p1);
        auto plane = [&](int k, PairPlane& pm, PairPlane& pc, PairPlane& pn, float* D, float* E, const float* Em) {
            const float dn = ldd(k + 2);
            if (k < k1) ld_plane(k + 1, pn);
            if (y < eh) D[me] = dc;
            if (hok) D[hs] = pc.o;
            __syncthreads();
            float e1 = 0.f;
            if (col && k < nk) e1 = step(dc, D, dm, dp, k, pc);
            if (core && k > k0) {
                const float r = step(ec, Em, em, e1, k - 1, pm);
                const O l = cb + sk * (O)(k - 1);
                sto(dout, l, r);
                if (dout2) sto(dout2, l, r);
                if (err && !vfinite(r)) atomicOr(err, (unsigned)kErrNonFinite);
            }
            if (y < eh) E[me] = e1;
            em = ec;
            ec = e1;
            dm = dc;
            dc = dp;
            dp = dn;
        };
        // planes ks .. k1 (k1 = nk: the second step alone), three at a time so
        // that registers and buffers keep their places
        for (int k = ks;;) {
            plane(k, p0, p1, p2, sd[1], se[1], se[0]);
            if (++k > k1) break;
            plane(k, p1, p2, p0, sd[2], se[2], se[1]);
            if (++k > k1) break;
            plane(k, p2, p0, p1, sd[0], se[0], se[2]);
            if (++k > k1) break;
        }
        __syncthreads();   // the next tile writes the buffers that this one's last plane reads
    }
}

// Reverse of one recorded pseudo-step from its stored coefficients (cf:
// A'_0..2, B'_0..2, ld apart), on flat tiles marching in k.  Bound
// by its bytes: eight words per node.  A node's own lam and coefficients come
// one plane ahead, what the plane below takes of it (lam, A'_2) two, its share
// of the plane above is carried; the x and y neighbours are plain loads that
// mostly hit L1.  512 x 256 x 256: 213 us (32 x 8 tiles, own values shuffled,
// the plane above awaited) -> 204 us, 128^3 18 -> 15 us; five blocks per SM
// (six: 215 us, eight: 228 us: too many planes at once for L2).
template <typename T, typename O>
__global__ void __launch_bounds__(kStageThreads, sizeof(T) == 4 ? 5 : 3) k_adj_reinit_c(const Inst* __restrict__ inst,
        Tiles tl, const T* __restrict__ cf, long long ld, const T* __restrict__ lam, T* __restrict__ lam_out) {
    struct Pl {
        T A0, A1, B0, B1, B2;
    };
    const int t = threadIdx.x;
    for (int blk = blockIdx.x; blk < tl.n; blk += gridDim.x) {
        const ABrick ab = adj_brick(tl, blk);
        const Inst& I = inst[ab.inst];
        const int ni = I.ni, nj = I.nj, nk = I.nk;
        const int y = t / I.sw, x = t - y * I.sw;
        const int i = ab.i0 + x, j = ab.j0 + y;
        if (y >= I.sh || i >= ni || j >= nj) continue;
        const int k0 = ab.k0, k1 = min(k0 + tl.len, nk);
        const bool xm = i > 0, xp = i < ni - 1, ym = j > 0, yp = j < nj - 1;
        constexpr O E = sizeof(T);
        const O sj = E * (O)ni, sk = sj * (O)nj;
        O l = E * (O)I.off + E * (O)i + sj * (O)j + sk * (O)k0;   // plane k
        auto ld_own = [&](O l, Pl& p) {
            p.A0 = ldo(cf, l);
            p.A1 = ldo(cf + ld, l);
            p.B0 = ldo(cf + 3 * ld, l);
            p.B1 = ldo(cf + 4 * ld, l);
            p.B2 = ldo(cf + 5 * ld, l);
        };
        Pl a, b;
        ld_own(l, a);
        T L = ldo(lam, l), A2 = ldo(cf + 2 * ld, l), Ln = T(0), An = T(0);
        if (k0 + 1 < nk) {
            Ln = ldo(lam, l + sk);
            An = ldo(cf + 2 * ld, l + sk);
        }
        T zb = k0 > 0 ? ldo(lam, l - sk) * ldo(cf + 5 * ld, l - sk) : T(0);   // lam B'_2 of the plane below
        auto plane = [&](int k, const Pl& c, Pl& n) {
            T Lnn = T(0), Ann = T(0);
            if (k + 1 < k1) {
                ld_own(l + sk, n);
                if (k + 2 < nk) {
                    Lnn = ldo(lam, l + 2 * sk);
                    Ann = ldo(cf + 2 * ld, l + 2 * sk);
                }
            }
            T t0 = L * (c.A0 - c.B0), t1 = L * (c.A1 - c.B1);
            if (xp) t0 -= ldo(lam, l + E) * ldo(cf, l + E);
            if (xm) t0 += ldo(lam, l - E) * ldo(cf + 3 * ld, l - E);
            if (yp) t1 -= ldo(lam, l + sj) * ldo(cf + ld, l + sj);
            if (ym) t1 += ldo(lam, l - sj) * ldo(cf + 4 * ld, l - sj);
            const T t2 = L * (A2 - c.B2) - Ln * An + zb;
            sto(lam_out, l, L - t0 - t1 - t2);
            zb = L * c.B2;
            L = Ln;
            A2 = An;
            Ln = Lnn;
            An = Ann;
            l += sk;
        };
        for (int k = k0;;) {
            plane(k, a, b);
            if (++k >= k1) break;
            plane(k, b, a);
            if (++k >= k1) break;
        }
    }
}

// P0 after the last pseudo-step: interior from its output, boundary nodes
// recomputed from its input (their output slots are being overwritten).
template <typename T>
struct P0Reinit {
    FieldsT<T> f;
    const T *din, *dout;
    const Inst* I;
    __device__ T operator()(int i, int j, int k) const {
        const long long l = I->off + i + (long long)I->ni * (j + (long long)I->nj * k);
        const bool bnd = i == 0 || i == I->ni - 1 || j == 0 || j == I->nj - 1 || k == 0 || k == I->nk - 1;
        return bnd ? reinit_node(f, din, *I, l, i, j, k) : dout[l];
    }
};

template <typename T>
__global__ void k_bc_reinit(const Inst* __restrict__ inst, int ninst, long long nface, BC bc, FieldsT<T> f,
                            const T* __restrict__ din, T* dout) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= nface) return;
    const Inst& I = inst[face_instance(inst, ninst, t)];
    int i, j, k;
    if (!face_coords(I, (unsigned)(t - I.face0), &i, &j, &k)) return;
    P0Reinit<T> p0{f, din, dout, &I};
    dout[I.off + i + (long long)I.ni * (j + (long long)I.nj * k)] = bc_value<T, true>(bc, p0, I.ni, I.nj, I.nk, i, j, k);
}

// ------------------------------------------------------------ volume
// Water volume of one tetrahedron of an interface cell: the same regions as
// MarchingTetrahedron + GetWaterVolume (src/TetrahedronMethods.F90:26-954),
// each sub-tetrahedron's share of the tetrahedron evaluated in barycentric
// closed form: one determinant per tetrahedron instead of up to four
// (equal in exact arithmetic, rounding differs).  G is the geometry type:
// FP64 for the FP64 stencils, FP32 for the FP32 ones (vertices relative to
// the cell's first vertex, see k_vol_iface).
template <typename G>
__device__ __forceinline__ G tetvol_g(const G (&a)[3], const G (&b)[3], const G (&c)[3], const G (&d)[3]) {
    const G u0 = b[0] - a[0], u1 = b[1] - a[1], u2 = b[2] - a[2];
    const G v0 = c[0] - a[0], v1 = c[1] - a[1], v2 = c[2] - a[2];
    const G w0 = d[0] - a[0], w1 = d[1] - a[1], w2 = d[2] - a[2];
    const G t = w0 * (u1 * v2 - u2 * v1) + w1 * (u2 * v0 - u0 * v2) + w2 * (u0 * v1 - u1 * v0);
    return fabs(t) * G(1.0 / 6.0);
}

// 4-way selection without indexing (keeps the tetrahedron in registers)
template <typename X>
__device__ __forceinline__ X sel4(const X (&a)[4], int i) {
    return i == 0 ? a[0] : (i == 1 ? a[1] : (i == 2 ? a[2] : a[3]));
}

// ------------------------------------------------------------ dual numbers
// Forward-mode derivatives of the tetrahedron water volume with respect to
// its vertex values (the mass correction and its adjoint): a value and K
// partials; S is a scalar or itself a Dual (second derivatives).
template <typename S, int K>
struct Dual {
    S v;
    S d[K];
};
template <typename X> struct DualTraits { using Base = X; };
template <typename S, int K> struct DualTraits<Dual<S, K>> { using Base = typename DualTraits<S>::Base; };
template <typename X> __device__ __forceinline__ typename DualTraits<X>::Base dval(const X& x) { return x; }
template <typename S, int K> __device__ __forceinline__ typename DualTraits<S>::Base dval(const Dual<S, K>& x) {
    return dval(x.v);
}
// constant (all partials zero)
template <typename X> struct Lift { __device__ static X of(typename DualTraits<X>::Base c) { return X(c); } };
template <typename S, int K> struct Lift<Dual<S, K>> {
    __device__ static Dual<S, K> of(typename DualTraits<S>::Base c) {
        Dual<S, K> r;
        r.v = Lift<S>::of(c);
#pragma unroll
        for (int k = 0; k < K; ++k) r.d[k] = Lift<S>::of(typename DualTraits<S>::Base(0));
        return r;
    }
};
template <typename S, int K>
__device__ __forceinline__ Dual<S, K> operator+(const Dual<S, K>& a, const Dual<S, K>& b) {
    Dual<S, K> r;
    r.v = a.v + b.v;
#pragma unroll
    for (int k = 0; k < K; ++k) r.d[k] = a.d[k] + b.d[k];
    return r;
}
template <typename S, int K>
__device__ __forceinline__ Dual<S, K> operator-(const Dual<S, K>& a, const Dual<S, K>& b) {
    Dual<S, K> r;
    r.v = a.v - b.v;
#pragma unroll
    for (int k = 0; k < K; ++k) r.d[k] = a.d[k] - b.d[k];
    return r;
}
template <typename S, int K>
__device__ __forceinline__ Dual<S, K> operator-(const Dual<S, K>& a) {
    Dual<S, K> r;
    r.v = -a.v;
#pragma unroll
    for (int k = 0; k < K; ++k) r.d[k] = -a.d[k];
    return r;
}
template <typename S, int K>
__device__ __forceinline__ Dual<S, K> operator*(const Dual<S, K>& a, const Dual<S, K>& b) {
    Dual<S, K> r;
    r.v = a.v * b.v;
#pragma unroll
    for (int k = 0; k < K; ++k) r.d[k] = a.d[k] * b.v + a.v * b.d[k];
    return r;
}
template <typename S, int K>
__device__ __forceinline__ Dual<S, K> operator/(const Dual<S, K>& a, const Dual<S, K>& b) {
    Dual<S, K> r;
    r.v = a.v / b.v;
#pragma unroll
    for (int k = 0; k < K; ++k) r.d[k] = (a.d[k] - r.v * b.d[k]) / b.v;
    return r;
}
// scalar (geometry) factor times a dual
template <typename S, int K>
__device__ __forceinline__ Dual<S, K> operator*(typename DualTraits<S>::Base c, const Dual<S, K>& a) {
    Dual<S, K> r;
    r.v = c * a.v;
#pragma unroll
    for (int k = 0; k < K; ++k) r.d[k] = c * a.d[k];
    return r;
}
template <typename S, int K>
__device__ __forceinline__ Dual<S, K> operator-(typename DualTraits<S>::Base c, const Dual<S, K>& a) {
    return Lift<Dual<S, K>>::of(c) - a;
}

// Water (phi > 0) volume of one tetrahedron with vertices V and vertex
// values ph (the reference's MarchingTetrahedron + GetWaterVolume cases,
// src/TetrahedronMethods.F90:586-954, in closed form).  X is the vertex
// value type: the geometry type G, or a Dual of it for the derivatives with
// respect to the vertex values (the case chosen by the values themselves).
template <typename G, typename X>
__device__ __forceinline__ X tet_water_x(const G (&V)[4][3], const X (&ph)[4]) {
    const G TV = tetvol_g(V[0], V[1], V[2], V[3]);
    const G tiny = G(sizeof(G) == 8 ? kTinyD : 0.0);   // tiny(1d0); in FP32 every nonzero value exceeds it
    const X zero = Lift<X>::of(G(0)), one = Lift<X>::of(G(1)), full = Lift<X>::of(TV);
    int s[4], nz = 0, fi = 0;
    bool allp = true, alln = true, allge = true, allle = true;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const G pv = dval(ph[v]);
        s[v] = pv > tiny ? 1 : (pv < -tiny ? -1 : 0);
        allp &= s[v] == 1; alln &= s[v] == -1; nz += s[v] == 0;
        allge &= s[v] >= 0; allle &= s[v] <= 0;
        if (s[v] == -1) fi |= 1 << v;
    }
    if (allp) return full;
    if (alln) return zero;
    if (nz > 0 && (allge || allle)) {
        // the reference's zero-vertex cases: full or empty tetrahedron
        int water = -1;
        if (nz == 1) {
            if (s[0] == 0) water = s[1] == 1; else if (s[1] == 0) water = s[0] == 1;
            else if (s[2] == 0) water = s[0] == 1; else water = s[0] == 1;
        } else if (nz == 2) {
            if (s[0] == 0 && s[1] == 0) water = s[2] == 1;
            else if (s[1] == 0 && s[2] == 0) water = s[0] == 1;
            else if (s[2] == 0 && s[0] == 0) water = s[1] == 1;
            else if (s[0] == 0 && s[3] == 0) water = s[1] == 1;
            else if (s[1] == 0 && s[3] == 0) water = s[0] == 1;
            else water = s[0] == 1;
        } else if (nz == 3) {
#pragma unroll
            for (int v = 0; v < 4; ++v)
                if (water < 0 && s[v] != 0) water = s[v] == 1;   // the non-zero vertex
        }
        return water == 0 ? zero : full;   // four zero vertices: full (FlagIndex 0)
    }
    // one vertex isolated from the other three (cases 2/15, 3/14, 5/12, 9/8)
    int iso = -1;
    if (fi == 1 || fi == 14) iso = 0; else if (fi == 2 || fi == 13) iso = 1;
    else if (fi == 4 || fi == 11) iso = 2; else if (fi == 8 || fi == 7) iso = 3;
    if (iso >= 0) {
        // prod_k p_iso / (p_iso - p_k) over one division (the differences
        // all carry the sign of p_iso: no cancellation); the factor of k =
        // iso is an exact 1
        const X pI = sel4(ph, iso);
        X num = one, den = one;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            num = num * (k != iso ? pI : one);
            den = den * (k != iso ? pI - ph[k] : one);
        }
        const X AV = TV * (num / den);
        return (sel4(s, iso) == -1) ? TV - AV : AV;   // isolated vertex negative: the rest is water
    }
    // two against two (cases 4/13, 6/11, 7/10): pair (A, B) as listed by the
    // reference's sub-tetrahedra, C, D the other pair:
    //   fi 3/12: A 0, B 1, C 2;  fi 5/10: A 0, B 2, C 1;  else A 1, B 2, C 0;  D 3
    const int cs = (fi == 3 || fi == 12) ? 0 : ((fi == 5 || fi == 10) ? 1 : 2);
    // with the edge fractions aX = pA / (pA - pX), bX = pB / (pB - pX) the
    // share is aC aD (1 - bD) + aC bD (1 - bC) + bC bD; over the common
    // denominator (pA - pC)(pA - pD)(pB - pC)(pB - pD), using 1 - bX =
    // -pX / (pB - pX), it needs one division, and its three numerator terms
    // share one sign (A, B on one side of the interface, C, D on the other)
    const X pA = cs == 2 ? ph[1] : ph[0];
    const X pB = cs == 0 ? ph[1] : ph[2];
    const X pC = cs == 0 ? ph[2] : (cs == 1 ? ph[1] : ph[0]);
    const X pD = ph[3];
    const X dAC = pA - pC, dAD = pA - pD, dBC = pB - pC, dBD = pB - pD;
    const X num = pB * pB * dAC * dAD - pA * pA * pD * dBC - pA * pB * pC * dAD;
    const X AV = TV * (num / (dAC * dAD * dBC * dBD));
    return ((cs == 2 ? s[1] : s[0]) == -1) ? TV - AV : AV;
}

template <typename G>
__device__ __forceinline__ G tet_water(const G (&V)[4][3], const G (&ph)[4]) {
    return tet_water_x<G, G>(V, ph);
}

// vertex v of tetrahedron t of CellAnalysis's split (the c_tets table
// {0,5,1,6}, {0,1,2,6}, {0,2,3,6}, {0,3,7,6}, {0,7,4,6}, {0,4,5,6}) as a
// constant expression, so that unrolled loops index registers
__host__ __device__ constexpr int cell_tet(int t, int v) {
    return v == 0 ? 0
                  : v == 3 ? 6
                           : v == 1 ? (t == 0 ? 5 : t == 1 ? 1 : t == 2 ? 2 : t == 3 ? 3 : t == 4 ? 7 : 4)
                                    : (t == 0 ? 1 : t == 1 ? 2 : t == 2 ? 3 : t == 3 ? 7 : t == 4 ? 4 : 5);
}

// CellAnalysis's tetrahedron classes: pct (phase change, a K tetrahedron)
// or second (all water); the phi-type compares equal the FP64 ones.
template <typename P>
__device__ __forceinline__ void tet_class(const P (&ph8)[8], int t, bool* pct_out, bool* second_out) {
    const P es = P(kEpsSims);
    bool pct = false, second = true;
    const P pa = ph8[cell_tet(t, 0)];
    if (pa <= es) second = false;
    if (fabs(pa) < es) pct = true;
    const P sg = signbit(pa) ? P(-1) : P(1);
#pragma unroll
    for (int v = 1; v < 4; ++v) {
        const P pb = ph8[cell_tet(t, v)];
        if (sg * pb < P(0) || fabs(pb) < es) {
            if (pb <= es) second = false;
            pct = true;
        }
    }
    *pct_out = pct;
    *second_out = second;
}

// whether CellAnalysis splits the cell (a vertex within eps_sims of zero or
// a sign change)
template <typename P>
__device__ __forceinline__ bool cell_is_interface(const P (&ph8)[8]) {
    const P es = P(kEpsSims);
    bool pcc = false;
#pragma unroll
    for (int v = 0; v < 8; ++v) pcc |= fabs(ph8[v]) < es;
    if (!pcc) {
        const P sg = signbit(ph8[0]) ? P(-1) : P(1);   // copysign(1, phi)
#pragma unroll
        for (int v = 1; v < 8; ++v) pcc |= sg * ph8[v] < P(0);
    }
    return pcc;
}

// CellAnalysis's split of an interface cell (src/TetrahedronMethods.F90:
// 1823-2121): phase-change tetrahedra -> K, all-water tetrahedra -> S.
// The classification runs in the phi type P (eps_sims = 2^-52 and +-1 are
// exact in FP32, so its compares equal the FP64 ones on the same values),
// the geometry in P as well, on vertex coordinates relative to the cell's
// first vertex (C, formed in FP64 by the caller).  Fully unrolled: every
// array index is a constant (no local memory).  With SLOPE, *A also gets
// dK/dC, the derivative of the K volume under a uniform shift phi + C
// (forward-mode dual numbers through the same case formulas).
template <typename P, bool SLOPE = false>
__device__ void cell_water_fast(const P (&ph8)[8], const P (&C)[8][3], double* K, double* S, double* A = nullptr) {
    P k = P(0), s2 = P(0), a = P(0);
    if (cell_is_interface(ph8)) {
#pragma unroll
        for (int t = 0; t < 6; ++t) {
            bool pct, second;
            tet_class(ph8, t, &pct, &second);
            if (pct || second) {
                P V[4][3], ph[4];
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    V[v][0] = C[cell_tet(t, v)][0];
                    V[v][1] = C[cell_tet(t, v)][1];
                    V[v][2] = C[cell_tet(t, v)][2];
                    ph[v] = ph8[cell_tet(t, v)];
                }
                if (pct) {
                    if constexpr (SLOPE) {
                        Dual<P, 1> pd[4];
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            pd[v].v = ph[v];
                            pd[v].d[0] = P(1);
                        }
                        const Dual<P, 1> w = tet_water_x<P, Dual<P, 1>>(V, pd);
                        k += w.v;
                        a += w.d[0];
                    } else {
                        k += tet_water(V, ph);
                    }
                } else {
                    s2 += tetvol_g(V[0], V[1], V[2], V[3]);
                }
            }
        }
    }
    *K = (double)k; *S = (double)s2;
    if (A) *A = (double)a;
}

// Mass-correction adjoint weights of one interface cell: for each vertex v
// the derivative of the cell's K volume g_v = dK/dphi_v plus Cs h_v with
// h_v = d(dK/dC)/dphi_v (second-order dual numbers), so that the shift
// C = (target - V) / A has dC/dphi_v = -(g_v + C h_v) / A summed over the
// cells around the node.
template <typename P>
__device__ void cell_mass_weights(const P (&ph8)[8], const P (&C)[8][3], P Cs, P (&w8)[8]) {
#pragma unroll
    for (int v = 0; v < 8; ++v) w8[v] = P(0);
    if (!cell_is_interface(ph8)) return;
    using D1 = Dual<P, 1>;
    using D2 = Dual<D1, 4>;
#pragma unroll
    for (int t = 0; t < 6; ++t) {
        bool pct, second;
        tet_class(ph8, t, &pct, &second);
        if (!pct) continue;
        P V[4][3];
        D2 pd[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            V[v][0] = C[cell_tet(t, v)][0];
            V[v][1] = C[cell_tet(t, v)][1];
            V[v][2] = C[cell_tet(t, v)][2];
            pd[v].v.v = ph8[cell_tet(t, v)];
            pd[v].v.d[0] = P(1);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                pd[v].d[u].v = u == v ? P(1) : P(0);
                pd[v].d[u].d[0] = P(0);
            }
        }
        const D2 r = tet_water_x<P, D2>(V, pd);
#pragma unroll
        for (int u = 0; u < 4; ++u) w8[cell_tet(t, u)] += r.d[u].v + Cs * r.d[u].d[0];
    }
}

// The volume pass runs in two kernels.  k_vol_scan_z streams every cell of
// every instance (a k march over the tiles of adjoint map 1): cells whose
// eight vertices are water (phi > eps_sims, in the phi type) add their
// precomputed FP64 hexahedron volume in 64-bit fixed point; interface cells
// (any other mix) are appended to a list, each warp reserving its slots with
// one atomic (list order is not fixed; every sum below is an integer sum, so
// the result does not depend on it).  k_vol_iface then runs the reference's
// six-tetrahedra split on the listed cells with every lane busy, in the
// stencil precision on coordinates relative to each cell's first vertex
// (differences formed in FP64; an FP32 batch keeps them per cell, formed
// once per geometry), optionally with the mass correction's slope
// dK/dC.  Each cell's shares are rounded to multiples of 2^-48 and added to
// the instance's accumulators with integer atomics after a warp sum: exact
// and order-independent.
// exact warp sum of 64-bit integers (two's complement, modulo 2^64): three
// limbs of 22, 22 and 20 bits, each summed by the warp's integer reduction
// (32 x 2^22 < 2^32), recombined; every lane gets the sum
__device__ __forceinline__ long long warp_sum_nn(long long v) {
    const unsigned long long u = (unsigned long long)v;
    const unsigned m = (1u << 22) - 1u;
    const unsigned long long s0 = __reduce_add_sync(0xffffffffu, (unsigned)(u & m));
    const unsigned long long s1 = __reduce_add_sync(0xffffffffu, (unsigned)((u >> 22) & m));
    const unsigned long long s2 = __reduce_add_sync(0xffffffffu, (unsigned)(u >> 44));
    return (long long)(s0 + (s1 << 22) + (s2 << 44));
}

// Bulk water volumes of the cells (added to acc[4 inst + 2]) and the
// interface-cell list, on the tiles of adjoint map 1 (FULL: tiles of the
// longest march, a constant that saves 4 registers and with them a block per
// SM: 111 against 125 us on 512 x 256 x 256 nodes): thread (lane, row) owns the cell column (i0 + lane, j0 +
// row) and marches the tile's planes in k.  A cell's eight vertices are the
// 2 x 2 quads of planes k and k + 1; a quad is the thread's own node and
// the one at j + 1 (loaded), with the i + 1 pair from the next lane by a
// shuffle (the tile's last lane loads it).  Each plane is loaded once, a
// plane ahead of its use; a quad is reduced to two flags (all water, all
// air) and a cell is water / air when both of its quads are.
template <typename T, bool FULL>
__global__ void __launch_bounds__(256) k_vol_scan_z(const Inst* __restrict__ inst, Tiles tl, FieldsT<T> f, const T* __restrict__ phi, unsigned long long* __restrict__ acc,
        unsigned* __restrict__ list, unsigned* __restrict__ count) {
    const T eps = T(kEpsSims);
    const unsigned FM = 0xffffffffu;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    long long Bq = 0;
    int cur = -1;
    auto flush = [&]() {
        const long long v = warp_sum_nn(Bq);
        if (tx == 0 && v != 0) atomicAdd(acc + 4 * (long long)cur + 2, (unsigned long long)v);
        Bq = 0;
    };
    for (int blk = blockIdx.x; blk < tl.n; blk += gridDim.x) {
        const ABrick ab = adj_brick(tl, blk);
        if (ab.inst != cur) {
            if (cur >= 0) flush();
            cur = ab.inst;
        }
        const Inst& I = inst[ab.inst];
        const int ni = I.ni, nj = I.nj, nk = I.nk;
        const long long sj = ni, sk = (long long)ni * nj;
        const int i = ab.i0 + tx, j = ab.j0 + ty;
        // cells k0 .. kc1 - 1 (a cell's top plane k + 1 stays inside the grid)
        const int k0 = ab.k0, kc1 = min(k0 + (FULL ? adj_shape(1).oz : tl.len), nk - 1);
        const bool cell = i < ni - 1 && j < nj - 1;
        const bool own = i < ni && j < nj - 1, edge = tx == 31 && i + 1 < ni && j < nj - 1;
        const long long cb = I.off + i + sj * j;
        struct Quad {
            T a, c, ae, ce;   // (i, j), (i, j + 1); the last lane's (i + 1, j), (i + 1, j + 1)
        };
        auto ld = [&](int k, Quad& q) {
            q.a = q.c = q.ae = q.ce = T(0);
            const long long l = cb + sk * k;
            if (own) {
                q.a = __ldg(phi + l);
                q.c = __ldg(phi + l + sj);
            }
            if (edge) {
                q.ae = __ldg(phi + l + 1);
                q.ce = __ldg(phi + l + 1 + sj);
            }
        };
        auto flags = [&](const Quad& q, bool& qw, bool& qa) {
            const T b = __shfl_down_sync(FM, q.a, 1), d = __shfl_down_sync(FM, q.c, 1);
            const T bb = tx == 31 ? q.ae : b, dd = tx == 31 ? q.ce : d;
            qw = q.a > eps && bb > eps && q.c > eps && dd > eps;
            qa = q.a < -eps && bb < -eps && q.c < -eps && dd < -eps;
        };
        bool qw0 = false, qa0 = false;
        Quad qn;
        long long cv = 0;
        if (k0 < kc1) {
            Quad q0;
            ld(k0, q0);
            ld(k0 + 1, qn);
            if (cell) cv = __ldg(f.cellfix + cb + sk * k0);
            flags(q0, qw0, qa0);
        }
        for (int k = k0; k < kc1; ++k) {
            Quad qq;
            long long cvn = 0;
            if (k + 1 < kc1) {
                ld(k + 2, qq);
                if (cell) cvn = __ldg(f.cellfix + cb + sk * (k + 1));
            }
            bool qw1, qa1;
            flags(qn, qw1, qa1);
            const bool allw = qw0 && qw1, alla = qa0 && qa1;
            if (cell && allw) Bq += cv;
            const bool mix = cell && !allw && !alla;
            const unsigned m = __ballot_sync(FM, mix);
            if (m) {
                unsigned base = 0;
                if (tx == 0) base = atomicAdd(count, (unsigned)__popc(m));
                base = __shfl_sync(FM, base, 0);
                if (mix) list[base + __popc(m & ((1u << tx) - 1u))] = (unsigned)(cb + sk * k);
            }
            qw0 = qw1;
            qa0 = qa1;
            qn = qq;
            cv = cvn;
        }
    }
    if (cur >= 0) flush();
}

// the eight vertex values and the coordinates relative to vertex 0 of the
// listed cell whose first node is l (instance I)
template <typename T>
__device__ __forceinline__ void cell_gather(const Inst& I, const FieldsT<T>& f, const T* __restrict__ phi,
                                            long long l, long long (&o)[8], T (&P8)[8], T (&C)[8][3]) {
    const long long sj = I.ni, sk = (long long)I.ni * I.nj;
    o[0] = l; o[1] = l + 1; o[2] = l + 1 + sj; o[3] = l + sj;
    o[4] = l + sk; o[5] = l + 1 + sk; o[6] = l + 1 + sj + sk; o[7] = l + sj + sk;
#pragma unroll
    for (int v = 0; v < 8; ++v) P8[v] = __ldg(phi + o[v]);
    if constexpr (sizeof(T) == 4) {
        if (f.cellrel) {
            // the same values, formed once per geometry (k_cell_rel)
            const float4* r = reinterpret_cast<const float4*>(f.cellrel + 24 * l);
            float q[24];
#pragma unroll
            for (int u = 0; u < 6; ++u) {
                const float4 w = __ldg(r + u);
                q[4 * u] = w.x; q[4 * u + 1] = w.y; q[4 * u + 2] = w.z; q[4 * u + 3] = w.w;
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) C[0][a] = T(0);
#pragma unroll
            for (int v = 1; v < 8; ++v)
#pragma unroll
                for (int a = 0; a < 3; ++a) C[v][a] = q[3 * (v - 1) + a];
            return;
        }
    }
    double X0[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) X0[a] = __ldg(f.xyz[a] + l);
#pragma unroll
    for (int v = 0; v < 8; ++v)
#pragma unroll
        for (int a = 0; a < 3; ++a) C[v][a] = (T)(__ldg(f.xyz[a] + o[v]) - X0[a]);
}

// instance of packed node t (binary search over the node offsets)
__device__ __forceinline__ int node_instance(const Flat& fl, long long t) {
    int lo = 0, hi = fl.ninst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (fl.offs[mid] <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// K and S volumes (and with SLOPE dK/dC) of the listed interface cells into
// acc[4 inst + 0, 1, 3].  The list holds short runs of an instance's cells, so
// a warp sums per instance: an atomic per lane on a few addresses clogged the
// memory pipe (64 grids of 32..96, 570 000 cells: 157 -> 46 us, with enough
// blocks to even out the warps: 61 us with eight per SM).
template <typename T, bool SLOPE>
__global__ void __launch_bounds__(128) k_vol_iface(Flat fl, FieldsT<T> f, const T* __restrict__ phi,
                                                   const unsigned* __restrict__ list, const unsigned* __restrict__ count,
                                                   unsigned long long* __restrict__ acc) {
    const unsigned FM = 0xffffffffu;
    const unsigned n = *count;
    const int lane = threadIdx.x & 31;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long e0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); e0 < n; e0 += stride) {
        const long long e = e0 + lane;
        const bool valid = e < n;
        long long Kq = 0, Sq = 0, Aq = 0;
        int q = -1;
        if (valid) {
            const long long l = list[e];
            q = node_instance(fl, l);
            long long o[8];
            T P8[8], C[8][3];
            cell_gather(fl.inst[q], f, phi, l, o, P8, C);
            double K = 0.0, S = 0.0, A = 0.0;
            cell_water_fast<T, SLOPE>(P8, C, &K, &S, &A);
            Kq = __double2ll_rn(K * kVolScale);
            Sq = __double2ll_rn(S * kVolScale);
            if (SLOPE) Aq = __double2ll_rn(A * kVolScale);
        }
        // one sum and one atomic per instance that the warp holds
        for (unsigned left = __ballot_sync(FM, valid); left;) {
            const int ql = __shfl_sync(FM, q, __ffs(left) - 1);
            const bool in = q == ql;
            left &= ~__ballot_sync(FM, in);
            const long long v[3] = {warp_sum_nn(in ? Kq : 0), warp_sum_nn(in ? Sq : 0), SLOPE ? warp_sum_nn(in ? Aq : 0) : 0};
            if (lane == 0) {
                if (v[0]) atomicAdd(acc + 4 * (long long)ql, (unsigned long long)v[0]);
                if (v[1]) atomicAdd(acc + 4 * (long long)ql + 1, (unsigned long long)v[1]);
                if (v[2]) atomicAdd(acc + 4 * (long long)ql + 3, (unsigned long long)v[2]);
            }
        }
    }
}

// converts each instance's accumulators (K, S, bulk, slope) to volumes and
// clears them for the next volume pass; with `mass` it also forms the
// mass correction C = (target - V) / A of the total V (C = 0 without a
// finite target or without interface), into mass[q] and, when recording,
// mrec[q]
__global__ void k_volume_final(int ninst, unsigned long long* __restrict__ acc, double* __restrict__ vols,
                               const double* __restrict__ target, Mass* __restrict__ mass, Mass* __restrict__ mrec) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= ninst) return;
    long long v[4];
    for (int c = 0; c < 4; ++c) {
        v[c] = (long long)acc[4 * q + c];
        acc[4 * q + c] = 0ull;
    }
    const double tot = (double)(v[0] + v[1] + v[2]) * kVolUnit;
    vols[4 * q] = (double)v[0] * kVolUnit;
    vols[4 * q + 1] = (double)v[1] * kVolUnit;
    vols[4 * q + 2] = (double)v[2] * kVolUnit;
    vols[4 * q + 3] = tot;
    if (mass) {
        Mass m;
        m.V = tot;
        m.A = (double)v[3] * kVolUnit;
        m.target = target[q];
        const double c = (target[q] - tot) / m.A;
        m.C = mass_on(m) ? c : 0.0;
        mass[q] = m;
        if (mrec) mrec[q] = m;
    }
}

// dst = src + C of the node's instance (the mass correction's uniform shift)
template <typename T>
__global__ void k_mass_shift(Flat fl, const Mass* __restrict__ mass, const T* __restrict__ src, T* __restrict__ dst) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < fl.n;
         t += (long long)gridDim.x * blockDim.x) {
        Node nd;
        flat_node(fl, t, &nd);
        dst[t] = src[t] + (T)mass[nd.inst].C;
    }
}

// Adjoint of the shift, part 1: every listed interface cell of the step's
// pre-correction field adds its vertices' weights g_v + C h_v
// (cell_mass_weights) to wfix in fixed point (integer atomics: exact and
// order-independent).
template <typename T>
__global__ void __launch_bounds__(128) k_mass_weights(Flat fl, FieldsT<T> f, const T* __restrict__ phi,
                                                      const unsigned* __restrict__ list,
                                                      const unsigned* __restrict__ count, const Mass* __restrict__ mass,
                                                      unsigned long long* __restrict__ wfix) {
    const unsigned n = *count;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x) {
        const long long l = list[e];
        const int q = node_instance(fl, l);
        const Mass M = mass[q];
        if (!mass_on(M)) continue;
        long long o[8];
        T P8[8], C[8][3], W8[8];
        cell_gather(fl.inst[q], f, phi, l, o, P8, C);
        cell_mass_weights<T>(P8, C, (T)M.C, W8);
#pragma unroll
        for (int v = 0; v < 8; ++v) {
            const long long w = __double2ll_rn((double)W8[v] * kVolScale);
            if (w != 0) atomicAdd(wfix + o[v], (unsigned long long)w);
        }
    }
}

// Adjoint of the shift, part 2: per tile of adjoint map 1 (32 x 8 columns
// x 32 planes, inside one instance) the sum of lam over the tile, in a
// fixed order (each thread its column, then a fixed tree), accumulated in
// FP64.  FP32 lam is first summed in FP32 over runs of 8 planes (the FP64
// pipe would otherwise take a conversion and an add per node).
template <typename T>
__global__ void __launch_bounds__(256) k_tile_sum(const Inst* __restrict__ inst, Tiles tl, const T* __restrict__ lam, double* __restrict__ part) {
    __shared__ double red[8];
    const int t = threadIdx.x, tx = t & 31, ty = t >> 5;
    for (int blk = blockIdx.x; blk < tl.n; blk += gridDim.x) {
        const ABrick ab = adj_brick(tl, blk);
        const Inst& I = inst[ab.inst];
        const int i = ab.i0 + tx, j = ab.j0 + ty, k1 = min(ab.k0 + tl.len, I.nk);
        double sacc = 0.0;
        if (i < I.ni && j < I.nj) {
            const long long sk = (long long)I.ni * I.nj;
            const T* p = lam + I.off + i + (long long)I.ni * j;
            if constexpr (sizeof(T) == 4) {
                for (int k = ab.k0; k < k1; k += 8) {
                    float r = 0.f;
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (k + u < k1) r += __ldg(p + sk * (k + u));
                    sacc += (double)r;
                }
            } else {
                for (int k = ab.k0; k < k1; ++k) sacc += (double)__ldg(p + sk * k);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sacc += __shfl_xor_sync(0xffffffffu, sacc, o);
        if (tx == 0) red[ty] = sacc;
        __syncthreads();
        if (t == 0) {
            double r = 0.0;
            for (int u = 0; u < 8; ++u) r += red[u];
            part[blk] = r;
        }
        __syncthreads();
    }
}

// part 3: one block per instance sums its tiles' partials in a fixed order
__global__ void __launch_bounds__(256) k_inst_sum(const Inst* __restrict__ inst, int len, const double* __restrict__ part,
                                                  double* __restrict__ out) {
    __shared__ double red[8];
    const Inst& I = inst[blockIdx.x];
    const int t0 = I.am[1][0];
    const int nt = I.am[1][1] * I.am[1][2] * ((I.nk + len - 1) / len);
    double s = 0.0;
    for (int u = threadIdx.x; u < nt; u += blockDim.x) s += part[t0 + u];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double r = 0.0;
        for (int u = 0; u < 8; ++u) r += red[u];
        out[blockIdx.x] = r;
    }
}

// part 4: lam_pre = lam - (S / A) w with S = sum(lam) of the instance and
// w = wfix in fixed point, on the vertices of the listed interface cells
// (the only nodes with a weight).  Each vertex's weight is taken and cleared
// for the next step by one atomic exchange, so exactly one thread applies
// it, whatever the list order.
template <typename T>
__global__ void __launch_bounds__(128) k_mass_apply(Flat fl, const Mass* __restrict__ mass,
                                                    const double* __restrict__ ssum, const unsigned* __restrict__ list,
                                                    const unsigned* __restrict__ count, T* __restrict__ lam,
                                                    unsigned long long* __restrict__ wfix) {
    const unsigned n = *count;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x) {
        const long long l = list[e];
        const int q = node_instance(fl, l);
        const Mass M = mass[q];
        if (!mass_on(M)) continue;
        const Inst& I = fl.inst[q];
        const long long sj = I.ni, sk = (long long)I.ni * I.nj;
        const long long o[8] = {l, l + 1, l + 1 + sj, l + sj, l + sk, l + 1 + sk, l + 1 + sj + sk, l + sj + sk};
        const double r = ssum[q] / M.A;
#pragma unroll
        for (int v = 0; v < 8; ++v) {
            const long long w = (long long)atomicExch(wfix + o[v], 0ull);
            if (w != 0) lam[o[v]] = (T)((double)lam[o[v]] - r * ((double)w * kVolUnit));
        }
    }
}

// fixed-point Davies-Salmond volume of every cell of one instance
__global__ void k_cell_hex(long long off, int ni, int nj, int nk, const double* __restrict__ x,
                           const double* __restrict__ y, const double* __restrict__ z, long long* __restrict__ cellfix) {
    const long long ncell = (long long)(ni - 1) * (nj - 1) * (nk - 1);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell;
         c += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(c % (ni - 1)), j = (int)((c / (ni - 1)) % (nj - 1));
        const int k = (int)(c / ((long long)(ni - 1) * (nj - 1)));
        const long long sj = ni, sk = (long long)ni * nj;
        const long long l = off + i + sj * j + sk * k;
        const long long o[8] = {l, l + 1, l + 1 + sj, l + sj, l + sk, l + 1 + sk, l + 1 + sj + sk, l + sj + sk};
        double C[8][3];
#pragma unroll
        for (int v = 0; v < 8; ++v) { C[v][0] = x[o[v]]; C[v][1] = y[o[v]]; C[v][2] = z[o[v]]; }
        cellfix[l] = __double2ll_rn(hex_volume(C) * kVolScale);
    }
}

// FP32 coordinates of the vertices 1..7 of every cell relative to its vertex
// 0, the differences formed in FP64 (cell_gather's values), 24 floats per
// cell by base node
__global__ void k_cell_rel(long long off, int ni, int nj, int nk, const double* __restrict__ x,
                           const double* __restrict__ y, const double* __restrict__ z, float* __restrict__ rel) {
    const long long ncell = (long long)(ni - 1) * (nj - 1) * (nk - 1);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell;
         c += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(c % (ni - 1)), j = (int)((c / (ni - 1)) % (nj - 1));
        const int k = (int)(c / ((long long)(ni - 1) * (nj - 1)));
        const long long sj = ni, sk = (long long)ni * nj;
        const long long l = off + i + sj * j + sk * k;
        const long long o[8] = {l, l + 1, l + 1 + sj, l + sj, l + sk, l + 1 + sk, l + 1 + sj + sk, l + sj + sk};
        const double X0[3] = {x[l], y[l], z[l]};
        float q[24];
#pragma unroll
        for (int v = 1; v < 8; ++v) {
            q[3 * (v - 1)] = (float)(x[o[v]] - X0[0]);
            q[3 * (v - 1) + 1] = (float)(y[o[v]] - X0[1]);
            q[3 * (v - 1) + 2] = (float)(z[o[v]] - X0[2]);
        }
        q[21] = q[22] = q[23] = 0.f;
        float4* r = reinterpret_cast<float4*>(rel + 24 * l);
#pragma unroll
        for (int u = 0; u < 6; ++u) r[u] = make_float4(q[4 * u], q[4 * u + 1], q[4 * u + 2], q[4 * u + 3]);
    }
}

// ================================================================ adjoint
// Reverse of face `face` of bcond_lsm: for every node b of that face plane,
// lam(n1) += a lam(b), lam(n2) += c lam(b), lam(b) = 0, with (a, c) the
// face rule's weights (the BigPhi switch evaluated on the forward value of
// n2 at that point of the face sequence).  Distinct nodes of one plane have
// distinct targets, so the kernel needs no atomics.
template <typename T>
__global__ void k_adj_face(Flat fl, int face0, long long nplane, int nface, BC bc, int kind,
                           const T* __restrict__ phin, const T* __restrict__ in, const T* __restrict__ out, T c1, T c2,
                           T* lam) {
    // nface 2: face0 (odd) and the opposite face face0 - 1 of the same axis in
    // one launch (no shared nodes, no shared targets when the axis has at
    // least 6 nodes in every instance)
    const long long tt = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (tt >= nplane * nface) return;
    const bool second = tt >= nplane;
    const int face = second ? face0 - 1 : face0;
    const long long t = second ? tt - nplane : tt;
    if (!face_on(bc, face)) return;
    const int ax = face >> 1;
    int lo = 0, hi = fl.ninst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (fl.inst[mid].fpre[ax] <= t) lo = mid; else hi = mid - 1;
    }
    const Inst& I = fl.inst[lo];
    const unsigned r = (unsigned)(t - I.fpre[ax]), ni = I.ni, nj = I.nj;
    int i, j, k;
    if (ax == 0) { i = (face == 0) ? 0 : I.ni - 1; j = (int)(r % nj); k = (int)(r / nj); }
    else if (ax == 1) { j = (face == 2) ? 0 : I.nj - 1; i = (int)(r % ni); k = (int)(r / ni); }
    else { k = (face == 4) ? 0 : I.nk - 1; i = (int)(r % ni); j = (int)(r / ni); }
    const int dir = (face & 1) ? -1 : 1;     // inward direction
    const long long sj = I.ni, sk = (long long)I.ni * I.nj;
    const long long st = ax == 0 ? 1 : (ax == 1 ? sj : sk);
    const long long l = I.off + i + sj * j + sk * k;
    const T g = lam[l];
    T a, c;
    const int type = bc.type[face];
    if (type == 0) { a = T(1); c = T(0); }
    else if (type == 2) { a = T(2); c = T(-1); }
    else {
        const int i2 = ax == 0 ? i + 2 * dir : i, j2 = ax == 1 ? j + 2 * dir : j, k2 = ax == 2 ? k + 2 * dir : k;
        T v2;
        if (kind == 0) {
            P0Stage<T> p0{phin, in, out, I.off, sj, sk, I.ni, I.nj, I.nk, c1, c2};
            v2 = bc_value<T, false>(bc, p0, I.ni, I.nj, I.nk, i2, j2, k2, ax);
        } else {
            P0Src<T> p0{out, I.off, sj, sk};
            v2 = bc_value<T, false>(bc, p0, I.ni, I.nj, I.nk, i2, j2, k2, ax);
        }
        if (fabs(v2) >= T(bc.BigPhi)) { a = T(1); c = T(0); }
        else { a = T(4.0 / 3.0); c = T(-1.0 / 3.0); }
    }
    lam[l + dir * st] += a * g;
    lam[l + 2 * dir * st] += c * g;
    lam[l] = T(0);
}

// value of rec3 on a stencil with differences eL, eR and smoothness t1, t0, and
// its gradient (one reciprocal r)
template <typename T>
__device__ __forceinline__ T rec3_vg(T fC, T eL, T eR, T t1, T t0, T* dL, T* dC, T* dR) {
    const T h = eL - eR, q = t1 * t1, a1 = t0 * t0;
    const T r = wrcp(vfma(T(2), q, a1));
    const T v = q * r, z = T(4) * r * h;
    // h dv / d eL = 4 t1 a1 r^2 h eL, h dv / d eR = -4 t0 t1^2 r^2 h eR
    const T xL = t1 * a1 * r * z * eL, xR = -(t0 * q * r) * z * eR;
    *dL = v - T(0.5) + xL;
    *dC = T(1.5) - T(2) * v - xL + xR;
    *dR = v - xR;
    return vfma(v, h, vfma(T(-0.5), eL, fC));
}

// D = Phi+ - Phi- of a node and the gradient G = lp w dD/ds of lp w D over its
// stencil s = -2 .. 2, the orientation frozen by w; the neighbours and `edge`
// as for weno_wind
template <typename T>
__device__ __forceinline__ T stage_node_grad(T q0, T q1, T c, T q3, bool edge, T w, T lp, T (&G)[5]) {
    const T fL = edge ? q3 : q0, fC = edge ? c : q1;
    const T e0 = fL - fC, e1 = q1 - c, e2 = c - q3;
    const T t0 = vfma(e0, e0, T(1.0e-6)), t1 = vfma(e1, e1, T(1.0e-6)), t2 = vfma(e2, e2, T(1.0e-6));
    T dL, dC, dR, uL, uC, uR;
    const T vd = rec3_vg(c, e1, e2, t1, t2, &dL, &dC, &dR);
    const T vu = rec3_vg(fC, e0, edge ? -e1 : e1, t0, t1, &uL, &uC, &uR);
    const bool up = w > T(0);
    const T k = lp * fabs(w), D = vd - vu;
    const T g0 = edge ? T(0) : -k * uL, g1 = k * (dL - (edge ? uR : uC)), g3 = k * (dR - (edge ? uL : T(0)));
    G[0] = up ? g0 : T(0);
    G[1] = up ? g1 : g3;
    G[2] = k * (dC - (edge ? uC : uR));
    G[3] = up ? g3 : g1;
    G[4] = up ? T(0) : g0;
    return up ? D : -D;
}
// the same from the stencil
template <typename T>
__device__ __forceinline__ T stage_node_grad(T m2, T m1, T c, T p1, T p2, bool lo, bool hi, T w, T lp, T (&G)[5]) {
    const bool up = w > T(0);
    return stage_node_grad(up ? m2 : p2, up ? m1 : p1, c, up ? p1 : m1, up ? lo : hi, w, lp, G);
}

// Stage adjoint, x and z parts and the pointwise terms, on flat tiles (Inst's
// xw x xh columns and, where they are not whole rows, a rim of two nodes in x;
// row-major over the threads) marching in k.  At plane q a thread evaluates
// G_z of its node, which it adds to the sums of the nodes q - 2 .. q + 2 in
// registers, and G_x, whose outer components its neighbours take from shared
// memory (one barrier per plane, two buffers; a node next to a row's end has
// no component across it).  Plane q - 2 is then complete: lam_in = c2 lamP0 -
// c3 (acc_x + acc_z) (+ lamPhin + c1 lamP0 when last), lamPhin, lamW_x and
// lamW_z.  Eleven words per node are read or written (fifteen in a pass each,
// x by warps along their rows); issue-bound then and now.  Measured on 512 x
// 256 x 256 nodes: 265 + 243 -> 474 us, 128^3 25 + 23 -> 30 us, two FP64 grids
// of 40^3 48 + 70 -> 57 us; 128 threads, so that a barrier holds up few warps,
// eight blocks per SM (256 threads: 454, 31 and 65 us; three quarters of the
// warps 502 us).
template <typename T, typename O>
__global__ void __launch_bounds__(kAdjThreads, sizeof(T) == 4 ? 8 : 4) k_adj_stage_xz(const Inst* __restrict__ inst,
        Tiles tl, FieldsT<T> f, const T* __restrict__ in, const T* __restrict__ lamP0, T* __restrict__ lam_in,
        T* __restrict__ lamPhin, T* __restrict__ lamW0, T* __restrict__ lamW2, T c1, T c2, T c3, int last) {
    __shared__ T gx[2][4][kAdjThreads + 4];   // components 4, 3, 1, 0 of the block's nodes, two zeros around
    struct Pl {
        T s, lp, W0, W2, phin, w0, w2;   // in of plane q + 2; plane q; the old values of plane q - 2
    };
    const int t = threadIdx.x;
    if (t < 32) {
        const int r = t & 3;
        gx[t >> 4][(t >> 2) & 3][r < 2 ? r : kAdjThreads + r] = T(0);
    }
    for (int blk = blockIdx.x; blk < tl.n; blk += gridDim.x) {
        const ABrick ab = adj_brick(tl, blk);
        const Inst& I = inst[ab.inst];
        const int ni = I.ni, nj = I.nj, nk = I.nk;
        const int rim = I.xw < ni ? 2 : 0, ew = I.xw + 2 * rim;
        const int y = t / ew, x = t - y * ew;
        const int i = ab.i0 + x - rim, j = ab.j0 + y;
        const bool col = y < I.xh && i >= 0 && i < ni && j < nj;
        const bool core = col && x >= rim && x < I.xw + rim;
        const bool ij_int = col && i > 0 && i < ni - 1 && j > 0 && j < nj - 1;
        const bool ilo = i == 1, ihi = i == ni - 2;
        const int k0 = ab.k0, k1 = min(k0 + tl.len, nk);
        constexpr O E = sizeof(T);
        const O sk = E * (O)ni * (O)nj;
        O l = E * (O)I.off + E * (O)i + E * (O)ni * (O)j + sk * (O)(k0 - 2);   // plane q
        T s0 = T(0), s1 = T(0), s2 = T(0), s3 = T(0);
        T A0 = T(0), A1 = T(0), A2 = T(0), A3 = T(0);   // z sums of planes q - 2 .. q + 1
        T ax1 = T(0), ax2 = T(0), d1 = T(0), d2 = T(0), z1 = T(0), z2 = T(0), p1 = T(0), p2 = T(0);
        // what plane q needs, one plane ahead
        auto ld = [&](int q, O l, Pl& p) {
            p.s = p.lp = T(0);
            if (!col) return;
            if (q + 2 < nk && q + 2 <= k1 + 3) p.s = ldo(in, l + 2 * sk);
            if (q >= 0 && q < nk && q < k1 + 2) {
                p.lp = ldo(lamP0, l);
                p.W0 = ldo(f.W[0], l);
                p.W2 = ldo(f.W[2], l);
            }
            if (core && q - 2 >= k0 && q - 2 < k1) {
                p.phin = ldv(lamPhin, l - 2 * sk);
                p.w0 = ldv(lamW0, l - 2 * sk);
                p.w2 = ldv(lamW2, l - 2 * sk);
            }
        };
        if (col) {
            if (k0 >= 4) s0 = ldo(in, l - 2 * sk);
            if (k0 >= 3) s1 = ldo(in, l - sk);
            if (k0 >= 2) s2 = ldo(in, l);
            if (k0 >= 1) s3 = ldo(in, l + sk);
        }
        Pl a, b;
        ld(k0 - 2, l, a);
        auto plane = [&](int q, const Pl& c, Pl& n, T (*g)[kAdjThreads + 4]) {
            ld(q + 1, l + sk, n);
            const T s4 = c.s;
            const bool zin = q > 0 && q < nk - 1;
            T Gz[5] = {T(0), T(0), T(0), T(0), T(0)}, dz = T(0), dx = T(0), ax = T(0);
            if (zin && core && ij_int)
                dz = stage_node_grad(s0, s1, s2, s3, s4, q == 1, q == nk - 2, c.W2, c.lp, Gz);
            if (q >= k0 && q < k1) {
                T Gx[5] = {T(0), T(0), T(0), T(0), T(0)};
                if (zin && ij_int) {
                    const bool up = c.W0 > T(0);
                    const O o = up ? E : O(0) - E;   // in the array for every interior node
                    dx = stage_node_grad(ldo(in, l - 2 * o), ldo(in, l - o), s2, ldo(in, l + o), up ? ilo : ihi, c.W0,
                                         c.lp, Gx);
                }
                g[0][t + 2] = Gx[4];
                g[1][t + 2] = Gx[3];
                g[2][t + 2] = Gx[1];
                g[3][t + 2] = Gx[0];
                __syncthreads();
                ax = g[0][t] + g[1][t + 1] + Gx[2] + g[2][t + 3] + g[3][t + 4];
            }
            const T acc = A0 + Gz[0];
            if (core && q - 2 >= k0) {
                const O lo = l - 2 * sk;
                sto(lamW0, lo, c.w0 - c3 * p2 * d2);
                sto(lamW2, lo, c.w2 - c3 * p2 * z2);
                T r = c2 * p2 - c3 * (ax2 + acc);
                if (last) r += c.phin + c1 * p2;
                sto(lamPhin, lo, last ? T(0) : c.phin + c1 * p2);
                sto(lam_in, lo, r);
            }
            A0 = A1 + Gz[1];
            A1 = A2 + Gz[2];
            A2 = A3 + Gz[3];
            A3 = Gz[4];
            ax2 = ax1;
            ax1 = ax;
            d2 = d1;
            d1 = dx;
            z2 = z1;
            z1 = dz;
            p2 = p1;
            p1 = c.lp;
            s0 = s1;
            s1 = s2;
            s2 = s3;
            s3 = s4;
            l += sk;
        };
        for (int q = k0 - 2;;) {
            plane(q, a, b, gx[0]);
            if (++q >= k1 + 2) break;
            plane(q, b, a, gx[1]);
            if (++q >= k1 + 2) break;
        }
        __syncthreads();   // the next tile writes the buffers that this one's last plane reads
    }
}

// Stage adjoint, y part: flat tiles of Inst's yw x yh columns in (i, k),
// marching in j as the z part does in k; lam_in -= c3 acc, lamW_y -= c3 lamP0 D.
// 512 x 256 x 256: 242 -> 202 us, 128^3 22 -> 18 us, two FP64 grids of 40^3 70
// -> 41 us.
template <typename T, typename O>
__global__ void __launch_bounds__(kAdjThreads, sizeof(T) == 4 ? 12 : 4) k_adj_stage_y(const Inst* __restrict__ inst,
        Tiles tl, FieldsT<T> f, const T* __restrict__ in, const T* __restrict__ lamP0, T* __restrict__ lam_in,
        T* __restrict__ lamW1, T c3) {
    struct Pl {
        T s, lp, W, lin, w;   // in of row q + 2; row q; the old values of row q - 2
    };
    const int t = threadIdx.x;
    for (int blk = blockIdx.x; blk < tl.n; blk += gridDim.x) {
        const ABrick ab = adj_brick(tl, blk);
        const Inst& I = inst[ab.inst];
        const int ni = I.ni, nj = I.nj, nk = I.nk;
        const int y = t / I.yw, x = t - y * I.yw;
        const int i = ab.i0 + x, k = ab.k0 + y;
        const bool col = y < I.yh && i < ni && k < nk;
        const bool line = col && i > 0 && i < ni - 1 && k > 0 && k < nk - 1;
        const int m0 = ab.j0, m1 = min(m0 + tl.len, nj);
        constexpr O E = sizeof(T);
        const O st = E * (O)ni;
        O l = E * (O)I.off + E * (O)i + st * (O)nj * (O)k + st * (O)(m0 - 2);   // row q
        T s0 = T(0), s1 = T(0), s2 = T(0), s3 = T(0);
        T A0 = T(0), A1 = T(0), A2 = T(0), A3 = T(0);
        T z1 = T(0), z2 = T(0), p1 = T(0), p2 = T(0);
        auto ld = [&](int q, O l, Pl& p) {
            p.s = p.lp = T(0);
            if (!col) return;
            if (q + 2 < nj && q + 2 <= m1 + 3) p.s = ldo(in, l + 2 * st);
            if (q >= 0 && q < nj && q < m1 + 2) {
                p.lp = ldo(lamP0, l);
                p.W = ldo(f.W[1], l);
            }
            if (q - 2 >= m0 && q - 2 < m1) {
                p.lin = ldv(lam_in, l - 2 * st);
                p.w = ldv(lamW1, l - 2 * st);
            }
        };
        if (col) {
            if (m0 >= 4) s0 = ldo(in, l - 2 * st);
            if (m0 >= 3) s1 = ldo(in, l - st);
            if (m0 >= 2) s2 = ldo(in, l);
            if (m0 >= 1) s3 = ldo(in, l + st);
        }
        Pl a, b;
        ld(m0 - 2, l, a);
        auto row = [&](int q, const Pl& c, Pl& n) {
            ld(q + 1, l + st, n);
            const T s4 = c.s;
            T G[5] = {T(0), T(0), T(0), T(0), T(0)}, D = T(0);
            if (line && q > 0 && q < nj - 1)
                D = stage_node_grad(s0, s1, s2, s3, s4, q == 1, q == nj - 2, c.W, c.lp, G);
            const T acc = A0 + G[0];
            if (col && q - 2 >= m0) {
                const O lo = l - 2 * st;
                sto(lam_in, lo, c.lin - c3 * acc);
                sto(lamW1, lo, c.w - c3 * p2 * z2);
            }
            A0 = A1 + G[1];
            A1 = A2 + G[2];
            A2 = A3 + G[3];
            A3 = G[4];
            z2 = z1;
            z1 = D;
            p2 = p1;
            p1 = c.lp;
            s0 = s1;
            s1 = s2;
            s2 = s3;
            s3 = s4;
            l += st;
        };
        for (int q = m0 - 2;;) {
            row(q, a, b);
            if (++q >= m1 + 2) break;
            row(q, b, a);
            if (++q >= m1 + 2) break;
        }
    }
}

// Reinitialisation adjoint coefficients of one node from its inputs:
// with w = dtau s lam / (2 G) and the Godunov selections of the forward
// pass, A_m = w dG^2/dmen_m, B_m = w dG^2/dmas_m (a physical face's single
// difference goes to B on the low face, to A on the high face; lo / hi flag
// the node's faces).  Branch-free: with sigma = sign(s) both Godunov
// branches are one, P = sigma max(sigma bb, 0), Q = sigma min(sigma ff, 0),
// and w dG^2/dmen_m = dtau |s| lam / G sum_x M[m][x] (P chosen ? sigma P : 0).
template <typename T>
struct CoefIn {
    T d[7];     // d at the node, -x, +x, -y, +y, -z, +z (any finite value where outside)
    T s, lam;
    T M[9];
};

template <typename T>
__device__ __forceinline__ void coef_eval(const CoefIn<T>& c, T dtau, const bool (&lo)[3], const bool (&hi)[3],
                                          T (&A)[3], T (&B)[3]) {
    const T sg = c.s > T(0) ? T(1) : T(-1), sc = sg * c.d[0];
    T mas[3], men[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        const T fwd = vfma(sg, c.d[2 + 2 * m], -sc), bwd = vfma(-sg, c.d[1 + 2 * m], sc);
        mas[m] = hi[m] ? bwd : fwd;
        men[m] = lo[m] ? fwd : bwd;
    }
    T e[3], g[3];
    const T acc = godunov_sel_v<true>(mas, men, c.M, e, g);
    const T wgt = (c.s != T(0) && acc > T(0)) ? dtau * fabs(c.s) * c.lam * vrsqrt(acc) : T(0);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        const T gmen = c.M[3 * m] * e[0] + c.M[3 * m + 1] * e[1] + c.M[3 * m + 2] * e[2];
        const T gmas = c.M[3 * m] * g[0] + c.M[3 * m + 1] * g[1] + c.M[3 * m + 2] * g[2];
        A[m] = lo[m] ? T(0) : wgt * (hi[m] ? gmen + gmas : gmen);
        B[m] = hi[m] ? T(0) : wgt * (lo[m] ? gmen + gmas : gmas);
    }
}

// Reverse of one reinitialisation pseudo-step d' = d - dtau s (G(d) - 1):
//   lam_out(j) = lam(j) - sum_m [A_m(j) - B_m(j) - A_m(j+e_m) + B_m(j-e_m)]
// (adjoint map 0).  A block of 32 x kReinRY threads covers nodes i0-1 ..
// i0+30, j0-1 .. j0+kReinRY-2 and writes the inner 30 x (kReinRY-2); it
// marches in k.  Iteration k evaluates the coefficients of plane k and
// writes plane k-1.  Each node loads its own d, s, lam and metrics only:
// the x neighbours of d come by warp shuffles (the tile's edge lanes load
// the one outside), the y neighbours from the plane in shared memory (the
// edge rows load the one outside), the z neighbours from a register window
// (d is fetched two planes ahead, the rest one plane ahead).  The
// coefficients travel the same way: A_x / B_x by shuffles, A_y / B_y
// through shared memory, A_z / B_z in registers.  One barrier per plane,
// shared planes double-buffered (a buffer is rewritten two iterations
// later, after every thread has passed the barrier between).
template <typename T>
__global__ void __launch_bounds__(32 * kReinRY, sizeof(T) == 4 ? 2 : 1) k_adj_reinit(const Inst* __restrict__ inst,
        Tiles tl, FieldsT<T> f, const T* __restrict__ d, const T* __restrict__ lam,
        T* __restrict__ lam_out) {
    constexpr int RY = kReinRY;
    __shared__ T sD[2][RY + 2][32];   // row ty + 1 holds row ty (rows 0, RY + 1: padding)
    __shared__ T sA1[2][RY][32], sB1[2][RY][32];
    const unsigned FM = 0xffffffffu;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int blk = blockIdx.x; blk < tl.n; blk += gridDim.x) {
        const ABrick ab = adj_brick(tl, blk);
        const Inst& I = inst[ab.inst];
        const int ni = I.ni, nj = I.nj, nk = I.nk;
        const long long sj = ni, sk = (long long)ni * nj;
        const int i = ab.i0 - 1 + tx, j = ab.j0 - 1 + ty;
        const int k0 = ab.k0, k1 = min(k0 + tl.len, nk);
        const bool node = i >= 0 && i < ni && j >= 0 && j < nj;
        const bool out = node && tx >= 1 && tx <= 30 && ty >= 1 && ty <= RY - 2;
        const T dtau = ipar<T>(I.dtau, I.dtau64);
        const long long cb = I.off + i + sj * j;   // this column at k = 0
        // the neighbour outside the tile that edge lanes / rows load
        const int ox = tx == 0 ? -1 : (tx == 31 ? 1 : 0), oy = ty == 0 ? -1 : (ty == RY - 1 ? 1 : 0);
        const bool ldx = node && ox != 0 && i + ox >= 0 && i + ox < ni;
        const bool ldy = node && oy != 0 && j + oy >= 0 && j + oy < nj;
        auto ldd = [&](int k) { return node && k >= 0 && k < nk ? __ldg(d + cb + sk * k) : T(0); };
        // plane-k inputs other than d (plane k evaluated iff 0 <= k < nk, k <= k1)
        struct PlaneIn {
            T s, lam, ex, ey, M[9];
        };
        auto ldp = [&](int k, PlaneIn& q) {
            q.s = q.lam = q.ex = q.ey = T(0);
            if (node && k >= 0 && k < nk && k <= k1) {
                const long long l = cb + sk * k;
                q.s = __ldg(f.sgn + l);
                q.lam = __ldg(lam + l);
                if (ldx) q.ex = __ldg(d + l + ox);
                if (ldy) q.ey = __ldg(d + l + oy * sj);
#pragma unroll
                for (int c = 0; c < 9; ++c) q.M[c] = __ldg(f.m[c] + l);
            }
        };
        __syncthreads();   // the previous tile's readers of sD / sA1 / sB1 are done
        T dm = ldd(k0 - 2), dc = ldd(k0 - 1), dp = ldd(k0);   // d at k-1, k, k+1 for k = k0-1
        PlaneIn cur, nxt;
        ldp(k0 - 1, nxt);
        T Ap[3] = {T(0), T(0), T(0)}, Bp[3] = {T(0), T(0), T(0)}, Bz2 = T(0), lamp = T(0);
        int it = 0;
#pragma unroll 2
        for (int k = k0 - 1; k <= k1; ++k, ++it) {
            cur = nxt;
            const T dnn = ldd(k + 2);   // two planes ahead
            ldp(k + 1, nxt);
            sD[it & 1][ty + 1][tx] = dc;
            if (it > 0) {
                sA1[(it - 1) & 1][ty][tx] = Ap[1];
                sB1[(it - 1) & 1][ty][tx] = Bp[1];
            }
            __syncthreads();
            // neighbours of d at plane k (one-sided copies on physical faces)
            CoefIn<T> c;
            c.s = cur.s;
            c.lam = cur.lam;
#pragma unroll
            for (int q = 0; q < 9; ++q) c.M[q] = cur.M[q];
            c.d[0] = dc;
            const T xl = __shfl_up_sync(FM, dc, 1), xr = __shfl_down_sync(FM, dc, 1);
            c.d[1] = tx == 0 ? cur.ex : xl;
            c.d[2] = tx == 31 ? cur.ex : xr;
            c.d[3] = ty == 0 ? cur.ey : sD[it & 1][ty][tx];
            c.d[4] = ty == RY - 1 ? cur.ey : sD[it & 1][ty + 2][tx];
            c.d[5] = dm;
            c.d[6] = dp;
            const bool lo[3] = {i == 0, j == 0, k == 0}, hi[3] = {i == ni - 1, j == nj - 1, k == nk - 1};
            T A[3], B[3];
            coef_eval(c, dtau, lo, hi, A, B);
            // plane k-1: x neighbours by shuffles, y from shared memory
            const T ax = __shfl_down_sync(FM, Ap[0], 1);
            const T bx = __shfl_up_sync(FM, Bp[0], 1);
            const int ko = k - 1;
            if (out && ko >= k0 && ko < k1) {
                const int q = (it - 1) & 1;
                T t0 = Ap[0] - Bp[0];
                if (i < ni - 1) t0 -= ax;
                if (i > 0) t0 += bx;
                T t1 = Ap[1] - Bp[1];
                if (j < nj - 1) t1 -= sA1[q][ty + 1][tx];
                if (j > 0) t1 += sB1[q][ty - 1][tx];
                T t2 = Ap[2] - Bp[2];
                if (ko < nk - 1) t2 -= A[2];
                if (ko > 0) t2 += Bz2;
                lam_out[cb + sk * ko] = lamp - t0 - t1 - t2;
            }
            Bz2 = Bp[2];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                Ap[m] = A[m];
                Bp[m] = B[m];
            }
            lamp = cur.lam;
            dm = dc;
            dc = dp;
            dp = dnn;
        }
    }
}

template <typename T>
__global__ void k_adj_contra(Flat fl, FieldsT<T> f, const T* __restrict__ w0, const T* __restrict__ w1,
                             const T* __restrict__ w2, T* __restrict__ u0, T* __restrict__ u1, T* __restrict__ u2) {
    const long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    Node nd;
    if (!flat_node(fl, l, &nd)) return;
    const T dt = ipar<T>(fl.inst[nd.inst].dt, fl.inst[nd.inst].dt64);
    const T lw[3] = {w0[l], w1[l], w2[l]};
    T* out[3] = {u0, u1, u2};
#pragma unroll
    for (int c = 0; c < 3; ++c)
        out[c][l] += dt * (f.m[c][l] * lw[0] + f.m[3 + c][l] * lw[1] + f.m[6 + c][l] * lw[2]);
}

// ------------------------------------------------------------ dispatch
template <template <typename, int, int, int> class Fn, typename T, class... A>
void dispatch(int shape, A... a) {
    if constexpr (sizeof(T) == 8) {
        (void)shape;
        Fn<T, 32, 4, 2>::run(a...);   // FP64 (gradient checks): one tile shape
    } else {
        switch (shape) {
        case 0: Fn<T, 32, 4, 2>::run(a...); break;
        case 1: Fn<T, 32, 8, 1>::run(a...); break;
        case 2: Fn<T, 64, 4, 1>::run(a...); break;
        case 3: Fn<T, 32, 2, 4>::run(a...); break;
        default: Fn<T, 128, 2, 1>::run(a...); break;
        }
    }
}

#define LSM_BATCH_RUNNER(NAME, KERNEL, PARAMS, ARGS)                                   \
    template <typename T, int TX, int TY, int TZ>                                      \
    struct NAME {                                                                       \
        static void run PARAMS {                                                        \
            ProfScope ps_(#KERNEL, s);                                                  \
            KERNEL<T, TX, TY, TZ><<<grid, TX * TY * TZ, 0, s>>> ARGS;                   \
        }                                                                               \
    };

LSM_BATCH_RUNNER(RunContra, k_contra,
                 (int grid, const Inst* inst, const Brick* bi, int nb, FieldsT<T> f, cudaStream_t s),
                 (inst, bi, nb, f))
LSM_BATCH_RUNNER(RunBcFull, k_bc_full,
                 (int grid, const Inst* inst, const Brick* bi, int nb, BC bc, const T* src, T* dst, unsigned* err,
                  cudaStream_t s),
                 (inst, bi, nb, bc, src, dst, err))
LSM_BATCH_RUNNER(RunReinit, k_reinit,
                 (int grid, const Inst* inst, const Brick* bi, int nb, FieldsT<T> f, const T* din, T* dout,
                  unsigned* err, cudaStream_t s),
                 (inst, bi, nb, f, din, dout, err))
LSM_BATCH_RUNNER(RunSignReinit, k_sign_reinit,
                 (int grid, const Inst* inst, const Brick* bi, int nb, FieldsT<T> f, const T* p0, T* dout,
                  unsigned* err, cudaStream_t s),
                 (inst, bi, nb, f, p0, dout, err))

template <typename T, int TX, int TY, int TZ>
struct Occupancy {
    static void run(int kernel, int* out) {
        const int nt = TX * TY * TZ;
        (void)kernel;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, k_contra<T, TX, TY, TZ>, nt, 0);
    }
};

inline unsigned flat_blocks(long long n) { return (unsigned)((n + 255) / 256); }

}  // namespace

// ------------------------------------------------------------ launchers
template <typename T>
void contra(int shape, int grid, const Inst* inst, const Brick* bi, int nb, FieldsT<T> f, cudaStream_t s) {
    dispatch<RunContra, T>(shape, grid, inst, bi, nb, f, s);
}
template <typename T>
void stage(int grid, const Inst* inst, Tiles tl, bool wide, FieldsT<T> f, const T* phin, const T* phi1, T* out,
           double c1, double c2, double c3, cudaStream_t s) {
    ProfScope ps_("k_stage", s);
    auto go = [&](auto kernel) {
        kernel<<<grid, kStageThreads, 0, s>>>(inst, tl, f, phin, phi1, out, T(c1), T(c2), T(c3));
    };
    if (wide) go(k_stage<T, unsigned long long>);
    else go(k_stage<T, unsigned>);
}
template <typename T>
int stage_blocks_per_sm() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_stage<T, unsigned>, kStageThreads, 0);
    return n;
}
void stage_tma(int grid, const CUtensorMap* tm, int a_in, const Inst* inst, Tiles tl,
               FieldsT<float> f, const float* phin, const float* phi1, float* out, double c1, double c2, double c3,
               unsigned* err, cudaStream_t s) {
    ProfScope ps_("k_stage_tma", s);
    k_stage_tma<<<grid, 256, 0, s>>>(*tm, a_in, inst, tl, f, phin, phi1, out, (float)c1, (float)c2, (float)c3,
                                     err);
}
int stage_tma_blocks_per_sm() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_stage_tma, 256, 0);
    return n;
}
template <typename T>
void bc_stage(const Inst* inst, int ninst, long long nface, BC bc, const T* phin, const T* phi1, T* out, double c1,
              double c2, cudaStream_t s) {
    ProfScope ps_("k_bc_stage", s);
    k_bc_stage<T><<<flat_blocks(nface), 256, 0, s>>>(inst, ninst, nface, bc, phin, phi1, out, T(c1), T(c2));
}
template <typename T>
void bc_full(int shape, int grid, const Inst* inst, const Brick* bi, int nb, BC bc, const T* src, T* dst, unsigned* err,
             cudaStream_t s) {
    dispatch<RunBcFull, T>(shape, grid, inst, bi, nb, bc, src, dst, err, s);
}
template <typename T>
void bc_faces(const Inst* inst, int ninst, long long nface, BC bc, const T* src, T* dst, unsigned* err,
              cudaStream_t s) {
    ProfScope ps_("k_bc_faces", s);
    k_bc_faces<T><<<flat_blocks(nface), 256, 0, s>>>(inst, ninst, nface, bc, src, dst, err);
}
template <typename T>
void reinit(int shape, int grid, const Inst* inst, const Brick* bi, int nb, FieldsT<T> f, const T* din, T* dout,
            unsigned* err, cudaStream_t s) {
    dispatch<RunReinit, T>(shape, grid, inst, bi, nb, f, din, dout, err, s);
}
template <typename T>
void sign_reinit(int shape, int grid, const Inst* inst, const Brick* bi, int nb, FieldsT<T> f, const T* phi0,
                 T* dout, unsigned* err, cudaStream_t s) {
    dispatch<RunSignReinit, T>(shape, grid, inst, bi, nb, f, phi0, dout, err, s);
}
template <typename T>
void reinit_z(int kind, int grid, const Inst* inst, Tiles tl, FieldsT<T> f, const T* din, T* dout,
              T* dout2, T* cf, long long ld, unsigned* err, cudaStream_t s) {
    switch (kind) {
    case 0: {
        ProfScope ps_("k_reinit_z", s);
        k_reinit_z<T, false, false><<<grid, 256, 0, s>>>(inst, tl, f, din, dout, dout2, cf, ld, err);
        break;
    }
    case 1: {
        ProfScope ps_("k_reinit_rec_z", s);
        k_reinit_z<T, false, true><<<grid, 256, 0, s>>>(inst, tl, f, din, dout, dout2, cf, ld, err);
        break;
    }
    case 2: {
        ProfScope ps_("k_sign_reinit_z", s);
        k_reinit_z<T, true, false><<<grid, 256, 0, s>>>(inst, tl, f, din, dout, dout2, cf, ld, err);
        break;
    }
    default: {
        ProfScope ps_("k_sign_reinit_rec_z", s);
        k_reinit_z<T, true, true><<<grid, 256, 0, s>>>(inst, tl, f, din, dout, dout2, cf, ld, err);
        break;
    }
    }
}
void reinit_pair(int grid, const Inst* inst, Tiles tl, bool wide, FieldsT<float> f, const float* din, float* dout,
                 float* dout2, unsigned* err, cudaStream_t s) {
    ProfScope ps_("k_reinit_pair", s);
    auto go = [&](auto kernel) { kernel<<<grid, kPairThreads, 0, s>>>(inst, tl, f, din, dout, dout2, err); };
    if (wide) go(k_reinit_pair<unsigned long long>);
    else go(k_reinit_pair<unsigned>);
}
int reinit_pair_blocks_per_sm() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_reinit_pair<unsigned>, kPairThreads, 0);
    return n;
}
template <typename T>
int reinit_z_blocks_per_sm() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_reinit_z<T, true, true>, 256, 0);
    return n;
}
template <typename T>
void adj_reinit_c(int grid, const Inst* inst, Tiles tl, bool wide, const T* cf, long long ld, const T* lam, T* lam_out,
                  cudaStream_t s) {
    ProfScope ps_("k_adj_reinit_c", s);
    auto go = [&](auto kernel) { kernel<<<grid, kStageThreads, 0, s>>>(inst, tl, cf, ld, lam, lam_out); };
    if (wide) go(k_adj_reinit_c<T, unsigned long long>);
    else go(k_adj_reinit_c<T, unsigned>);
}
template <typename T>
int adj_reinit_c_blocks_per_sm() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_adj_reinit_c<T, unsigned>, kStageThreads, 0);
    return n;
}
template <typename T>
void bc_reinit(const Inst* inst, int ninst, long long nface, FieldsT<T> f, BC bc, const T* din, T* dout,
               cudaStream_t s) {
    ProfScope ps_("k_bc_reinit", s);
    k_bc_reinit<T><<<flat_blocks(nface), 256, 0, s>>>(inst, ninst, nface, bc, f, din, dout);
}
inline unsigned list_blocks() { return 152 * 32; }
template <typename T>
void volume(int grid2, const Inst* inst, Tiles tl, const Flat& fl, FieldsT<T> f, const T* phi,
            unsigned long long* acc, bool slope, unsigned* list, unsigned* count, cudaStream_t s) {
    cudaMemsetAsync(count, 0, sizeof(unsigned), s);
    {
        ProfScope ps_("k_vol_scan_z", s);
        if (tl.len == adj_shape(1).oz) k_vol_scan_z<T, true><<<grid2, 256, 0, s>>>(inst, tl, f, phi, acc, list, count);
        else k_vol_scan_z<T, false><<<grid2, 256, 0, s>>>(inst, tl, f, phi, acc, list, count);
    }
    if (slope) {
        ProfScope ps_("k_vol_iface_slope", s);
        k_vol_iface<T, true><<<list_blocks(), 128, 0, s>>>(fl, f, phi, list, count, acc);
    } else {
        ProfScope ps_("k_vol_iface", s);
        k_vol_iface<T, false><<<list_blocks(), 128, 0, s>>>(fl, f, phi, list, count, acc);
    }
}
void volume_final(int ninst, unsigned long long* acc, double* vols, const double* target, Mass* mass, Mass* mrec,
                  cudaStream_t s) {
    ProfScope ps_("k_volume_final", s);
    k_volume_final<<<(ninst + 127) / 128, 128, 0, s>>>(ninst, acc, vols, target, mass, mrec);
}
template <typename T>
void mass_shift(const Flat& fl, const Mass* mass, const T* src, T* dst, cudaStream_t s) {
    ProfScope ps_("k_mass_shift", s);
    k_mass_shift<T><<<(unsigned)std::min<long long>((fl.n + 255) / 256, 152 * 16), 256, 0, s>>>(fl, mass, src, dst);
}
template <typename T>
void mass_adjoint(const Inst* inst, Tiles tl, const Flat& fl, FieldsT<T> f, const T* phi_pre,
                  const Mass* mass, T* lam, unsigned long long* wfix, double* part, double* ssum, const unsigned* list,
                  const unsigned* count, cudaStream_t s) {
    {
        ProfScope ps_("k_mass_weights", s);
        k_mass_weights<T><<<list_blocks(), 128, 0, s>>>(fl, f, phi_pre, list, count, mass, wfix);
    }
    {
        ProfScope ps_("k_tile_sum", s);
        k_tile_sum<T><<<std::min(tl.n, 152 * 8), 256, 0, s>>>(inst, tl, lam, part);
    }
    {
        ProfScope ps_("k_inst_sum", s);
        k_inst_sum<<<fl.ninst, 256, 0, s>>>(inst, tl.len, part, ssum);
    }
    ProfScope ps_("k_mass_apply", s);
    k_mass_apply<T><<<list_blocks(), 128, 0, s>>>(fl, mass, ssum, list, count, lam, wfix);
}
void w64(long long off, long long n, double dt, const double* const* m64, const double* const* u64,
         double* const* w, cudaStream_t s) {
    ProfScope ps_("k_w64", s);
    k_w64<<<(unsigned)std::min<long long>((n + 255) / 256, 152 * 16), 256, 0, s>>>(off, n, dt, m64, u64, w);
}
void cell_hex(long long off, int ni, int nj, int nk, const double* x, const double* y, const double* z,
              long long* cellfix, cudaStream_t s) {
    const long long ncell = (long long)(ni - 1) * (nj - 1) * (nk - 1);
    ProfScope ps_("k_cell_hex", s);
    k_cell_hex<<<(unsigned)std::min<long long>((ncell + 255) / 256, 152 * 16), 256, 0, s>>>(off, ni, nj, nk, x, y, z,
                                                                                             cellfix);
}
void cell_rel(long long off, int ni, int nj, int nk, const double* x, const double* y, const double* z, float* rel,
              cudaStream_t s) {
    const long long ncell = (long long)(ni - 1) * (nj - 1) * (nk - 1);
    ProfScope ps_("k_cell_rel", s);
    k_cell_rel<<<(unsigned)std::min<long long>((ncell + 255) / 256, 152 * 16), 256, 0, s>>>(off, ni, nj, nk, x, y, z,
                                                                                             rel);
}
int max_blocks_per_sm(int shape, int kernel) {
    int n = 0;
    dispatch<Occupancy, float>(shape, kernel, &n);
    return n;
}
template <typename T>
int vol_scan_blocks_per_sm() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_vol_scan_z<T, true>, 256, 0);
    return n;
}

template <typename T>
void adj_face(const Flat& fl, int face, long long nplane, int nface, BC bc, int kind, const T* phin, const T* in,
              const T* out, double c1, double c2, T* lam, cudaStream_t s) {
    ProfScope ps_("k_adj_face", s);
    k_adj_face<T><<<flat_blocks(nplane * nface), 256, 0, s>>>(fl, face, nplane, nface, bc, kind, phin, in, out, T(c1),
                                                              T(c2), lam);
}
template <typename T>
void adj_stage(const int (&grid)[2], const Inst* inst, const Tiles (&tl)[2], bool wide, FieldsT<T> f, const T* in,
               const T* lamP0, T* lam_in, T* lamPhin, T* lamW0, T* lamW1, T* lamW2, double c1, double c2, double c3,
               bool last, cudaStream_t s) {
    {
        ProfScope ps_("k_adj_stage_xz", s);
        auto go = [&](auto kernel) {
            kernel<<<grid[0], kAdjThreads, 0, s>>>(inst, tl[0], f, in, lamP0, lam_in, lamPhin, lamW0, lamW2, T(c1),
                                                   T(c2), T(c3), last ? 1 : 0);
        };
        if (wide) go(k_adj_stage_xz<T, unsigned long long>);
        else go(k_adj_stage_xz<T, unsigned>);
    }
    ProfScope ps_("k_adj_stage_y", s);
    auto go = [&](auto kernel) {
        kernel<<<grid[1], kAdjThreads, 0, s>>>(inst, tl[1], f, in, lamP0, lam_in, lamW1, T(c3));
    };
    if (wide) go(k_adj_stage_y<T, unsigned long long>);
    else go(k_adj_stage_y<T, unsigned>);
}
template <typename T>
int adj_stage_blocks_per_sm(int part) {
    int n = 0;
    if (part == 0) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_adj_stage_xz<T, unsigned>, kAdjThreads, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_adj_stage_y<T, unsigned>, kAdjThreads, 0);
    return n;
}
template <typename T>
void adj_reinit(int grid, const Inst* inst, Tiles tl, FieldsT<T> f, const T* d, const T* lam,
                T* lam_out, cudaStream_t s) {
    ProfScope ps_("k_adj_reinit", s);
    k_adj_reinit<T><<<grid, 32 * kReinRY, 0, s>>>(inst, tl, f, d, lam, lam_out);
}
template <typename T>
int adj_reinit_blocks_per_sm() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_adj_reinit<T>, 32 * kReinRY, 0);
    return n;
}
template <typename T>
void adj_contra(const Flat& fl, FieldsT<T> f, const T* w0, const T* w1, const T* w2, T* u0, T* u1, T* u2,
                cudaStream_t s) {
    ProfScope ps_("k_adj_contra", s);
    k_adj_contra<T><<<flat_blocks(fl.n), 256, 0, s>>>(fl, f, w0, w1, w2, u0, u1, u2);
}

#define LSM_BATCH_INSTANTIATE(T)                                                                                      \
    template void contra<T>(int, int, const Inst*, const Brick*, int, FieldsT<T>, cudaStream_t);                       \
    template int stage_blocks_per_sm<T>();                                                                      \
    template void stage<T>(int, const Inst*, Tiles, bool, FieldsT<T>, const T*, const T*, T*, double, double, double,  \
                           cudaStream_t);                                                                         \
    template void bc_stage<T>(const Inst*, int, long long, BC, const T*, const T*, T*, double, double, cudaStream_t);   \
    template void bc_full<T>(int, int, const Inst*, const Brick*, int, BC, const T*, T*, unsigned*, cudaStream_t);      \
    template void bc_faces<T>(const Inst*, int, long long, BC, const T*, T*, unsigned*, cudaStream_t);                 \
    template void bc_reinit<T>(const Inst*, int, long long, FieldsT<T>, BC, const T*, T*, cudaStream_t);              \
    template void reinit<T>(int, int, const Inst*, const Brick*, int, FieldsT<T>, const T*, T*, unsigned*,             \
                            cudaStream_t);                                                                            \
    template void sign_reinit<T>(int, int, const Inst*, const Brick*, int, FieldsT<T>, const T*, T*, unsigned*,      \
                                 cudaStream_t);                                                                   \
    template void reinit_z<T>(int, int, const Inst*, Tiles, FieldsT<T>, const T*, T*, T*, T*, long long, \
                              unsigned*, cudaStream_t);                                                         \
    template int reinit_z_blocks_per_sm<T>();                                                                   \
    template void adj_reinit_c<T>(int, const Inst*, Tiles, bool, const T*, long long, const T*, T*,           \
                                  cudaStream_t);                                                                \
    template int adj_reinit_c_blocks_per_sm<T>();                                                               \
    template void volume<T>(int, const Inst*, Tiles, const Flat&, FieldsT<T>, const T*,                \
                            unsigned long long*, bool, unsigned*, unsigned*, cudaStream_t);                          \
    template int vol_scan_blocks_per_sm<T>();                                                                   \
    template void mass_shift<T>(const Flat&, const Mass*, const T*, T*, cudaStream_t);                                 \
    template void mass_adjoint<T>(const Inst*, Tiles, const Flat&, FieldsT<T>, const T*, const Mass*,  \
                                  T*, unsigned long long*, double*, double*, const unsigned*, const unsigned*,          \
                                  cudaStream_t);                                                                     \
    template void adj_face<T>(const Flat&, int, long long, int, BC, int, const T*, const T*, const T*, double, double, \
                              T*, cudaStream_t);                                                                     \
    template void adj_stage<T>(const int (&)[2], const Inst*, const Tiles (&)[2], bool, FieldsT<T>, const T*,          \
                               const T*, T*, T*, T*, T*, T*, double, double, double, bool, cudaStream_t);          \
    template int adj_stage_blocks_per_sm<T>(int);                                                                  \
    template void adj_reinit<T>(int, const Inst*, Tiles, FieldsT<T>, const T*, const T*, T*,            \
                                cudaStream_t);                                                                \
    template int adj_reinit_blocks_per_sm<T>();                                                                     \
    template void adj_contra<T>(const Flat&, FieldsT<T>, const T*, const T*, const T*, T*, T*, T*, cudaStream_t);

LSM_BATCH_INSTANTIATE(float)
LSM_BATCH_INSTANTIATE(double)

}  // namespace batch
}  // namespace lsm
