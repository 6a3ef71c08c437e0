// Enough of CUDA's device dialect to run this repository's warp kernels on the
// host (tests only): the 32 lanes of a warp are fibers that take turns, each
// running up to its next warp-wide operation.  Every lane has to make the same
// sequence of full-mask operations.  Found before CUDA's own header by the
// tests' include path.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <ucontext.h>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __constant__ static const
#define __shared__ static
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __launch_bounds__(...)

struct uint3 { unsigned x, y, z; };
struct alignas(16) float4 { float x, y, z, w; };
struct float2 { float x, y; };
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
inline float2 make_float2(float x, float y) { return {x, y}; }

static uint3 threadIdx, blockIdx, blockDim{1, 1, 1}, gridDim{1, 1, 1};

template <class T> inline T __ldg(const T* p) { return *p; }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline int max(int a, int b) { return a > b ? a : b; }
inline int min(int a, int b) { return a < b ? a : b; }
inline double __longlong_as_double(long long v) { double d; std::memcpy(&d, &v, 8); return d; }
inline float __double2float_rd(double d) { const float f = (float)d; return (double)f > d ? nextafterf(f, -INFINITY) : f; }
inline float __double2float_ru(double d) { const float f = (float)d; return (double)f < d ? nextafterf(f, INFINITY) : f; }
inline float __uint_as_float(unsigned v) { float f; std::memcpy(&f, &v, 4); return f; }
inline unsigned __float_as_uint(float f) { unsigned v; std::memcpy(&v, &f, 4); return v; }
inline double __hiloint2double(int h, int l) { return __longlong_as_double((long long)((uint64_t)(unsigned)h << 32 | (unsigned)l)); }
inline int __double2hiint(double d) { uint64_t u; std::memcpy(&u, &d, 8); return (int)(u >> 32); }
inline int __double2loint(double d) { uint64_t u; std::memcpy(&u, &d, 8); return (int)(unsigned)u; }
using std::isfinite;
inline float rsqrtf(float x) { return 1.0f / sqrtf(x); }
inline unsigned atomicOr(unsigned* p, unsigned v) { const unsigned o = *p; *p |= v; return o; }

namespace simt {

struct Warp {
    ucontext_t main, ctx[32];
    std::vector<char> stack[32];
    std::function<void()> body;
    uint64_t slot[2][32];
    unsigned round[32];
    unsigned lane = 0, base = 0;
};
inline Warp& warp() { static Warp w; return w; }
inline void enter(unsigned lane) {
    warp().lane = lane;
    threadIdx.x = warp().base + lane;
}
inline void trampoline() {
    Warp& w = warp();
    const unsigned me = w.lane;
    w.body();
    if (me < 31) { enter(me + 1); setcontext(&w.ctx[me + 1]); }
    setcontext(&w.main);
}
// every lane's value, once all have come here
inline const uint64_t* exchange(uint64_t v) {
    Warp& w = warp();
    const unsigned me = w.lane, b = w.round[me]++ & 1u;
    w.slot[b][me] = v;
    const unsigned next = (me + 1) & 31u;
    if (w.round[next] + 1 < w.round[me]) abort();
    enter(next);
    swapcontext(&w.ctx[me], &w.ctx[next]);
    return w.slot[b];
}
// `f` on the lanes of one warp, whose first thread is `base` of the block
inline void run(unsigned base, std::function<void()> f) {
    Warp& w = warp();
    w.body = f;
    w.base = base;
    for (unsigned l = 0; l < 32; ++l) {
        w.stack[l].resize(1 << 18);
        w.round[l] = 0;
        getcontext(&w.ctx[l]);
        w.ctx[l].uc_stack.ss_sp = w.stack[l].data();
        w.ctx[l].uc_stack.ss_size = w.stack[l].size();
        w.ctx[l].uc_link = nullptr;
        makecontext(&w.ctx[l], trampoline, 0);
    }
    enter(0);
    swapcontext(&w.main, &w.ctx[0]);
}

template <class T> inline uint64_t pack(T v) { uint64_t u = 0; std::memcpy(&u, &v, sizeof v); return u; }
template <class T> inline T unpack(uint64_t u) { T v; std::memcpy(&v, &u, sizeof v); return v; }

}  // namespace simt

inline unsigned __ballot_sync(unsigned, bool p) {
    const uint64_t* s = simt::exchange(p);
    unsigned m = 0;
    for (int l = 0; l < 32; ++l) m |= (unsigned)(s[l] != 0) << l;
    return m;
}
inline bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
template <class T> inline T __shfl_sync(unsigned, T v, int l) { return simt::unpack<T>(simt::exchange(simt::pack(v))[l & 31]); }
template <class T> inline T __shfl_xor_sync(unsigned, T v, int o) {
    const int me = (int)simt::warp().lane;
    return simt::unpack<T>(simt::exchange(simt::pack(v))[(me ^ o) & 31]);
}
template <class T> inline T __shfl_up_sync(unsigned, T v, int o) {
    const int me = (int)simt::warp().lane;
    return simt::unpack<T>(simt::exchange(simt::pack(v))[me >= o ? me - o : me]);
}
inline void __syncwarp() { simt::exchange(0); }
inline void __syncthreads() { abort(); }   // kernels of one warp only
