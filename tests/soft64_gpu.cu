// Test kernels (built by tests/test_gpu_soft64_device.py): the FP64 operations
// on the integer pipes (csrc/lsm_soft64.cuh) on the device.
#include "lsm_soft64.cuh"

using namespace lsm;

namespace {

// every argument of the FP32 seeds: 2^23 + 1 significands in [1, 2] of the
// reciprocal, 2^24 + 1 in [1, 4] of the reciprocal root; the largest distance from
// the correctly rounded seed in units of the last place
__global__ void seeds(unsigned* worst) {
    const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q > 1u << 24) return;
    const unsigned b = 0x3F800000u + q;
    const double x = (double)__uint_as_float(b);
    auto off = [](unsigned got, double want) {
        const int d = (int)(got - __float_as_uint((float)want));
        return (unsigned)(d < 0 ? -d : d);
    };
    if (q <= 1u << 23) atomicMax(worst, off(rcp_bits(b), 1.0 / x));
    atomicMax(worst + 1, off(rsqrt_bits(b), 1.0 / sqrt(x)));
}

// r[0..3]: sdiv, ssqrt, umul0, usqr of a and b; r[4..7]: CUDA's operators
__global__ void ops(long long n, const double* a, const double* b, double* r) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= n) return;
    const double x = a[q], y = b[q];
    double* o = r + 8 * q;
    o[0] = sdiv(x, y); o[1] = ssqrt(x); o[2] = umul0(x, y); o[3] = usqr(x);
    o[4] = x / y; o[5] = sqrt(x); o[6] = __dmul_rn(x, y); o[7] = __dmul_rn(x, x);
}

}  // namespace

extern "C" int soft64_seeds(unsigned* worst) {
    cudaMemset(worst, 0, 8);
    seeds<<<(1 << 16) + 1, 256>>>(worst);
    return (int)cudaDeviceSynchronize();
}
extern "C" int soft64_ops(long long n, const double* a, const double* b, double* r) {
    ops<<<(unsigned)((n + 255) / 256), 256>>>(n, a, b, r);
    return (int)cudaDeviceSynchronize();
}
