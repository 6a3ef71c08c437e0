// Test harness (built by tests/test_soft64_cpu.py): exposes the fixed-point
// FP64 operations (csrc/lsm_soft64.cuh, host instantiation) on arrays.
// `ulps` moves the FP32 seeds, standing for the approximate instructions.
#include "lsm_soft64.cuh"

extern "C" void soft64_run(int op, long n, const double* a, const double* b, double* r, int ulps) {
    using namespace lsm;
    soft64_seed_ulps() = ulps;
    double q;
    for (long i = 0; i < n; ++i) {
        switch (op) {
        case 0: r[i] = sdiv(a[i], b[i]); break;
        case 1: r[i] = ssqrt(a[i]); break;
        case 2: udiv2(a[i], b[i], b[i], &r[i], &q); break;
        case 3: r[i] = umul0(a[i], b[i]); break;
        case 4: r[i] = usqr(a[i]); break;
        default: r[i] = gt0(a[i]) ? 1.0 : (lt0(a[i]) ? -1.0 : 0.0); break;
        }
    }
    soft64_seed_ulps() = 0;
}
