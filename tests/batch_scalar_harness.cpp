// Test harness (built by tests/test_batch_scalar_cpu.py): the scalar device
// functions of the batched path (csrc/lsm_batch_scalar.cuh) on the host.
#include "lsm_batch_scalar.cuh"

using namespace lsm::batch;

namespace {

// the reconstruction with its weight as one rounded quotient
double rec3_quotient(double fL, double fC, double fR) {
    const double eL = fL - fC, eR = fC - fR;
    const double t0 = std::fma(eR, eR, 1.0e-6), t1 = std::fma(eL, eL, 1.0e-6), a0 = (t1 + t1) * t1;
    const double w0 = a0 / std::fma(t0, t0, a0);
    return std::fma(w0, std::fma(0.5, fL + fR, -fC), std::fma(1.5, fC, -0.5 * fL));
}

}  // namespace

// s: n stencils of 5 along the wind; r: per stencil the library's value and
// the expression's of a face, and of the difference of a node's two faces
extern "C" void weno_faces(long n, const double* s, double* r) {
    for (long q = 0; q < n; ++q) {
        const double* v = s + 5 * q;
        r[4 * q] = rec3(v[0], v[1], v[2]);
        r[4 * q + 1] = rec3_quotient(v[0], v[1], v[2]);
        r[4 * q + 2] = weno_wind(v[0], v[1], v[2], v[3], false);
        r[4 * q + 3] = rec3_quotient(v[1], v[2], v[3]) - rec3_quotient(v[0], v[1], v[2]);
    }
}

// conversions by the integer pipes; ok: where they hold
extern "C" void convert(long n, const float* f, double* wide, const double* d, float* near, unsigned char* ok) {
    for (long q = 0; q < n; ++q) {
        bool a = true, b = true;
        wide[q] = widen(f[q], a);
        near[q] = narrow(d[q], b);
        ok[2 * q] = a;
        ok[2 * q + 1] = b;
    }
}

// v: n x 3 doubles and 8 floats of a stage's combination; r: by the integer pipes and by conversions
extern "C" void combine(long n, const double* W, const float* v, float* r) {
    for (long q = 0; q < n; ++q) {
        const double* w = W + 3 * q;
        const float* a = v + 8 * q;
        r[2 * q] = stage_band(w[0], w[1], w[2], a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]);
        r[2 * q + 1] = stage_band_any(w[0], w[1], w[2], a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]);
    }
}
