"""The FP64 operations on the integer pipes (csrc/lsm_soft64.cuh) against IEEE
arithmetic, bit for bit, on the CPU: random operands over the whole range
(zeros, subnormals, infinities and NaN where the operation takes them),
significands at the ends of [1, 2) and next to each other, squares and their
neighbours; the FP32 seeds moved by up to two units in the last place, which
covers the error bounds of rcp.approx (1 ulp) and rsqrt.approx (2^-22.9)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ns-lsm-single-phase_gb300", "csrc")
DIV, SQRT, DIV2, MUL, SQR, SIGN = range(6)


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("needs g++")
    out = str(tmp_path_factory.mktemp("soft64") / "libsoft64.so")
    r = subprocess.run([gxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", CSRC,
                        os.path.join(HERE, "soft64_harness.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(out)

    def f(op, a, b, ulps=0):
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        r = np.empty_like(a)
        lib.soft64_run(op, C.c_long(a.size), *(C.c_void_p(x.ctypes.data) for x in (a, b, r)), ulps)
        return r
    return f


def operands(n, seed, lo=0, hi=2047):
    """Bit patterns with exponent fields lo .. hi and special significands mixed in."""
    g = np.random.default_rng(seed)
    frac = g.integers(0, 1 << 52, n, dtype=np.uint64)
    k = g.integers(0, 6, n)
    near = g.integers(0, 8, n, dtype=np.uint64)
    frac = np.where(k == 1, near, np.where(k == 2, (1 << 52) - 1 - near, np.where(k == 3, frac & ~np.uint64(0xFFFFFFFF),
                                                                                  frac))).astype(np.uint64)
    e = g.integers(lo, hi + 1, n, dtype=np.uint64)
    s = g.integers(0, 2, n, dtype=np.uint64)
    return (s << np.uint64(63) | e << np.uint64(52) | frac).view(np.float64)


def same(x, y):
    return ((x.view(np.uint64) == y.view(np.uint64)) | (np.isnan(x) & np.isnan(y))).all()


@pytest.mark.parametrize("ulps", [-2, 0, 2])
def test_division_and_root(run, ulps):
    n = 400000
    with np.errstate(all="ignore"):
        for lo, hi in ((0, 2047), (1000, 1050)):
            a, b = operands(n, 1, lo, hi), operands(n, 2, lo, hi)
            b[::7] = np.nextafter(a[::7], b[::7])       # quotients next to 1
            assert same(run(DIV, a, b, ulps), a / b)
            assert same(run(SQRT, a, b, ulps), np.sqrt(a))
            q = np.abs(a[(np.abs(a) < 1e150) & (np.abs(a) > 1e-150)]) ** 2
            for v in (q, np.nextafter(q, 0.0), np.nextafter(q, np.inf)):
                assert same(run(SQRT, v, v, ulps), np.sqrt(v))
        a, b = operands(n, 3, 600, 1400), operands(n, 4, 600, 1400)
        assert same(run(DIV2, a, b, ulps), a / b)


def test_products_and_signs(run):
    n = 400000
    a, b = operands(n, 5, 600, 1400), operands(n, 6, 600, 1400)
    a[::11] = 0.0
    b[::13] = -0.0
    assert same(run(MUL, a, b), a * b)
    a = operands(n, 7, 523, 1522)
    assert same(run(SQR, a, a), a * a)
    assert (run(SQR, np.array([0.0, -1e-200]), np.zeros(2)) == 0.0).all()
    a = operands(n, 8)
    a[:3] = 0.0, -0.0, np.nan
    want = np.where(a > 0, 1.0, np.where(a < 0, -1.0, 0.0))
    assert same(run(SIGN, a, a), want)
