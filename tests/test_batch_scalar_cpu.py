"""Scalar device functions of the batched path (csrc/lsm_batch_scalar.cuh) on
the CPU, bit for bit: the FP64 reconstruction's weight is one rounded
quotient, and the conversions on the integer pipes are IEEE conversions
wherever they say that they hold, which is the whole normal range."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ns-lsm-single-phase_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("needs g++")
    out = str(tmp_path_factory.mktemp("scalar") / "libscalar.so")
    r = subprocess.run([gxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I",
                        os.path.join(HERE, "simt"), "-I", CSRC, os.path.join(HERE, "batch_scalar_harness.cpp"), "-o",
                        out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(out)


def ptr(a):
    return C.c_void_p(a.ctypes.data)


@pytest.mark.parametrize("scale", [1e-4, 1e-3, 1e-2, 1.0, 100.0])
def test_fp64_weight_is_one_rounded_quotient(lib, scale):
    rng = np.random.default_rng(1)
    n = 200000
    s = np.ascontiguousarray(rng.standard_normal((n, 1)) + scale * rng.standard_normal((n, 5)) *
                             10.0 ** rng.uniform(-2, 0, (n, 5)))
    r = np.empty((n, 4))
    lib.weno_faces(C.c_long(n), ptr(s), ptr(r))
    assert np.array_equal(r[:, 0], r[:, 1])
    assert np.array_equal(r[:, 2], r[:, 3])


def floats(n, seed):
    """Bit patterns of every exponent, ends of the significand mixed in."""
    g = np.random.default_rng(seed)
    frac = g.integers(0, 1 << 23, n, dtype=np.uint32)
    k, near = g.integers(0, 4, n), g.integers(0, 4, n, dtype=np.uint32)
    frac = np.where(k == 1, near, np.where(k == 2, (1 << 23) - 1 - near, frac)).astype(np.uint32)
    return (g.integers(0, 2, n, dtype=np.uint32) << np.uint32(31) | g.integers(0, 256, n, dtype=np.uint32) <<
            np.uint32(23) | frac).view(np.float32)


def test_conversions(lib):
    n = 2000000
    g = np.random.default_rng(3)
    f = floats(n, 4)
    f[:4] = 0.0, -0.0, np.inf, np.nan
    # doubles around floats: between two of them, half-way, a unit beside half-way
    d = np.ldexp(g.choice([1.0, -1.0], n) * (1 + g.integers(0, 1 << 23, n) / 2.0 ** 23),
                 g.integers(-160, 140, n)).astype(np.float64)
    half = np.ldexp(1.0, np.frexp(d)[1] - 25) * g.choice([0.0, 0.5, 1.0, 1.5], n)
    with np.errstate(all="ignore"):
        d = d + np.sign(d) * half
        d[::3] = np.nextafter(d[::3], np.inf)
        d[1::3] = np.nextafter(d[1::3], -np.inf)
        d[::11] = g.standard_normal(d[::11].size)
        d[:4] = 0.0, -0.0, np.inf, np.nan
        wide, near, ok = np.empty(n), np.empty(n, np.float32), np.empty((n, 2), np.uint8)
        lib.convert(C.c_long(n), ptr(f), ptr(wide), ptr(d), ptr(near), ptr(ok))
        a, b = ok[:, 0] != 0, ok[:, 1] != 0
        mag = np.abs(f)
        assert np.array_equal(a, (mag == 0) | ((mag >= np.float32(2.0 ** -126)) & np.isfinite(f)))
        assert np.array_equal(wide[a].view(np.uint64), f[a].astype(np.float64).view(np.uint64))
        size = np.abs(d)
        assert np.array_equal(b, (size >= 2.0 ** -126) & (size < 2.0 ** 127))
        assert np.array_equal(near[b].view(np.uint32), d[b].astype(np.float32).view(np.uint32))


def test_stage_combination(lib):
    g = np.random.default_rng(5)
    n = 300000
    W = g.standard_normal((n, 3)) * 10.0 ** g.uniform(-3, 2, (n, 3))
    v = (g.standard_normal((n, 8)) * 10.0 ** g.uniform(-4, 1, (n, 8))).astype(np.float32)
    v[::50] = floats(v[::50].size, 6).reshape(-1, 8)
    v[::7, 1] = 0.0
    r = np.empty((n, 2), np.float32)
    with np.errstate(all="ignore"):
        lib.combine(C.c_long(n), ptr(W), ptr(v), ptr(r))
    same = (r.view(np.uint32)[:, 0] == r.view(np.uint32)[:, 1]) | (np.isnan(r).all(1))
    assert same.all()
