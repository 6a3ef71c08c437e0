"""Scalar device functions of the batched path (csrc/lsm_batch_scalar.cuh) on
the CPU, bit for bit: the FP64 reconstruction's weight is one rounded
quotient."""
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
