"""The FP64 operations on the integer pipes (csrc/lsm_soft64.cuh) on the
device: every argument that the FP32 seeds can get, whose results may be two
units in the last place from the correctly rounded ones (the CPU test moves
them by as many), and the operations against CUDA's operators bit for bit."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from test_soft64_cpu import CSRC, HERE, operands, same

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from nslsm.build import ARCH, nvcc
    out = str(tmp_path_factory.mktemp("soft64") / "libsoft64_gpu.so")
    r = subprocess.run([nvcc(), *ARCH, "-O3", "-std=c++17", "--fmad=false", "-shared", "-Xcompiler", "-fPIC", "-I", CSRC,
                        HERE + "/soft64_gpu.cu", "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(out)


def test_every_seed_within_two_units(lib):
    worst = torch.zeros(2, dtype=torch.int32, device="cuda")
    assert lib.soft64_seeds(C.c_void_p(worst.data_ptr())) == 0
    assert (worst.cpu().numpy() <= 2).all(), worst


@pytest.mark.parametrize("lo,hi", [(0, 2047), (1000, 1050)])
def test_operations_equal_cudas(lib, lo, hi):
    n = 1 << 21
    a, b = operands(n, 11, lo, hi), operands(n, 12, lo, hi)
    b[::7] = np.nextafter(a[::7], b[::7])
    with np.errstate(all="ignore"):
        a[::5] = np.nextafter(a[::5] * a[::5], np.inf)   # roots next to a 53-bit number
    r = torch.empty((n, 8), dtype=torch.float64, device="cuda")
    t = [torch.from_numpy(v).cuda() for v in (a, b)]
    assert lib.soft64_ops(C.c_longlong(n), *(C.c_void_p(v.data_ptr()) for v in (*t, r))) == 0
    r = r.cpu().numpy()
    for q in (0, 1):
        assert same(np.ascontiguousarray(r[:, q]), np.ascontiguousarray(r[:, 4 + q]))
    if lo == 1000:   # products and squares have the narrower range
        for q in (2, 3):
            k = np.abs(a) < 2.0 ** 400
            assert same(np.ascontiguousarray(r[k, q]), np.ascontiguousarray(r[k, 4 + q]))
