"""FP32 batches with 64-bit offsets (what a batch of 2^30 nodes and more runs)
against the 32-bit ones, each in a process of its own: phi of steps with paired
pseudo-steps and the gradients of a recorded run, bit for bit."""
import os
import subprocess
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def dump(path):
    from test_gpu_reinit_pair import SIZES, _batch
    out = {}
    b = _batch(5, 5)
    b.step(2, volumes=False)
    for q in range(len(SIZES)):
        out["phi%d" % q] = b.get_phi(q)
    b = _batch(3, 5)
    b.forward_record(2, 1)
    for q, n in enumerate(SIZES):
        b.set_grad_phi(q, np.asfortranarray(np.random.default_rng(q).standard_normal(n)))
    b.backward()
    for q in range(len(SIZES)):
        out["gp%d" % q], out["gq%d" % q] = b.get_grad_phi0(q), b.get_grad_velocity(q)
    np.savez(path, **out)


def test_fp32_offsets_of_both_widths_agree(lib_built, tmp_path):
    got = []
    for wide in ("0", "1"):
        f = str(tmp_path / ("w%s.npz" % wide))
        env = dict(os.environ, PYTHONPATH=os.pathsep.join(sys.path), LSM_BATCH_WIDE=wide)
        r = subprocess.run([sys.executable, "-c", "import test_gpu_wide_fp32 as t; t.dump(%r)" % f], env=env,
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        got.append(np.load(f))
    assert len(got[0].files) == 21
    for k in got[0].files:
        assert np.isfinite(got[0][k]).all() and np.abs(got[0][k]).max() > 0, k
        assert np.array_equal(got[0][k], got[1][k]), k
