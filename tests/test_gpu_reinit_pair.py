"""Kernels on flat tiles: FP32 pseudo-steps run two at a time against the same
steps one at a time, and the RK stage against the oracle.

Both forms of a pseudo-step compute every value by the same operations in the same order, so phi has
to agree bit for bit: on instances narrower and wider than a tile, with fewer
rows than a tile holds, with one or several marches in k, and for every number
of pseudo-steps left over.
"""
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = [(40, 30, 9), (140, 11, 5), (700, 5, 6), (6, 90, 7), (33, 34, 71), (5, 5, 5), (522, 8, 5)]


def _batch(R, shape):
    from nslsm.batch import LevelSetBatch
    b = LevelSetBatch([(*n, 2e-3, 0.3 / max(n), 3.0 / max(n)) for n in SIZES], RNitermax=R, autotune=False, shape=shape)
    for q, n in enumerate(SIZES):
        rng = np.random.default_rng(q)
        x, y, z = np.meshgrid(*(np.linspace(0.0, 1.0, m) for m in n), indexing="ij")
        met = [np.asfortranarray(rng.normal(0.0, 0.2, (3, *n)) + np.eye(3)[m].reshape(3, 1, 1, 1) * (n[m] - 1))
               for m in range(3)]
        f = [np.asfortranarray(a) for a in (x, y, z)]
        b.set_geometry(q, *f, *met)
        b.set_velocity(q, np.asfortranarray(rng.normal(0.0, 1.0, (4, *n))))
        b.set_phi(q, np.asfortranarray(0.2 - np.sqrt((x - 0.4) ** 2 + (y - 0.5) ** 2 + (z - 0.5) ** 2)))
    return b


@pytest.mark.parametrize("R", [2, 3, 4, 5])
def test_pairs_equal_single_pseudo_steps(lib_built, R):
    check_pairs(R)


def check_pairs(R):
    a, b = _batch(R, 0), _batch(R, 5)   # 0: brick table, one at a time; 5: in pairs
    a.step(2, volumes=False)
    b.step(2, volumes=False)
    assert b.launches_per_step == a.launches_per_step - (R - 1) // 2
    for q in range(len(SIZES)):
        assert np.array_equal(a.get_phi(q), b.get_phi(q)), SIZES[q]


@pytest.mark.parametrize("offsets", ["32", "64"])
def test_flat_tiles_match_fp64_oracle(oracle, lib_built, offsets):
    """The FP64 RK stage and (64-bit offsets) the FP32 pairs in a process of
    their own; widths below, at and above a tile's."""
    import subprocess
    import sys
    code = "import test_gpu_reinit_pair as t; t.check_stage()" + ("; t.check_pairs(5)" if offsets == "64" else "")
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(sys.path))
    env.pop("LSM_BATCH_WIDE", None)
    if offsets == "64":
        env["LSM_BATCH_WIDE"] = "1"
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]


def check_stage():
    """Three RK stages with their faces, about a hundred FP64 operations on values near 1 per node
    in another order than the oracle's: 1e-12."""
    import oracle as O
    from nslsm import configs
    from nslsm.batch import LevelSetBatch
    o = O.Oracle()
    for k, n in enumerate([(40, 30, 9), (256, 5, 6), (300, 7, 5), (5, 6, 70), (77, 67, 5)]):
        it = configs.batched_instances(n_inst=1, lo=5, hi=5, seed=k)[0]
        rng = np.random.default_rng(k)
        x, y, z = (np.asfortranarray(a + 0.02 * np.sin(3 * b)) for a, b in zip(*[
            np.meshgrid(*(np.linspace(0.0, 1.0, m) for m in n), indexing="ij")] * 2))
        phi = np.asfortranarray(z - 0.5 - 0.1 * np.cos(5 * x + 3 * y))
        q = np.asfortranarray(rng.normal(0.0, 1.0, (4, *n)))
        g = O.make_grid(*n)
        csi, eta, zet, aj = o.mg_metrics(g, x, y, z)
        dt = 0.3 / max(float(np.abs((m * q[1:4]).sum(0)).max()) for m in (csi, eta, zet))
        p = O.make_params(epslsm=it.eps, delti_lsm=dt, RNitermax=0, RNtimestep=it.dtau, BigPhi=5.0)
        ref, _ = o.levelsetmethod(g, p, q, csi, eta, zet, aj, phi, phi, x, y, z, 1)
        b = LevelSetBatch([(*n, dt, it.dtau, it.eps)], RNitermax=0, precision="fp64")
        b.set_geometry(0, x, y, z, csi, eta, zet)
        b.set_velocity(0, q)
        b.set_phi(0, phi)
        b.step(1, volumes=False)
        assert float(np.abs(b.get_phi(0) - ref).max()) <= 1e-12, n
