"""The stage adjoint and the reverse pseudo-step on flat tiles: instances wider
than a tile (a rim in x), of whole rows, and longer than a march, with 32- and
64-bit offsets (a process of its own), against the FP64 torch tape to the 1e-10
of the other adjoint tests."""
import os
import subprocess
import sys
from types import SimpleNamespace

import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [(300, 6, 7), (129, 9, 40), (40, 70, 6), (7, 8, 90)]


def check():
    import lsm_tape as T
    from nslsm.configs import _mesh
    from test_gpu_adjoint import NSTEPS, _adjoint, _batch, _rel, _weights
    oracle = O.Oracle()
    cases = []
    for shape in SHAPES:
        X, Y, Z = _mesh(*shape)
        X, Y, Z = X + 0.05 * Y, Y - 0.03 * Z, Z + 0.04 * X
        F = lambda a: np.asfortranarray(a, dtype=np.float64)  # noqa: E731
        q = np.zeros((4,) + shape, order="F")
        q[1] = 0.6 * np.sin(2 * np.pi * X + Y)
        q[2] = -0.4 * np.cos(2 * np.pi * X)
        q[3] = 0.2 * np.sin(2 * np.pi * Y) - 0.1
        h = 1.0 / (max(shape) - 1)
        it = SimpleNamespace(grid=SimpleNamespace(shape=shape), x=F(X), y=F(Y), z=F(Z),
                             phi0=F(Z - 0.5 - 0.04 * np.cos(2 * np.pi * (2 * X + Y))), q=q, dtau=0.5 * h, eps=1.5 * h)
        g = O.make_grid(*shape)
        csi, eta, zet, aj = oracle.mg_metrics(g, it.x, it.y, it.z)
        smax = max(float(np.abs(m[0] * q[1] + m[1] * q[2] + m[2] * q[3]).max()) for m in (csi, eta, zet))
        cases.append(dict(it=it, g=g, csi=csi, eta=eta, zet=zet, aj=aj, dt=0.4 / smax))
    b, wts = _batch(cases, 2), _weights(cases)
    gphi, gq = _adjoint(b, cases, wts)
    for k, c in enumerate(cases):
        M = T.metrics_torch(c["csi"], c["eta"], c["zet"], "cuda")
        p = T.to_torch(c["it"].phi0, "cuda").requires_grad_(True)
        q = T.to_torch(c["it"].q, "cuda").requires_grad_(True)
        out = T.run(p, q, M, c["dt"], c["it"].dtau, c["it"].eps, 2, NSTEPS)
        (out * T.to_torch(wts[k], "cuda")).sum().backward()
        assert _rel(gphi[k], np.asfortranarray(p.grad.cpu().numpy().T)) <= 1e-10, SHAPES[k]
        assert _rel(gq[k], np.asfortranarray(q.grad.cpu().numpy().T)) <= 1e-10, SHAPES[k]


@pytest.mark.parametrize("wide", ["", "1"])
def test_adjoint_on_flat_tiles_matches_torch_tape(oracle, lib_built, wide):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(sys.path))
    env.pop("LSM_BATCH_WIDE", None)
    if wide:
        env["LSM_BATCH_WIDE"] = wide
    r = subprocess.run([sys.executable, "-c", "import test_gpu_adj_flat as t; t.check()"], env=env, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
