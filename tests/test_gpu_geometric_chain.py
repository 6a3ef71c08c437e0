"""The distance chains of the geometric reinitialisation against the CPU
oracle, bit for bit, where their kernels branch: noisy surfaces (distances
that fall by more than a factor 2 from pnode to pnode), surfaces on and
near the nodes (short edges, equal distances), several surfaces inside one
+-4 box, coordinates far from the origin (wide FP32 enclosures) and
phicorrected values of any size (above 10, tiny, zero).  The tolerance is
equality: only which distances are evaluated differs from the sequential
loops."""
import numpy as np
import pytest

import cases
import oracle as O
from test_gpu_geometric import seed
from test_gpu_parity import G, P, dev, host

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def surface(kind):
    n = (23, 17, 20)
    rng = np.random.default_rng(7)
    X, Y, Z = np.meshgrid(*(np.linspace(0, 1, m) for m in n), indexing="ij")
    phi = Z - 0.48 - 0.1 * np.sin(6 * X) * np.cos(4 * Y)
    if kind == "noisy":
        phi = phi + 0.02 * rng.standard_normal(n)
    elif kind == "on_nodes":
        phi = np.round(phi * 16) / 16 + np.where(rng.random(n) < 0.1, 1e-12, 0.0)
    elif kind == "layers":
        phi = np.sin(9 * np.pi * Z + X) * 0.1
    elif kind == "far":
        X, Y, Z = X + 5000.0, Y - 300.0, Z * 0.2
    return O.make_grid(*n), cases.F(X), cases.F(Y), cases.F(Z), cases.F(phi)


@pytest.mark.parametrize("start", ["seed", "any"])
@pytest.mark.parametrize("kind", ["noisy", "on_nodes", "layers", "far"])
def test_distance_chains_bit_identical(ls, oracle, kind, start):
    g, x, y, z, phi = surface(kind)
    p = O.make_params()
    pc = seed(phi)
    if start == "any":
        rng = np.random.default_rng(3)
        pc = cases.F(rng.standard_normal(phi.shape) * rng.choice([20.0, 0.1, 1e-3, 0.0], phi.shape))
    ref, rids, _ = oracle.geometric_reinitialisation(g, p, phi, x, y, z, 0.0, pc)
    out, ids, _ = ls.geometric_reinitialisation(G(g), P(p), *map(dev, (phi, x, y, z)), 0.0, dev(pc))
    assert np.array_equal(host(ids), rids)
    assert np.array_equal(host(out), ref)
