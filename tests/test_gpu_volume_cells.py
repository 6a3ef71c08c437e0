"""The FP64 water volume on the GPU against the CPU oracle where its kernel
branches: chunks of cells that end inside rows, all-water and all-air grids
(walls only), water against every wall, every marching-tetrahedra case
(random signs with exact zeros, values within epsilon and tiny ones), and a
ghosted subdomain.  Per-cell volumes and the band are equal bit for bit; the
sums, formed in another order and the bulk from the faces of the water's
surface, agree to 1e-12 (normwise, as in the other volume tests)."""
import numpy as np
import pytest

import cases
import oracle as O
from test_gpu_parity import G, dev, host

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def grid(kind, seed=0):
    shape = {"small": (5, 4, 6), "ragged": (37, 11, 9), "large": (70, 51, 60)}.get(kind, (19, 14, 12))
    g, x, y, z, phi, _ = cases.curvilinear(*shape, seed=4)
    rng = np.random.default_rng(seed)
    if kind == "signs":
        phi = rng.standard_normal(shape)
        v = np.array([0.0, -0.0, 1e-310, -1e-310, 1e-17, -1e-17, 2.0 ** -52, -(2.0 ** -52)])
        phi = cases.F(np.where(rng.random(shape) < 0.4, rng.choice(v, shape), phi))
    elif kind == "water":
        phi = cases.F(np.abs(phi) + 0.1)
    elif kind == "air":
        phi = cases.F(-np.abs(phi) - 0.1)
    return g, x, y, z, phi


@pytest.mark.parametrize("kind", ["small", "ragged", "large", "signs", "water", "air"])
def test_volume_against_oracle(ls, oracle, kind):
    for seed in range(3 if kind == "signs" else 1):
        g, x, y, z, phi = grid(kind, seed)
        a = [dev(v) for v in (phi, x, y, z)]
        assert np.array_equal(host(ls.cell_water_volumes(G(g), *a)), oracle.cell_water_volumes(g, phi, x, y, z))
        v, nodes = ls.total_water_volume(G(g), *a, with_nodes=True)
        rv, rnodes = oracle.total_water_volume(g, phi, x, y, z, with_nodes=True)
        assert np.array_equal(host(nodes), rnodes)
        scale = max(abs(rv[3]), 1e-300)
        assert np.abs(v - rv).max() <= 1e-12 * scale, (v, rv)


def test_volume_of_a_ghosted_subdomain(ls, oracle):
    _, x, y, z, phi, _ = cases.curvilinear(21, 16, 13, seed=6)
    g = O.make_grid(21, 16, 13, igp=2, jgp=2, kgp=2, physical=(1, 0, 0, 1, 1, 0))
    v = ls.total_water_volume(G(g), *(dev(a) for a in (phi, x, y, z)))
    rv = oracle.total_water_volume(g, phi, x, y, z)
    assert np.abs(v - rv).max() <= 1e-12 * rv[3]
