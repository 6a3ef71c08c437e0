"""The geometric reinitialisation against the CPU oracle, bit for bit, on
grids with a node at the coordinate origin (a corner or the middle) and a
surface 0.3 to 0.003 cells from it, on cells of aspect 1 to 100, smooth and
rough: point and distance are small there while the triangles are a cell wide.
The tolerance is equality: only which distances are evaluated differs from the
sequential loops."""
import numpy as np
import pytest

import cases
import oracle as O
from test_geometric_chain_cpu import SEEDS, deciding, grid, rough
from test_gpu_geometric import seed
from test_gpu_parity import G, P, dev, host

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def check(ls, oracle, g, p, phi, x, y, z):
    pc = seed(phi)
    ref, rids, _ = oracle.geometric_reinitialisation(g, p, phi, x, y, z, 0.0, pc)
    out, ids, _ = ls.geometric_reinitialisation(G(g), P(p), *map(dev, (phi, x, y, z)), 0.0, dev(pc))
    assert np.array_equal(host(ids), rids)
    assert np.array_equal(host(out), ref)


@pytest.mark.parametrize("place", ["corner", "middle"])
@pytest.mark.parametrize("aspect", [1, 10, 100])
def test_origin_nodes_bit_identical(ls, oracle, place, aspect):
    n, at = 13, 0 if place == "corner" else 6
    g, p = O.make_grid(n, n, n), O.make_params()
    for off in (0.3, 0.03, 0.003):
        for amp in (0.0, 0.3, 2.0):
            rng = np.random.default_rng([aspect, int(off * 1000), int(amp * 10)])
            h = np.array([1.0, 1.0, 1.0 / aspect]) * rng.choice([0.02, 1.0])
            x, y, z = (cases.F(c) for c in grid(n, at, h))
            phi = cases.F(rough(rng, n, at, h, off, amp))
            check(ls, oracle, g, p, phi, x, y, z)


@pytest.mark.parametrize("case", SEEDS[::3])
def test_surfaces_that_decide_by_an_enclosure(ls, oracle, case):
    n, _, xyz, phi = deciding(case)
    check(ls, oracle, O.make_grid(n, n, n), O.make_params(), cases.F(phi), *(cases.F(c) for c in xyz))
