"""The bulk water volume in FP64: its error against extended precision for a
small body far from the grid's first node (the cells' volumes are formed from
their own edges, so the total is good to the rounding of a sum: 5e-16), its
agreement with the cells' own volumes, and a coordinate inside the water that
is no number."""
import math

import numpy as np
import pytest

import cases
import oracle as O
from test_gpu_parity import G, dev, host

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def corners(a):
    s = (slice(None, -1), slice(1, None))
    return [a[s[i], s[j], s[k]] for i, j, k in ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0),
                                                (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))]


def bulk(x, y, z, phi):
    """The water cells' volume: the origin-free sum of their six face terms in extended precision."""
    C = [np.stack(c, -1) for c in zip(*(corners(a.astype(np.longdouble)) for a in (x, y, z)))]
    mid = sum(C) / 8
    v = 0
    for a, b, c, d in ((0, 3, 2, 1), (4, 5, 6, 7), (0, 1, 5, 4), (3, 7, 6, 2), (0, 4, 7, 3), (1, 2, 6, 5)):
        v = v + ((C[a] + C[b] + C[c] + C[d] - 4 * mid) * np.cross(C[c] - C[a], C[d] - C[b])).sum(-1) / 24
    return v[np.all([p > 2.0 ** -52 for p in corners(phi)], axis=0)].sum()


def body(n, r):
    """A ball of r cells' radius next to the last node of n^3 curved cells."""
    X, Y, Z = np.meshgrid(*(np.linspace(0, 1, n),) * 3, indexing="ij")
    c = 1 - (r + 3) / n
    phi = r / n - np.sqrt((X - c) ** 2 + (Y - c) ** 2 + (Z - c) ** 2)
    xyz = X + 0.3 / n * np.sin(9 * Y + 3 * Z), Y + 0.3 / n * np.cos(8 * Z), Z + 0.2 / n * np.sin(7 * X)
    return (O.make_grid(n, n, n), cases.F(phi)) + tuple(cases.F(a) for a in xyz)


@pytest.mark.parametrize("n,r", [(96, 2.5), (160, 2.5), (160, 4.0), (160, 10.0), (64, 25.0)])
def test_small_body_far_from_the_first_node(ls, n, r):
    g, phi, x, y, z = body(n, r)
    want = bulk(x, y, z, phi)
    a = [dev(v) for v in (phi, x, y, z)]
    v = ls.total_water_volume(G(g), *a)
    assert abs(v[2] - want) <= 5e-16 * want
    cells = math.fsum(host(ls.cell_water_volumes(G(g), *a)).ravel())
    assert abs(v[3] - cells) <= 1e-15 * cells


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_coordinate_that_is_no_number(ls, oracle, bad):
    g, x, y, z, phi, _ = cases.curvilinear(21, 16, 13, seed=6)
    phi = cases.F(np.abs(phi) + 0.1)
    y[10, 8, 6] = bad
    v = ls.total_water_volume(G(g), *(dev(a) for a in (phi, x, y, z)))
    with np.errstate(all="ignore"):
        assert np.isnan(oracle.total_water_volume(g, phi, x, y, z)[3])
    assert np.isnan(v[2]) and np.isnan(v[3])
