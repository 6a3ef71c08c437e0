"""FP32 pseudo-steps run two at a time against the same steps one at a time.

Both compute every value by the same operations in the same order, so phi has
to agree bit for bit: on instances narrower and wider than a tile, with fewer
rows than a tile holds, with one or several marches in k, and for every number
of pseudo-steps left over.
"""
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
    a, b = _batch(R, 0), _batch(R, 5)   # 0: brick table, one at a time; 5: in pairs
    a.step(2, volumes=False)
    b.step(2, volumes=False)
    assert b.launches_per_step == a.launches_per_step - (R - 1) // 2
    for q in range(len(SIZES)):
        assert np.array_equal(a.get_phi(q), b.get_phi(q)), SIZES[q]
