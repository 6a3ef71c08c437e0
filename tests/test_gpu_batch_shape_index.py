"""The shape index of an autotuned batch names its pseudo-steps' plan: a batch
made with it, without autotuning, launches no more kernels per step (an index
of the brick table for a batch that runs pairs launched single pseudo-steps)."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,lo,hi", [(1, 9, 12), (3, 12, 24), (32, 32, 96)])
def test_index_of_a_tuned_batch(lib_built, count, lo, hi):
    from nslsm.batch import LevelSetBatch
    rng = np.random.default_rng(3)
    dims = [tuple(int(v) for v in rng.integers(lo, hi + 1, 3)) for _ in range(count)]

    def batch(**kw):
        b = LevelSetBatch([(*n, 1e-3, 1e-2, 0.1) for n in dims], RNitermax=5, **kw)
        for q, n in enumerate(dims):
            x, y, z = (np.asfortranarray(a) for a in np.meshgrid(*(np.linspace(0, 1, m) for m in n), indexing="ij"))
            met = [np.asfortranarray(np.zeros((3, *n)) + np.eye(3)[m].reshape(3, 1, 1, 1) * (n[m] - 1))
                   for m in range(3)]
            b.set_geometry(q, x, y, z, *met)
            b.set_velocity(q, np.zeros((4, *n), order="F"))
            b.set_phi(q, np.asfortranarray(z - 0.4))
        b.step(1)
        return b

    tuned = batch()
    again = batch(autotune=False, shape=tuned.shape[0])
    assert again.shape[0] == tuned.shape[0]
    assert again.launches_per_step <= tuned.launches_per_step
