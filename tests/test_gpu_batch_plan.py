"""lsm_batch_launches_per_step before the first step, where no autotuning
decides it: what the steps then take."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("shape", range(6))
def test_launches_per_step_known_before(lib_built, precision, shape):
    from nslsm.batch import LevelSetBatch
    n = (9, 8, 10)
    b = LevelSetBatch([(*n, 1e-3, 1e-2, 0.1)], RNitermax=5, autotune=False, shape=shape, precision=precision)
    before = b.launches_per_step
    x, y, z = (np.asfortranarray(a) for a in np.meshgrid(*(np.linspace(0, 1, m) for m in n), indexing="ij"))
    met = [np.asfortranarray(np.zeros((3, *n)) + np.eye(3)[m].reshape(3, 1, 1, 1) * (n[m] - 1)) for m in range(3)]
    b.set_geometry(0, x, y, z, *met)
    b.set_velocity(0, np.zeros((4, *n), order="F"))
    b.set_phi(0, np.asfortranarray(z - 0.4))
    b.step(1)
    assert b.launches_per_step == before
