"""The live reinitialisation with many allowed iterations: it stops soon after
convergence (launches counted), also where far more are allowed than any
workspace could hold, and runs on through several host looks, converging in any
of them, as the CPU oracle does.  Tolerance: 1e-13 normwise for the few
iterations of the other tests, growing with their number (CUDA's sin and cos)."""
import numpy as np
import pytest

import cases
import oracle as O
from test_gpu_parity import G, P, dev, host

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def front(oracle):
    g, x, y, z, _, _ = cases.curvilinear(34, 11, 10, seed=2)
    csi, eta, zet, _ = oracle.mg_metrics(g, x, y, z)
    return g, cases.F(1.07 * (z - 0.45) + 0.01 * np.sin(3 * x)), csi, eta, zet


def params(R, tol, dt=0.04):
    return O.make_params(epslsm=0.1, RNitermax=R, RNtimestep=dt, epsReinitialisation=tol)


@pytest.mark.parametrize("R", [17, 1000, 2**31 - 1])
def test_stops_soon_after_convergence(ls, oracle, front, R):
    g, phi, *met = front
    ref, it = oracle.reinitialisation_test2(g, params(5, 0.1), phi, *met)
    assert it == 4
    args = [dev(a) for a in (phi, *met)]
    n0 = ls.launches
    got, n = ls.reinitialisation_test2(G(g), P(params(R, 0.1)), *args)
    assert n == it and cases.relerr(host(got), ref) <= 1e-13
    assert ls.launches - n0 <= 3 * 16 + 10


@pytest.mark.parametrize("R,tol,dt,want", [
    (16, 0.0, 0.001, 16), (17, 0.0, 0.001, 17), (48, 0.0, 0.001, 48), (130, 0.0, 0.001, 130),
    (300, 0.09, 0.002, 19), (300, 0.08, 0.002, 34), (300, 0.09, 0.001, 46), (300, 0.08, 0.001, 77)])
def test_through_several_looks(ls, oracle, front, R, tol, dt, want):
    g, phi, *met = front
    p = params(R, tol, dt)
    ref, it = oracle.reinitialisation_test2(g, p, phi, *met)
    got, n = ls.reinitialisation_test2(G(g), P(p), *(dev(a) for a in (phi, *met)))
    assert n == it == want and cases.relerr(host(got), ref) <= 1e-13 * max(1.0, it / 5)
