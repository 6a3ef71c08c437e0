"""FP64 stage and pseudo-step on the GPU against the CPU oracle, bit for bit,
where their kernels branch: the three tile sizes of the stage with ragged
edges, sign changes of the contravariant velocity inside a tile, masks, and
values outside the range of the integer-pipe arithmetic (zeros, plateaus,
huge and tiny values, infinities and NaN).  The tolerance is equality: every
operation is rounded as written in either route."""
import numpy as np
import pytest

import cases
import oracle as O
from test_gpu_parity import G, P, dev, host

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def field(shape, kind, seed=0):
    rng = np.random.default_rng(seed)
    i, j, k = np.meshgrid(*(np.arange(n) for n in shape), indexing="ij")
    f = 0.2 * np.sin(0.31 * i) * np.cos(0.23 * j) + 0.05 * k - 0.3 + 0.02 * rng.standard_normal(shape)
    if kind == "extreme":
        f = np.where((k // 3) % 2 == 0, 9.9, f)                   # plateaus: exact zero differences
        v = np.array([0.0, -0.0, 1e-310, -4e-324, 1e-200, 1e30, -1e30, 1e160, -1e200, np.inf, -np.inf, np.nan])
        at = rng.integers(0, f.size, 4 * v.size)
        f.reshape(-1)[at] = np.resize(v, at.size)
    return cases.F(f)


def same(a, b):
    return np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("kind", ["plain", "extreme"])
@pytest.mark.parametrize("shape", [(4, 5, 4), (33, 6, 5), (64, 41, 37), (65, 101, 103)])
def test_stage_tiles_bit_exact(ls, oracle, shape, kind):
    """32 x 2 x 2, 32 x 4 x 2 and 32 x 8 x 4 tiles (the last shape) and their remainders."""
    g = O.make_grid(*shape)
    rng = np.random.default_rng(1)
    phi = field(shape, kind)
    ucn = cases.F(rng.standard_normal((3,) + shape) * (rng.random((3,) + shape) > 0.1))
    aj = cases.F(1.0 + rng.random(shape))
    mask = np.asfortranarray(rng.integers(-1, 2, shape), dtype=np.int32)
    p = O.make_params(delti_lsm=0.01, btype_lsm=(1, 2, 0, 1, 1, 0), BigPhi=0.3)
    with np.errstate(all="ignore"):
        for m in (None, mask):
            dm = None if m is None else dev(m)
            assert same(host(ls.calc_rh_ad_weno3(G(g), dev(phi), dev(ucn), dm)),
                        oracle.calc_rh_ad_weno3(g, phi, ucn, m))
            assert same(host(ls.ad_rktvd3(G(g), P(p), dev(phi), dev(ucn), dev(aj), dm)),
                        oracle.ad_rktvd3(g, p, phi, ucn, aj, m))


@pytest.mark.parametrize("kind", ["plain", "extreme"])
@pytest.mark.parametrize("spacing", [(1.0, 1.0, 1.0), (0.5, 1.0, 3.0)])
def test_godunov_bit_exact(ls, oracle, spacing, kind):
    shape = (34, 9, 11)
    g = O.make_grid(*shape)
    g.dc, g.de, g.dz = spacing
    rng = np.random.default_rng(2)
    d = field(shape, kind, 3)
    met = [cases.F(rng.standard_normal((3,) + shape) * (rng.random((3,) + shape) > 0.3)) for _ in range(3)]
    sign = cases.F(rng.choice([-1.0, 1.0, 0.0, 0.37, -1e-9, 1e-310, np.nan], shape))
    with np.errstate(all="ignore"):
        assert same(host(ls.calc_rh_rn(G(g), dev(d), dev(sign), *map(dev, met))), oracle.calc_rh_rn(g, d, sign, *met))
        _, ng = ls.calc_sign_ini(G(g), dev(d), *map(dev, met), 0.1)
        assert same(host(ng), oracle.calc_sign_ini(g, d, *met, 0.1)[1])


@pytest.mark.parametrize("kind", ["plain", "extreme"])
@pytest.mark.parametrize("spacing", [(1.0, 1.0, 1.0), (0.5, 1.0, 3.0)])
def test_eno_norm_bit_exact(ls, oracle, spacing, kind):
    shape = (35, 10, 9)
    g = O.make_grid(*shape)
    g.dc, g.de, g.dz = spacing
    rng = np.random.default_rng(4)
    d, zero = field(shape, kind, 5), field(shape, kind, 6)
    met = [cases.F(rng.standard_normal((3,) + shape) * (rng.random((3,) + shape) > 0.3)) for _ in range(3)]
    for order in (1, 3):
        p = O.make_params(OrderReinitialisationBoundaries=order)
        with np.errstate(all="ignore"):
            assert same(host(ls.calc_normgrad_d(G(g), P(p), dev(d), dev(zero), *map(dev, met))),
                        oracle.calc_normgrad_d(g, p, d, zero, *met))


@pytest.mark.parametrize("tol,want", [(1e-5, 5), (0.1, 4), (10.0, 0)])
def test_live_reinitialisation_stops_where_the_oracle_does(ls, oracle, tol, want):
    """The device-side convergence test: all iterations, some, none (1e-13
    normwise where CUDA's sin and cos enter, as in the other tests)."""
    g, x, y, z, _, _ = cases.curvilinear(34, 11, 10, seed=2)
    csi, eta, zet, _ = oracle.mg_metrics(g, x, y, z)
    phi = cases.F(1.07 * (z - 0.45) + 0.01 * np.sin(3 * x))
    p = O.make_params(epslsm=0.1, RNitermax=5, RNtimestep=0.04, epsReinitialisation=tol)
    ref, it = oracle.reinitialisation_test2(g, p, phi, csi, eta, zet)
    got, n = ls.reinitialisation_test2(G(g), P(p), *map(dev, (phi, csi, eta, zet)))
    assert n == it == want and cases.relerr(host(got), ref) <= 1e-13
