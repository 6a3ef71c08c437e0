"""The FP64 gradient norms where tiny factors cancel to much less: the products
of metrics and differences are about 2^-470 and leave 2^-510 of each other, so
the square is a subnormal number that counts.  Bit for bit as the oracle."""
import numpy as np
import pytest

import cases
import oracle as O
from test_gpu_parity import G, P, dev, host

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("em,ed", [(-235, -235), (-201, -239), (-199, -199), (-240, -240), (-120, -120)])
def test_cancelled_products_bit_exact(ls, oracle, em, ed):
    shape = (7, 6, 8)
    g = O.make_grid(*shape)
    i, j, _ = np.meshgrid(*(np.arange(n) for n in shape), indexing="ij")
    f = cases.F(2.0 ** ed * ((1 + 2.0 ** -40) * i - j + 64.0))
    one = np.zeros((3,) + shape)
    one[0] = 2.0 ** em
    met = [cases.F(one), cases.F(one), cases.F(np.zeros((3,) + shape))]
    sign = cases.F(np.where(i % 2, 1.0, -1.0))
    for d in (f, cases.F(-f)):
        _, ng = ls.calc_sign_ini(G(g), dev(d), *map(dev, met), 0.1)
        want = oracle.calc_sign_ini(g, d, *met, 0.1)[1]
        assert want[3, 3, 3] == 2.0 ** (em + ed - 40)
        assert np.array_equal(host(ng), want)
        p = O.make_params(OrderReinitialisationBoundaries=1)
        assert np.array_equal(host(ls.calc_normgrad_d(G(g), P(p), dev(d), dev(d), *map(dev, met))),
                              oracle.calc_normgrad_d(g, p, d, d, *met))
