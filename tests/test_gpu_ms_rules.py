"""Marching squares by strips and by two passes, each route of the rules on sizes, tapes and
shapes, bit for bit against the oracle, in every precision."""
import numpy as np
import pytest
import torch

from helpers import assert_cells_bitwise, bits, cc, po

pytestmark = pytest.mark.gpu
PREC = [("f64", 1), ("f32", 0), ("mixed", 2)]


def _body(k):
    rng = np.random.default_rng(k)
    c = [cc.Circle(tuple(rng.uniform(0, 1, 2)), float(rng.uniform(0.02, 0.2))) for _ in range(k)]
    return c[0] if k == 1 else cc.Union(*c)


def _cache(g, prec):
    return cc.allocate_cache(g, cc.MarchingSquaresCutCell(), dtype=torch.float64 if prec == 1 else torch.float32,
                             precision="mixed" if prec == 2 else "plain")


def _grid(n):
    return cc.CartesianGrid((-0.02, 0.01), n, (1.0 / max(n),) * 2)


# a narrow grid, a wider one, few and many cells of one circle; unions that take strips at one precision,
# both or neither
CASES = [((3, 700), 1), ((33, 3001), 1), ((41, 3001), 1), ((257, 255), 1), ((257, 257), 1), ((100, 33), 8),
         ((1003, 1001), 8), ((1003, 1001), 20), ((1003, 1001), 60)]


@pytest.mark.parametrize("pname,prec", PREC)
@pytest.mark.parametrize("n,k", CASES)
def test_update_by_every_route(n, k, pname, prec):
    g, tape = _grid(n), cc.flatten(_body(k), 2)
    c = cc.update_cache(_cache(g, prec), tape, g)
    phi, ref = po.ms_update(g, tape, prec)
    assert np.array_equal(bits(c.phi.cpu().numpy()), bits(phi))
    assert_cells_bitwise(c.to_host(), ref, label=f"{n} {k}")


@pytest.mark.parametrize("pname,prec", PREC)
@pytest.mark.parametrize("n", [(33, 9), (2500, 2401)])
def test_given_values_by_every_route(n, pname, prec):
    g = _grid(n)
    phi, ref = po.ms_update(g, cc.flatten(_body(5), 2), prec)
    c = cc.update_cache(_cache(g, prec), cc.NodalField(torch.from_numpy(phi)), g)
    assert_cells_bitwise(c.to_host(), ref, label=str(n))
