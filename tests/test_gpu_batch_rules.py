"""Batches taken a CTA per tile and a warp per strip: both routes of the rule, bit for bit against the oracle, in
every precision."""
import numpy as np
import pytest
import torch

from helpers import assert_cells_bitwise, bits, cc, po

pytestmark = pytest.mark.gpu
B = __import__("cutcell_b200.batch", fromlist=["batch"])
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


@pytest.mark.parametrize("pname,prec", PREC)
@pytest.mark.parametrize("sizes,k", [([(50, 41)] * 4, 9), ([(700, 333)] * 7 + [(5, 900), (33, 700)], 1), ([(701, 699)] * 3, 9)])
def test_batch_by_every_route(sizes, k, pname, prec):
    """Few strips (a CTA per tile) and many (a warp per strip), the launch shape changed in between."""
    b, items = B.Batch(dtype=torch.float64 if prec == 1 else torch.float32, precision="mixed" if prec == 2 else "plain"), []
    for i, n in enumerate(sizes):
        g, body = _grid(n), _body(k)
        items.append((g, cc.flatten(body, 2), _cache(g, prec)))
        b.add(items[-1][2], body, g)
    want = {}
    for shape in (dict(tile_x=32, tile_y=8, threads=256, ctas_per_sm=4, chunk=2), dict(ctas_per_sm=1, chunk=1),
                  dict(tile_x=64, tile_y=4, threads=128, ctas_per_sm=8, chunk=1), dict(chunk=4)):
        b.configure(band_percent=0, **shape)
        for _, _, c in items:
            c.phi.zero_()
            c.cells.volume_fraction.fill_(7.0)
            c.cells.kind.fill_(9)
        b.run()
        for g, tape, c in items:
            if g.n not in want:
                want[g.n] = po.ms_update(g, tape, prec)
            phi, ref = want[g.n]
            assert np.array_equal(bits(c.phi.cpu().numpy()), bits(phi)), (g.n, shape)
            assert_cells_bitwise(c.to_host(), ref, label=f"{g.n} {shape}")
