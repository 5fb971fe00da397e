"""Marching cubes over grids of many tiles and few layers: with the GPU full the fill takes its deepest
pencils, whose depth depends on the precision and on whether every column leaves by TMA (x a multiple of
16). Layer counts one below, at and one above the depths and their multiples; every column bit for bit
against the oracle."""
import numpy as np
import pytest
import torch

from helpers import assert_cells_bitwise, bits, cc, po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,prec", [((512, 256, 18), 0), ((512, 256, 19), 0), ((512, 256, 39), 2),
                                    ((500, 264, 15), 0), ((503, 260, 16), 2), ((501, 257, 31), 0),
                                    ((256, 264, 10), 1), ((256, 264, 11), 1), ((256, 260, 23), 1),
                                    ((252, 264, 31), 1), ((251, 263, 32), 1), ((250, 257, 33), 1)])
def test_update_matches_oracle_at_the_deepest_pencils(n, prec):
    h = 2.0 / max(n)
    g = cc.CartesianGrid((-1.0, -0.5, -0.5 * h * n[2]), n, (h, h, h))
    body = cc.workloads.csg_body(0)
    table = cc.mc_tables.project_table()
    cache = cc.allocate_cache(g, cc.MarchingCubesCutCell(), dtype=torch.float64 if prec == 1 else torch.float32,
                              precision="mixed" if prec == 2 else "plain")
    cc.update_cache(cache, body, g)
    phi, ref = po.mc_update(g, cc.geometry.as_tape(body, 3), table, prec)
    assert np.array_equal(bits(cache.phi.cpu().numpy()), bits(phi))
    assert_cells_bitwise(cache.to_host(), ref, label=f"{n}")
    assert int((cache.to_host()["kind"] == 2).sum()) > 1000
