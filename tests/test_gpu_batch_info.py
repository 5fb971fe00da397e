"""total_tiles counts the configuration's own tiles and leaf chunks, however the kernel takes them."""
import pytest
import torch

from helpers import cc

pytestmark = pytest.mark.gpu
B = __import__("cutcell_b200.batch", fromlist=["batch"])

GRIDS = [(1, 1), (33, 17), (100, 37), (257, 129)]


def _tiles(leaves, tile_x, tile_y, threads):
    return sum(-(-a // tile_x) * -(-b // tile_y) for a, b in GRIDS) + -(-leaves // threads)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_total_tiles_are_the_configurations(dtype):
    b = B.Batch(dtype=dtype)
    body = cc.Circle((0.1, -0.05), 0.6)
    tree, _, _ = cc.star_curve_tree(3, 3, 8)
    for d in [cc.CartesianGrid((-1.0, -1.0), n, (2.0 / n[0], 2.0 / n[1])) for n in GRIDS] + [tree]:
        b.add(cc.allocate_cache(d, cc.MarchingSquaresCutCell(), dtype=dtype), body, d)
    assert b.total_tiles() == -1
    for tx, ty, threads in [(32, 8, 256), (64, 8, 128), (128, 2, 256), (96, 3, 64), (16, 16, 128)]:
        b.configure(tile_x=tx, tile_y=ty, threads=threads, band_percent=0)
        assert b.total_tiles() == -1
        b.run()
        want = _tiles(tree.nleaves, tx, ty, threads)
        assert b.total_tiles() == want, (tx, ty, threads)
        b.configure(band_percent=50)  # the same tiles
        assert b.total_tiles() == want
        b.run()
        assert b.total_tiles() == want
