"""Columns that start anywhere: a caller's arrays need only their element's alignment, so every wide store has
a narrow form. Each column is a slice one element into its buffer; results equal the aligned cache's bit
for bit, and the element before each column stays untouched."""
import importlib

import numpy as np
import pytest
import torch

from helpers import FIELDS, bits, cc

pytestmark = pytest.mark.gpu
B = importlib.import_module("cutcell_b200.batch")

PRECISIONS = [(torch.float32, "plain"), (torch.float64, "plain"), (torch.float32, "mixed")]
EXTRA = ("normals", "intercepts", "is_valid", "phi")


def _shift(cache):
    """Every column of the cache moved one element into a larger buffer."""
    guards = []
    for owner, names in ((cache.cells, FIELDS), (cache, EXTRA)):
        for f in names:
            old = getattr(owner, f, None)
            if old is None:
                continue
            buf = torch.full((old.numel() + 1,), 77, dtype=old.dtype, device=old.device)
            new = buf[1:].view(old.shape)
            new.copy_(old)
            setattr(owner, f, new)
            guards.append(buf)
    return guards


def _same(a, b, names):
    for f in names:
        x, y = (getattr(c.cells, f, None) if f in FIELDS else getattr(c, f, None) for c in (a, b))
        if x is not None:
            assert np.array_equal(bits(x.cpu().numpy()), bits(y.cpu().numpy())), f


@pytest.mark.parametrize("dtype,precision", PRECISIONS)
@pytest.mark.parametrize("method,n", [("ms", (70, 33)), ("plic", (40, 19, 21)), ("mc", (48, 17, 35)), ("mc", (33, 9, 5))])
def test_update_into_unaligned_columns(method, n, dtype, precision):
    m = {"ms": cc.MarchingSquaresCutCell, "plic": cc.PLICCutCell, "mc": cc.MarchingCubesCutCell}[method]()
    h = 1.0 / max(n)
    g = cc.CartesianGrid((-0.03,) * len(n), n, (h,) * len(n))
    body = cc.Circle((0.4, 0.2), 0.17) if method == "ms" else cc.workloads.sphere_cloud(5, 40)
    want = cc.update_cache(cc.allocate_cache(g, m, dtype=dtype, precision=precision), body, g)
    got = cc.allocate_cache(g, m, dtype=dtype, precision=precision)
    guards = _shift(got)
    cc.update_cache(got, body, g)
    _same(got, want, FIELDS + EXTRA)
    assert all(int(b[0]) == 77 for b in guards)
    if method == "ms":
        batch = B.Batch(dtype=dtype, precision=precision)
        batch.add(got, body, g)
        for f in FIELDS:
            getattr(got.cells, f).zero_()
        batch.run()
        _same(got, want, FIELDS + ("phi",))
        assert all(int(b[0]) == 77 for b in guards)
