"""Cut cells at the edges of the construction's arithmetic, against the oracle: every face with
opposite corners open, corner values from subnormal to huge, infinite and NaN corners, and cells so
small that a third of a coordinate leaves the range of the division by a constant. Equal bit for bit;
a NaN (whose payload differs between CPU and GPU) equals a NaN."""
import numpy as np
import pytest
import torch

from helpers import FIELDS, bits, cc, po

pytestmark = pytest.mark.gpu


def _values(kind, n, rng, T):
    v = rng.uniform(-1.0, 1.0, n)
    if kind == "checker":  # alternating signs: all faces ambiguous
        z, y, x = np.meshgrid(*[np.arange(k) for k in (10, 9, 12)], indexing="ij")
        v = np.abs(v).reshape(10, 9, 12) * np.where((x + y + z) % 2 == 0, 1.0, -1.0)
    elif kind == "wide":
        v = v * 10.0 ** rng.uniform(-44 if T == np.float32 else -320, 37, n)
    elif kind == "zeros":
        v = np.where(rng.random(n) < 0.4, 0.0, v)
    elif kind == "not_finite":
        bad = rng.random(n)
        v = np.where(bad < 0.04, np.nan, np.where(bad < 0.07, np.inf, np.where(bad < 0.1, -np.inf, v)))
    return np.ascontiguousarray(np.asarray(v, np.float64).reshape(-1).astype(T))


@pytest.mark.parametrize("kind", ["random", "checker", "wide", "zeros", "not_finite"])
@pytest.mark.parametrize("h", [(1.0, 0.5, 2.0), (2.0 ** -98, 2.0 ** -100, 2.0 ** -97)])
@pytest.mark.parametrize("pname,prec", [("f64", 1), ("f32", 0), ("mixed", 2)])
def test_cut_cells_against_the_oracle(kind, h, pname, prec):
    T = np.float64 if prec == 1 else np.float32
    if prec == 1 and h[0] < 1e-20:
        h = tuple(k * 2.0 ** -810 for k in h)
    g = cc.CartesianGrid((0.0, 0.0, 0.0), (11, 8, 9), h)
    with np.errstate(over="ignore"):
        vals = _values(kind, g.nnode, np.random.default_rng(7), T)
    dtype = torch.float64 if prec == 1 else torch.float32
    c = cc.allocate_cache(g, cc.MarchingCubesCutCell(), dtype=dtype, precision="mixed" if prec == 2 else "plain")
    cc.update_cache(c, cc.NodalField(torch.as_tensor(vals)), g)
    with np.errstate(all="ignore"):
        ref = po.mc_cells_from_phi(g, vals, cc.mc_tables.project_table(), prec)
    host = c.to_host()
    assert int((host["kind"] == 2).sum()) > 300
    for f in FIELDS:
        a = np.asarray(host[f]).reshape(len(ref[f]), -1)
        b = np.asarray(ref[f]).reshape(len(ref[f]), -1)
        same = bits(a) == bits(b)
        if a.dtype.kind == "f":
            same |= np.isnan(a) & np.isnan(b)
        bad = np.flatnonzero(~same.all(axis=1))
        assert bad.size == 0, (f, bad.size, a[bad[0]], b[bad[0]])
