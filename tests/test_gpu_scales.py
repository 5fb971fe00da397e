"""Unions of spheres on grids of any size: the passes that prune them bound distances in Float32, which must
not lose a sphere where Float32's squares vanish or overflow. The same body scaled to every extent, bit for
bit against the oracle, which evaluates whole tapes."""
import math

import numpy as np
import pytest
import torch

from helpers import FIELDS, bits, cc, po

pytestmark = pytest.mark.gpu

PREC = [("f64", 1), ("f32", 0), ("mixed", 2)]
# at Float64 the last on each side are beyond the range whose squares are normal; at Float32 those beyond
# 1e-14 and 1e18 are
EXTENTS = [1e-30, 1e-22, 1e-18, 1e-13, 1.0, 1e17, 4e19, 1e22, 1e30]
EXTENTS_F64 = [1e-160, 1e-90, 1e90, 1e160]
N = (40, 21, 18)


def _body(extent, smooth):
    rng = np.random.default_rng(7)
    s = [cc.Sphere(tuple(extent * rng.uniform(0.0, 0.9, 3)), extent * float(rng.uniform(0.03, 0.12))) for _ in range(48)]
    if smooth:
        return cc.SmoothUnion(*s, k=0.03 * extent)
    return cc.Union(*s, cc.Sphere((0.3 * extent, 0.2 * extent, 0.2 * extent), 0.2 * extent))


def _grid(extent):
    return cc.CartesianGrid((-0.05 * extent, 0.0, 0.01 * extent), N, (extent / max(N),) * 3)


def _extents(prec):
    return EXTENTS + (EXTENTS_F64 if prec == 1 else [])


def _same(dev, ref, label):
    """Equal bits, any NaN for a NaN (a device's and a host's differ in sign)."""
    a, b = np.asarray(dev).reshape(-1), np.asarray(ref).reshape(-1)
    if a.dtype.kind == "f":
        bad = np.flatnonzero((bits(a) != bits(b)) & ~(np.isnan(a) & np.isnan(b)))
    else:
        bad = np.flatnonzero(a != b)
    assert bad.size == 0, f"{label}: {bad.size} differ, first at {bad[0]}: {a[bad[0]]} for {b[bad[0]]}"


def _cache(g, method, prec):
    return cc.allocate_cache(g, method, dtype=torch.float64 if prec == 1 else torch.float32,
                             precision="mixed" if prec == 2 else "plain")


@pytest.mark.parametrize("smooth", [False, True])
@pytest.mark.parametrize("pname,prec", PREC)
def test_marching_cubes_at_every_scale(pname, prec, smooth):
    for L in _extents(prec):
        g, tape = _grid(L), cc.flatten(_body(L, smooth), 3)
        c = cc.update_cache(_cache(g, cc.MarchingCubesCutCell(), prec), tape, g)
        phi, ref = po.mc_update(g, tape, cc.mc_tables.project_table(), prec)
        _same(c.phi.cpu().numpy(), phi, f"phi {L}")
        dev = c.to_host()
        for f in FIELDS:
            _same(dev[f], ref[f], f"{f} {L}")


@pytest.mark.parametrize("smooth", [False, True])
@pytest.mark.parametrize("pname,prec", PREC)
def test_plic_at_every_scale(pname, prec, smooth):
    T = np.float64 if prec == 1 else np.float32
    for L in _extents(prec):
        g, tape = _grid(L), cc.flatten(_body(L, smooth), 3)
        c = cc.update_cache(_cache(g, cc.PLICCutCell(), prec), tape, g)
        ref, rn, ri, rv = po.plic_update(g, tape, prec)
        _same(c.normals.cpu().numpy(), rn, f"normals {L}")
        _same(c.intercepts.cpu().numpy(), ri, f"intercepts {L}")
        _same(c.is_valid.cpu().numpy(), rv, f"is_valid {L}")
        dev = c.to_host()
        fields = ["kind", "volume_fraction"]
        with np.errstate(over="ignore", under="ignore"):
            area = T(g.d[0]) * T(g.d[0])
        if np.finfo(T).tiny < area < np.inf:  # a face fraction is an area over the face's
            fields.append("face_fraction")
        # of a plane with infinite components (where squared distances vanish) the clip's quotient is not a
        # number, but the device's clip returns before it
        plane = np.isfinite(rn).all(axis=1) & np.isfinite(ri)
        for f in fields:
            _same(dev[f][plane], ref[f][plane], f"{f} {L}")


@pytest.mark.parametrize("smooth", [False, True])
@pytest.mark.parametrize("pname,prec", PREC)
def test_calc_volume_at_every_scale(pname, prec, smooth):
    """The compensated sum of n fractions is within 2 u of exact, plus n u^2; times the cell's volume it
    rounds once more, and so does this test's division."""
    T = np.float64 if prec == 1 else np.float32
    for L in _extents(prec):
        g, tape = _grid(L), cc.flatten(_body(L, smooth), 3)
        total = math.fsum(po.plic_fractions(g, tape, prec).tolist())
        with np.errstate(over="ignore", under="ignore"):
            pd = float(T(g.d[0]) * T(g.d[0]) * T(g.d[0]))
        v = cc.calc_volume(tape, g, dtype=torch.float64 if prec == 1 else torch.float32,
                           precision="mixed" if prec == 2 else "plain")
        if 0.0 < pd < math.inf and pd >= np.finfo(np.float64).tiny:
            assert abs(v / pd - total) <= 6 * 2.0 ** -53 * max(1.0, total), (L, v / pd, total)
        else:
            want = total * pd
            assert v == want or (math.isnan(v) and math.isnan(want)), (L, v, want)


@pytest.mark.parametrize("pname,prec", PREC)
def test_a_far_sphere_of_another_scale(pname, prec):
    """A sphere so large and far that Float32 cannot square its distance, united with small ones."""
    g = _grid(1.0)
    for far in (1e12, 1e20):
        tape = cc.flatten(cc.Union(cc.Sphere((far, 0.3, 0.2), far), *_body(1.0, False).children), 3)
        phi, _ = po.mc_update(g, tape, cc.mc_tables.project_table(), prec)
        c = cc.update_cache(_cache(g, cc.MarchingCubesCutCell(), prec), tape, g)
        _same(c.phi.cpu().numpy(), phi, f"phi {far}")
        p = cc.update_cache(_cache(g, cc.PLICCutCell(), prec), tape, g)
        ref, rn, ri, rv = po.plic_update(g, tape, prec)
        _same(p.normals.cpu().numpy(), rn, f"normals {far}")
        _same(p.to_host()["volume_fraction"], ref["volume_fraction"], f"volume_fraction {far}")
        total = math.fsum(po.plic_fractions(g, tape, prec).tolist())
        T = np.float64 if prec == 1 else np.float32
        pd = float(T(g.d[0]) * T(g.d[0]) * T(g.d[0]))
        v = cc.calc_volume(tape, g, dtype=torch.float64 if prec == 1 else torch.float32,
                           precision="mixed" if prec == 2 else "plain")
        assert abs(v / pd - total) <= 6 * 2.0 ** -53 * max(1.0, total), (far, v / pd, total)
