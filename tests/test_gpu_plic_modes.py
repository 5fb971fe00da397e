"""The 3D PLIC update, one case per way the fit evaluates a body (hard and smooth unions of spheres
pruned per warp, hard combinators whose gradient is one primitive's, smooth minima on duals), at
sizes around the row of 32 cells, the 8 rows of a CTA and the layers of a warp, bit for bit against
the oracle in every precision."""
import math

import numpy as np
import pytest
import torch

from helpers import assert_cells_bitwise, bits, cc, po

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (33, 9, 5), (31, 17, 131), (64, 8, 64), (97, 3, 33)]
PREC = [("f64", 1), ("f32", 0), ("mixed", 2)]


def _grid(n):
    return cc.CartesianGrid((-0.07, 0.03, -0.02), n, (1.0 / max(n),) * 3)


def _spheres(k, smooth=None):
    rng = np.random.default_rng(40 + k)
    s = [cc.Sphere(tuple(rng.uniform(0.0, 0.9, 3)), float(rng.uniform(0.03, 0.12))) for _ in range(k)]
    return cc.SmoothUnion(*s, k=smooth) if smooth else cc.Union(*s)


def _mixed(k):
    """Primitives of every kind that evaluates alike on host and device, some far from the grid."""
    rng = np.random.default_rng(k)
    out = []
    for i in range(k):
        c = tuple(rng.uniform(-0.5, 1.5, 3))
        if i % 4 == 0:
            out.append(cc.Box(c, tuple(rng.uniform(0.02, 0.2, 3))))
        elif i % 4 == 1:
            out.append(cc.Torus(c, 0.2, 0.05, cc.quat_to_matrix(rng.normal(size=4)) * rng.uniform(0.5, 2.0)))
        elif i % 4 == 2:
            out.append(cc.Plane((c[0], c[1], -0.3), (0.1 * c[0], 0.2, 1.5)))
        else:
            out.append(cc.Sphere(c, float(rng.uniform(0.02, 0.15))))
    return out + [cc.Const(0.4)]


def _bodies():
    sphere, box = cc.Sphere((0.3, 0.25, 0.4), 0.22), cc.Box((0.45, 0.35, 0.5), (0.2, 0.12, 0.3))
    torus = cc.Torus((0.5, 0.4, 0.3), 0.25, 0.08, cc.quat_to_matrix((0.8, 0.1, -0.5, 0.3)))
    return {
        "spheres_2": _spheres(2), "spheres_33": _spheres(33), "spheres_200": _spheres(200),
        "smooth_5": _spheres(5, 0.08), "smooth_70": _spheres(70, 0.05),
        "union": cc.Union(sphere, box, torus),
        "union_long": cc.Union(*_mixed(45)),
        "one_sphere": sphere, "plane": cc.Plane((0.4, 0.3, 0.5), (0.6, -0.64, 0.48)),
        "select": cc.Subtraction(cc.Union(sphere, box, torus), cc.Intersection(cc.Sphere((0.5, 0.4, 0.5), 0.15), box)),
        "negated": cc.Negate(cc.Union(cc.Negate(cc.Intersection(sphere, torus)), box)),
        "smooth_mixed": cc.SmoothUnion(box, cc.Subtraction(sphere, torus), torus, k=0.06),
        "nothing": cc.EmptyGeo(1.0),
    }


@pytest.mark.parametrize("name", sorted(_bodies()))
@pytest.mark.parametrize("pname,prec", PREC)
def test_plic_update_bitwise(name, pname, prec):
    dtype = torch.float64 if prec == 1 else torch.float32
    for n in SHAPES:
        g = _grid(n)
        tape = cc.flatten(_bodies()[name], 3)
        c = cc.allocate_cache(g, cc.PLICCutCell(), dtype=dtype, precision="mixed" if prec == 2 else "plain")
        c.cells.face_fraction.fill_(7.0)
        cc.update_cache(c, tape, g)
        ref, rn, ri, rv = po.plic_update(g, tape, prec)
        assert_cells_bitwise(c.to_host(), ref, fields=("kind", "volume_fraction", "face_fraction"), label=f"{name} {n}")
        assert np.array_equal(bits(c.normals.cpu().numpy()), bits(rn)), n
        assert np.array_equal(bits(c.intercepts.cpu().numpy()), bits(ri)), n
        assert np.array_equal(c.is_valid.cpu().numpy(), rv), n


VOLUME_BODIES = dict(_bodies(), inside=cc.Const(-1.0), zero=cc.Const(0.0),
                     steep=cc.Plane((0.4, 0.3, 0.5), (3.0, -4.0, 12.0)),
                     stretched=cc.Torus((0.5, 0.4, 0.3), 0.25, 0.08, 2.5 * np.eye(3)),
                     waves=cc.Union(cc.Trig(0.4, (9.0, 7.0, 5.0), 0.05), cc.Sphere((0.1, 0.2, 0.2), 0.1)))


@pytest.mark.parametrize("name", sorted(VOLUME_BODIES))
@pytest.mark.parametrize("pname,prec", PREC)
def test_calc_volume_is_the_sum_of_the_cell_fractions(name, pname, prec):
    """Boxes settled by the body's bounds count as their cells do: the compensated sum of the oracle's
    fractions, at sizes around the box of 8 x 4 x 8 cells and the 32 boxes a warp looks at, and on a
    grid far from the origin, where rounding is a cell's size at Float32. A sum of n fractions in
    [0, 1], compensated in Float64, is within 2 u of exact, plus n u^2; the product with the cell's
    volume rounds twice more."""
    dtype = torch.float64 if prec == 1 else torch.float32
    T = np.float64 if prec == 1 else np.float32
    tape = cc.flatten(VOLUME_BODIES[name], 3)
    for n, x0, h in [((1, 1, 1), 0.0, 0.7), ((9, 5, 17), -0.1, 0.08), ((70, 33, 41), -0.05, 1.0 / 64),
                     ((40, 40, 40), 0.0, 1.0 / 40), ((33, 9, 20), 2.0 ** 17, 0.01)]:
        g = cc.CartesianGrid((x0, -0.03, 0.02), n, (h,) * 3)
        frac = po.plic_fractions(g, tape, prec)
        if name == "waves":  # sin differs from the host's by an ulp: a fraction moves by about u / h
            tol = 64 * np.finfo(T).eps / h * max(n) * len(frac) ** (2 / 3)
        else:
            tol = 4 * 2.0 ** -53 * max(1.0, math.fsum(frac.tolist()))
        pd = float(T(h) * T(h) * T(h))
        v = cc.calc_volume(tape, g, dtype=dtype, precision="mixed" if prec == 2 else "plain")
        assert abs(v / pd - math.fsum(frac.tolist())) <= tol, (name, n)


@pytest.mark.parametrize("name", ["union", "union_long", "spheres_33", "spheres_200", "smooth_70"])
@pytest.mark.parametrize("pname,prec", PREC)
def test_marching_cubes_of_pruned_unions_bitwise(name, pname, prec):
    """The fill evaluates a pencil's nodes with the ops it keeps: phi and every column as the oracle's whole
    tape gives them, at sizes around the pencil and far from the origin."""
    dtype = torch.float64 if prec == 1 else torch.float32
    tape = cc.flatten(_bodies()[name], 3)
    for n, x0 in [((1, 1, 1), 0.0), ((33, 9, 5), -0.07), ((31, 17, 66), 0.0), ((64, 24, 35), -0.02), ((20, 20, 20), 300.0)]:
        g = cc.CartesianGrid((x0, 0.03, -0.02), n, (1.0 / max(n),) * 3)
        c = cc.allocate_cache(g, cc.MarchingCubesCutCell(), dtype=dtype, precision="mixed" if prec == 2 else "plain")
        cc.update_cache(c, tape, g)
        phi, ref = po.mc_update(g, tape, cc.mc_tables.project_table(), prec)
        assert np.array_equal(bits(c.phi.cpu().numpy()), bits(phi)), n
        assert_cells_bitwise(c.to_host(), ref, label=f"{name} {n}")
