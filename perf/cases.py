"""What this framework is timed on: cut-cell updates, surfaces and volumes through its public entry points.

A case is a dict of plain values; ``path`` says which entry point it takes:

* ``mc``       ``update_cache`` of a marching-cubes cache from a body (with ``report``: and ``cut_cell_report``)
* ``field``    ``update_cache`` of a marching-cubes cache from nodal values that a solver holds (``NodalField``)
* ``learned``  ``update_cache_learned``: the update with the network's volume-fraction correction
* ``plic``     ``update_cache`` of a PLIC cache
* ``volume``   ``calc_volume`` of a body
* ``batch``    ``Batch.run``: many marching-squares updates of one moving body at once
* ``ms``       ``update_cache`` of one marching-squares grid
* ``tree``     ``update_cache`` of the leaves of a quadtree
* ``mesh``     ``generate_mesh`` of a marching-cubes cache
* ``plic_mesh``  ``generate_mesh`` of a PLIC cache

Grids are ``n0 x n1 x n2`` cells; ``dtype`` is the cache's element type and ``mixed`` Float32 with
Float64 islands. Bodies: ``csg`` (sphere + box + rotated torus over [-1,1]^3), ``spheres`` (a cloud
of 64 over the unit cube) and ``blob`` (a smooth union of a few spheres), all made from the seed.

``exact`` gives, in 64 bits and without the framework, the fields that follow from the body alone:
the nodal values, everything of the 2D and PLIC cells, and the marching-cubes cells' face fractions
and face centroids. A marching-cubes cell's volume fraction, centroid and interface centroid, and a
mesh's vertices, also depend on which triangles the caller's tiling table takes, and have none.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

from __graft_entry__ import load_package

cc = load_package()

F32, F64 = "float32", "float64"


# ---------------------------------------------------------------------------------------------
# the cases

def _case(path, n, dtype=F32, **kw):
    c = {"path": path, "dtype": dtype, "mixed": False}
    for a, v in enumerate(n):
        c["n%d" % a] = int(v)
    c.update(kw)
    return c


def listed():
    return [
        # the headline: a moving body on a fine grid, all columns rewritten at every time step
        _case("mc", (512, 512, 512), body="csg", report=False, name="mc_512_f32"),
        # the default element type at an ordinary size, with the report a driver prints per step
        _case("mc", (256, 256, 256), F64, body="csg", report=True, name="mc_256_f64_report"),
        # a coarse design sweep or a unit test's grid: the smallest 3D call
        _case("mc", (64, 64, 64), body="csg", report=False, name="mc_64_f32"),
        # a channel grid that fits no tile, in mixed precision
        _case("mc", (301, 187, 130), body="csg", report=False, mixed=True, name="mc_301x187x130_mixed"),
        # a flow solver's own level set, many cells cut, some faces ambiguous
        _case("field", (192, 160, 129), F64, name="field_192x160x129_f64"),
        # the corrected update in the resolution range it was trained for
        _case("learned", (256, 256, 256), body="blob", name="learned_256_f32"),
        # a droplet or particle cloud in a volume-of-fluid code, at production resolution
        _case("plic", (512, 512, 512), body="spheres", name="plic_512_f32"),
        # a machined part on a small odd grid, in the default element type
        _case("plic", (150, 97, 131), F64, body="csg", name="plic_150x97x131_f64"),
        # the conservation check of a volume-of-fluid run: one number per step
        _case("volume", (256, 256, 256), F64, body="spheres", name="volume_256_f64"),
        # a parameter study of a translating cylinder: one launch over grids of many sizes
        _case("batch", (64, 1024), updates=96, tuned=True, name="batch_96_f32"),
        # one 2D update at the size of the reference's own test, where latency counts
        _case("ms", (200, 200), F64, name="ms_200_f64"),
        # the body's surface for output or for a mesh-based solver
        _case("mesh", (384, 384, 384), body="csg", name="mesh_384_f32"),
    ]


def _size(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _size3(rng, lo, hi, most):
    """Three extents around one drawn scale, any residue, at most ``most`` cells."""
    while True:
        m = _size(rng, lo, hi)
        n = [max(8, int(m * rng.uniform(0.6, 1.3))) for _ in range(3)]
        if rng.random() < 0.3:
            n = [16 * max(1, round(v / 16)) for v in n]
        if n[0] * n[1] * n[2] <= most:
            return n


def draw(rng):
    path = rng.choice(("mc", "mc", "mc", "field", "learned", "plic", "plic", "volume", "batch", "ms", "tree", "mesh",
                       "plic_mesh"))
    dtype = rng.choice((F32, F32, F64))
    mixed = dtype == F32 and rng.random() < 0.25
    if path in ("mc", "mesh"):
        n = _size3(rng, 24, 420, 60_000_000)
        kw = {"report": rng.random() < 0.3} if path == "mc" else {}
        return _case(path, n, dtype, mixed=mixed, body=rng.choice(("csg", "csg", "spheres", "blob")), **kw)
    if path == "field":
        return _case(path, _size3(rng, 24, 300, 30_000_000), dtype, mixed=mixed)
    if path == "learned":
        return _case(path, _size3(rng, 48, 360, 60_000_000), F32, body="blob")
    if path in ("plic", "plic_mesh"):
        return _case(path, _size3(rng, 24, 420, 60_000_000), dtype, mixed=mixed,
                     body=rng.choice(("csg", "spheres", "spheres", "blob")))
    if path == "volume":
        return _case(path, _size3(rng, 24, 420, 60_000_000), dtype, mixed=mixed, body=rng.choice(("csg", "spheres")))
    if path == "batch":
        lo = _size(rng, 32, 300)
        return _case(path, (lo, rng.randint(2 * lo, 4 * lo)), dtype, mixed=mixed, updates=rng.randint(8, 96),
                     tuned=rng.random() < 0.5)
    if path == "ms":
        return _case(path, (_size(rng, 40, 3000), _size(rng, 40, 3000)), dtype, mixed=mixed)
    return _case("tree", (rng.randint(3, 5), rng.randint(8, 12)), dtype, mixed=mixed)


# ---------------------------------------------------------------------------------------------
# what a program holds before the call

def _dtype(case):
    return torch.float32 if case["dtype"] == F32 else torch.float64


def _precision(case):
    return "mixed" if case["mixed"] else "plain"


def _grid3(case, iso=False):
    n = (case["n0"], case["n1"], case["n2"])
    lo, span = (-1.0, 2.0) if case.get("body", "csg") == "csg" else (0.0, 1.0)
    d = [span / max(n)] * 3 if iso else [span / k for k in n]
    return cc.CartesianGrid((lo, lo, lo), n, d)


def _body3(case, seed):
    W = cc.workloads
    return {"csg": W.csg_body, "spheres": W.sphere_cloud, "blob": W.smooth_blob}[case["body"]](seed)


_WAVES = 6


def _waves(seed):
    """A seeded sum of plane waves with a few crests per axis: a random smooth level set."""
    r = np.random.default_rng(seed)
    k = r.normal(size=(_WAVES, 3))
    k = k / np.linalg.norm(k, axis=1, keepdims=True) * r.uniform(15.0, 45.0, (_WAVES, 1))
    return k, r.uniform(0.0, 2.0 * math.pi, _WAVES), r.uniform(0.5, 1.0, _WAVES) / 20.0


def _field(case, seed, dev):
    k, ph, amp = _waves(seed)
    ax = [torch.arange(case["n%d" % a] + 1, dtype=torch.float64, device=dev) / case["n%d" % a] for a in range(3)]
    v = torch.zeros(len(ax[2]), len(ax[1]), len(ax[0]), dtype=torch.float64, device=dev)
    for q in range(_WAVES):
        v += amp[q] * torch.sin(k[q, 0] * ax[0][None, None, :] + k[q, 1] * ax[1][None, :, None] +
                                k[q, 2] * ax[2][:, None, None] + ph[q])
    return v.reshape(-1).to(_dtype(case))


def _updates(case, seed):
    """Grids of many sizes, the same for every seed, with a circle further along on each (as
    ``workloads.moving_circle_updates``), which starts where the seed says."""
    off = np.random.default_rng(seed).uniform(-0.2, 0.2, 2)
    return [(g, cc.Circle(tuple(np.asarray(b.center) + off), b.radius), n)
            for g, b, n in cc.workloads.moving_circle_updates(case["updates"], 0, case["n0"], case["n1"])]


def _star(case, seed):
    """A quadtree fitted to a star curve, and the curve a little later: grown or shrunk by the seed
    within the band of finest leaves."""
    tree, amp, ph = cc.star_curve_tree(0, case["n0"], case["n1"])
    r0 = 0.5 + np.random.default_rng(seed).uniform(-1.0, 1.0) * 2.0 / 2 ** case["n1"]
    return tree, cc.Star((0.0, 0.0), float(r0), tuple(float(a) for a in amp), tuple(float(p) for p in ph))


def _circle2(case, seed):
    """One grid over [-1,1]^2 with square cells along its longer axis, and a circle on it."""
    r = np.random.default_rng(seed)
    n = (case["n0"], case["n1"])
    h = 2.0 / max(n)
    g = cc.CartesianGrid((-0.5 * h * n[0], -0.5 * h * n[1]), n, (h, h))
    radius = 0.5 * min(n) / max(n)
    c = tuple(r.uniform(-0.1, 0.1, 2) * min(n) / max(n))
    return g, c, float(radius)


FIELDS = ("kind", "ambiguous", "volume_fraction", "centroid", "face_fraction", "face_centroid_local",
          "interface_centroid")
PLIC_FIELDS = ("kind", "volume_fraction", "face_fraction")


def _pool(caches, dtype, dev):
    """One buffer per field for the caches of a study, each cache's columns a slice of it."""
    widths = {"kind": 1, "ambiguous": 1, "volume_fraction": 1, "centroid": 2, "face_fraction": 4,
              "face_centroid_local": 4, "interface_centroid": 2, "phi": 1}
    sizes = [c.cells.kind.numel() for c in caches], [c.phi.numel() for c in caches]
    pool = {}
    for f, w in widths.items():
        each = [-(-v * w // 64) * 64 for v in sizes[f == "phi"]]  # 64 elements: every slice well aligned
        kind = torch.int8 if f == "kind" else torch.uint8 if f == "ambiguous" else dtype
        pool[f] = torch.zeros(sum(each), dtype=kind, device=dev)
        at = 0
        for c, room in zip(caches, each):
            old = c.phi if f == "phi" else getattr(c.cells, f)
            new = pool[f][at:at + old.numel()].view(old.shape)
            new.copy_(old)
            setattr(*((c, "phi") if f == "phi" else (c.cells, f)), new)
            at += room
    return pool


def _vertex_buffers(case, dtype, dev):
    """What a renderer or a coupled solver keeps for the surface: room for more than any of the bodies
    has (a marching-cubes surface shares its vertices, a PLIC surface does not)."""
    n = max(case["n0"], case["n1"], case["n2"])
    nodes, elements = (6 * n * n + 4096, 12 * n * n + 8192) if case["path"] == "mesh" else (40 * n * n, 30 * n * n)
    return {"nodes": torch.zeros(nodes, 3, dtype=dtype, device=dev),
            "elements": torch.zeros(elements, 3, dtype=torch.int32, device=dev),
            "cells": torch.zeros(elements, dtype=torch.int64, device=dev)}


def prepare(case, seed):
    dev, dt, pr, path = torch.device("cuda"), _dtype(case), _precision(case), case["path"]
    s = {"path": path, "report": case.get("report", False)}
    if path in ("mc", "learned", "mesh"):
        s["grid"], s["body"] = _grid3(case), _body3(case, seed)
        s["cache"] = cc.allocate_cache(s["grid"], cc.MarchingCubesCutCell(), dtype=dt, device=dev, precision=pr)
        if path == "learned":
            s["L"] = importlib.import_module("cutcell_b200.learned")
            s["mlp"] = s["L"].pretrained()
        if path == "mesh":
            s["S"] = importlib.import_module("cutcell_b200.surface")
            s["buffers"] = _vertex_buffers(case, dt, dev)
            cc.update_cache(s["cache"], s["body"], s["grid"])
    elif path == "field":
        s["grid"], s["body"] = _grid3(case), cc.NodalField(_field(case, seed, dev))
        s["cache"] = cc.allocate_cache(s["grid"], cc.MarchingCubesCutCell(), dtype=dt, device=dev, precision=pr)
    elif path in ("plic", "plic_mesh"):
        s["grid"], s["body"] = _grid3(case, iso=True), _body3(case, seed)
        s["cache"] = cc.allocate_cache(s["grid"], cc.PLICCutCell(), dtype=dt, device=dev, precision=pr)
        if path == "plic_mesh":
            s["S"] = importlib.import_module("cutcell_b200.surface")
            s["buffers"] = _vertex_buffers(case, dt, dev)
            cc.update_cache(s["cache"], s["body"], s["grid"])
    elif path == "volume":
        s["grid"], s["body"], s["dtype"], s["precision"] = _grid3(case, iso=True), _body3(case, seed), dt, pr
    elif path == "batch":
        ups = _updates(case, seed)
        caches = [cc.allocate_cache(g, cc.MarchingSquaresCutCell(), dtype=dt, device=dev, precision=pr)
                  for g, _, _ in ups]
        s["pool"] = _pool(caches, dt, dev)
        s["batch"] = importlib.import_module("cutcell_b200.batch").Batch(dtype=dt, precision=pr)
        for c, (g, body, _) in zip(caches, ups):
            s["batch"].add(c, body, g)
        if case["tuned"]:
            s["batch"].autotune(reps=1)
    elif path == "ms":
        s["grid"], c, r = _circle2(case, seed)
        s["body"] = cc.Circle(c, r)
        s["cache"] = cc.allocate_cache(s["grid"], cc.MarchingSquaresCutCell(), dtype=dt, device=dev, precision=pr)
    elif path == "tree":
        s["grid"], s["body"] = _star(case, seed)
        s["cache"] = cc.allocate_cache(s["grid"], cc.MarchingSquaresCutCell(), dtype=dt, device=dev, precision=pr)
    else:
        raise ValueError("unknown path %r" % path)
    return s


def run(s):
    path = s["path"]
    if path == "volume":
        return {"volume": cc.calc_volume(s["body"], s["grid"], dtype=s["dtype"], precision=s["precision"])}
    if path == "batch":
        s["batch"].run()
        return s["pool"]
    if path in ("mesh", "plic_mesh"):
        m = s["S"].generate_mesh(s["cache"], s["grid"])
        out = {"n_nodes": m.nodes.shape[0], "n_elements": m.elements.shape[0]}
        for name, buf in s["buffers"].items():
            v = getattr(m, name)
            buf[:v.shape[0]].copy_(v)
            out[name] = buf
        return out
    c, out = s["cache"], {}
    if path == "learned":
        out["fallback"] = s["L"].update_cache_learned(c, s["body"], s["grid"], s["mlp"])
    else:
        cc.update_cache(c, s["body"], s["grid"])
    if s["report"]:
        out["report"] = cc.cut_cell_report(c)
    if path == "plic":
        out.update({f: getattr(c.cells, f) for f in PLIC_FIELDS})
        out.update(normals=c.normals, intercepts=c.intercepts, is_valid=c.is_valid)
    else:
        out.update({f: getattr(c.cells, f) for f in FIELDS})
        out["phi"] = c.phi
    return out


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without

def _leaves(case):
    """Leaves of the quadtree, from its own counting rule: the curve (length about 3.3) crosses a
    few leaves per finest width, over a uniform coarse level."""
    return 4 ** case["n0"] + 3 * 2 ** case["n1"] * 8


def work(case):
    t, path = (4 if case["dtype"] == F32 else 8), case["path"]
    if path == "batch":
        mean2 = (case["n0"] ** 2 + case["n0"] * case["n1"] + case["n1"] ** 2) / 3.0
        cells = case["updates"] * mean2
        return {"bytes": cells * (2 + 14 * t), "flops": 25.0 * cells}
    if path == "tree":
        return {"bytes": _leaves(case) * (2.0 + 17 * t + 12), "flops": 100.0 * _leaves(case)}
    if path == "ms":
        cells = case["n0"] * case["n1"]
        return {"bytes": cells * (2.0 + 14 * t), "flops": 25.0 * cells}
    n = (case["n0"], case["n1"], case["n2"])
    cells, nodes = float(n[0] * n[1] * n[2]), float((n[0] + 1) * (n[1] + 1) * (n[2] + 1))
    if path == "volume":  # one distance and one gradient per cell; no array in or out
        return {"bytes": 8.0, "flops": 25.0 * cells}
    if path == "plic":  # kind, valid; fraction, plane (4), six faces
        return {"bytes": cells * (2 + 11 * t), "flops": 25.0 * cells}
    if path == "mesh":
        return {"bytes": nodes * t, "flops": 0}
    if path == "plic_mesh":
        return {"bytes": cells * (1 + 4 * t), "flops": 0}
    if path == "field":  # the caller's values read, phi and the columns written
        return {"bytes": cells * (2 + 25 * t) + 2 * nodes * t, "flops": 0}
    report = cells * 2 if case.get("report") else 0
    return {"bytes": cells * (2 + 25 * t) + nodes * t + report, "flops": 25.0 * nodes}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits, without the framework

def _sphere64(x, c, r):
    d = [x[a] - c[a] for a in range(len(c))]
    s = torch.sqrt(sum(v * v for v in d))
    return s - r, [v / s for v in d]


def _box64(x, c, h):
    d = [x[a] - c[a] for a in range(3)]
    q = [v.abs() - k for v, k in zip(d, h)]
    out = torch.sqrt(sum(v.clamp(min=0) ** 2 for v in q))
    top = torch.maximum(torch.maximum(q[0], q[1]), q[2])
    # an exact box distance has no gradient by this form inside the box: 0 / 0, as its square root has none
    return out + top.clamp(max=0), [torch.sign(v) * k.clamp(min=0) / out for v, k in zip(d, q)]


def _torus64(x, c, major, minor, R):
    R = np.asarray(R, float)
    d = [x[a] - c[a] for a in range(3)]
    l = [R[i, 0] * d[0] + R[i, 1] * d[1] + R[i, 2] * d[2] for i in range(3)]
    rho = torch.sqrt(l[0] ** 2 + l[1] ** 2)
    q = rho - major
    s = torch.sqrt(q * q + l[2] ** 2)
    gl = [q / s * l[0] / rho, q / s * l[1] / rho, l[2] / s]
    return s - minor, [R[0, a] * gl[0] + R[1, a] * gl[1] + R[2, a] * gl[2] for a in range(3)]


def _prims64(case, seed):
    """The body's primitives as functions of the coordinates, and the smoothing (None: a plain union)."""
    b = _body3(case, seed)
    out = []
    for p in b.children:
        kind = type(p).__name__
        if kind == "Sphere":
            out.append(lambda x, p=p: _sphere64(x, p.center, p.radius))
        elif kind == "Box":
            out.append(lambda x, p=p: _box64(x, p.center, p.half))
        else:
            out.append(lambda x, p=p: _torus64(x, p.center, p.major, p.minor, p.rotation))
    return out, (b.k if case["body"] == "blob" else None)


def _eval64(prims, k, x):
    """phi and its gradient of a (smooth) union at the broadcastable coordinates x."""
    v, g = prims[0](x)
    for p in prims[1:]:
        w, e = p(x)
        near = w < v
        if k is None:
            g = [torch.where(near, b, a) for a, b in zip(g, e)]
            v = torch.where(near, w, v)
        else:
            h = (k - (v - w).abs()).clamp(min=0) / k
            sg = torch.sign(v - w)
            on = (h > 0).to(v.dtype)
            g = [torch.where(near, b, a) + 0.5 * h * sg * on * (a - b) for a, b in zip(g, e)]
            v = torch.where(near, w, v) - 0.25 * k * h * h
    return v, g


def _axes64(g, dev, half):
    """Node (half 0) or centroid (half 0.5) coordinates per axis."""
    return [g.x0[a] + (torch.arange(g.n[a] + (0 if half else 1), dtype=torch.float64, device=dev) + half) * g.d[a]
            for a in range(g.dim)]


_BITS = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))
_FACES = ((0, 3, 7, 4), (1, 2, 6, 5), (0, 1, 5, 4), (3, 2, 6, 7), (0, 1, 2, 3), (4, 5, 6, 7))


def _walk64(P, f, joined):
    """Twice the area and the three-fold first moments of the open part (f >= 0) of the quads P
    [N, 4, 2]: its boundary segments, closed by a chord from each crossing out of the open part to
    the next crossing into it (``joined``) or to the one before."""
    op = f >= 0
    sa, sb, a2, m = [], [], 0.0, [0.0, 0.0]

    def add(p, q, on):
        nonlocal a2
        cr = torch.where(on, p[:, 0] * q[:, 1] - p[:, 1] * q[:, 0], 0.0)
        a2 = a2 + cr
        for i in (0, 1):
            m[i] = m[i] + (p[:, i] + q[:, i]) * cr

    for k in range(4):
        n = (k + 1) % 4
        t = torch.where(op[:, k] != op[:, n], f[:, k] / (f[:, k] - f[:, n]), 0.0)[:, None]
        x = P[:, k] + t * (P[:, n] - P[:, k])
        sa.append(torch.where(op[:, k, None], P[:, k], x))
        sb.append(torch.where(op[:, n, None], P[:, n], x))
        add(sa[k], sb[k], op[:, k] | op[:, n])
    into = [~op[:, k] & op[:, (k + 1) % 4] for k in range(4)]
    for k in range(4):
        out = op[:, k] & ~op[:, (k + 1) % 4]
        there = sb[k]
        for step in (3, 2, 1):
            for way, pick in ((step, joined), (-step, ~joined)):
                j = (k + way) % 4
                there = torch.where((into[j] & pick)[:, None], sa[j], there)
        add(sb[k], there, out)
    return a2, m


def _mc64(phi, n, d, eps, dev):
    """Face fractions [cells, 6] and face centroids [cells, 12] of the nodal values phi. eps, of the
    cache's element type, is part of the method: a corner nearer to 0 counts as outside by eps, and
    a face whose determinant is below it as joined."""
    cells = n[0] * n[1] * n[2]
    phi = torch.where(phi.abs() < eps, eps, phi)
    v = phi.reshape(n[2] + 1, n[1] + 1, n[0] + 1)
    corner = [v[c:c + n[2], b:b + n[1], a:a + n[0]] for a, b, c in _BITS]
    outs = sum((w >= 0).to(torch.int8) for w in corner).reshape(-1)
    ff = torch.zeros(cells, 6, dtype=torch.float64, device=dev)
    ff[outs == 8] = 1.0
    half = [0.5 * d[q] for c in range(3) for _ in (0, 1) for q in range(3) if q != c]
    fcl = torch.tensor(half, dtype=torch.float64, device=dev).repeat(cells, 1)
    cut = torch.nonzero((outs != 0) & (outs != 8)).reshape(-1)
    ph = torch.stack([w.reshape(-1)[cut] for w in corner], 1)
    for k, nodes in enumerate(_FACES):
        c = k // 2
        p, q = [a for a in range(3) if a != c]
        f = ph[:, list(nodes)]
        P = torch.tensor([[_BITS[i][p] * d[p], _BITS[i][q] * d[q]] for i in nodes], dtype=torch.float64, device=dev)
        P = P.expand(len(cut), 4, 2)
        # the asymptotic decider: the open corners of a face are joined where the bilinear saddle is open
        det = f[:, 0] * f[:, 2] - f[:, 1] * f[:, 3]
        joined = (det.abs() < eps) | (f[:, 0] * det >= 0)
        a2, m = _walk64(P, f, joined)
        ff[cut, k] = 0.5 * a2 / (d[p] * d[q])
        for i, h in ((0, 0.5 * d[p]), (1, 0.5 * d[q])):
            fcl[cut, 2 * k + i] = torch.where(a2 != 0, m[i] / (3 * a2), h)
    return ff, fcl


def _ms64(nd, f, cs):
    """All fields of the 2D cells with corners nd [N, 4, 2] and values f [N, 4]."""
    o = nd[:, 0]
    P, op = nd - o[:, None], f >= 0
    whole = op.all(1) | ~op.any(1)
    a2, m = _walk64(P, f, torch.ones_like(whole))
    ce = 0.5 * cs
    out = {"volume_fraction": torch.where(whole, op[:, 0].to(f.dtype), 0.5 * a2 / (cs[:, 0] * cs[:, 1])),
           "centroid": o + torch.where((a2 != 0)[:, None] & ~whole[:, None],
                                       torch.stack([v / (3 * a2) for v in m], 1), ce)}
    ff, fcl, seg = [None] * 4, [None] * 4, []
    for k, face in enumerate((2, 1, 3, 0)):
        n = (k + 1) % 4
        a, b = op[:, k], op[:, n]
        t = torch.where(a != b, f[:, k] / (f[:, k] - f[:, n]), 0.0)
        x = P[:, k] + t[:, None] * (P[:, n] - P[:, k])
        s, e = torch.where(a[:, None], P[:, k], x), torch.where(b[:, None], P[:, n], x)
        on = a | b
        ff[face] = torch.where(a & b, 1.0, torch.where(a, t, torch.where(b, 1 - t, 0.0)))
        axis = 1 if face < 2 else 0
        fcl[face] = torch.where(on, 0.5 * (s + e)[:, axis], 0.5 * (P[:, k] + P[:, n])[:, axis])
        seg.append((s, e, on, a & ~b, ~a & b))
    length, im = 0.0, 0.0
    for k in range(4):
        there = seg[k][1]
        for step in (3, 2, 1):
            j = (k + step) % 4
            there = torch.where(seg[j][4][:, None], seg[j][0], there)
        w = torch.where(seg[k][3], (seg[k][1] - there).norm(dim=1), 0.0)
        length = length + w
        im = im + 0.5 * w[:, None] * (seg[k][1] + there)
    out["interface_centroid"] = o + torch.where((length > 0)[:, None], im / length[:, None], ce)
    out["face_fraction"], out["face_centroid_local"] = torch.stack(ff, 1), torch.stack(fcl, 1)
    return out


def _grid_ms64(g, c, r, dev):
    ax = _axes64(g, dev, 0.0)
    x, y = ax[0][None, :].expand(len(ax[1]), -1), ax[1][:, None].expand(-1, len(ax[0]))
    phi = torch.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2) - r
    at = ((0, 0), (1, 0), (1, 1), (0, 1))
    n0, n1 = g.n
    nd = torch.stack([torch.stack([w[b:b + n1, a:a + n0].reshape(-1) for w in (x, y)], 1) for a, b in at], 1)
    f = torch.stack([phi[b:b + n1, a:a + n0].reshape(-1) for a, b in at], 1)
    out = _ms64(nd, f, torch.tensor([g.d], dtype=torch.float64, device=dev))
    out["phi"] = phi.reshape(-1)
    return out


def _tree64(tree, star, dev):
    h = torch.tensor([tree.base_d], dtype=torch.float64, device=dev) * \
        2.0 ** -torch.as_tensor(tree.level, device=dev).double()[:, None]
    at = torch.as_tensor(tree.coord, device=dev).double()
    x0 = torch.tensor([tree.x0], dtype=torch.float64, device=dev)
    nd = torch.stack([x0 + (at + torch.tensor([b], device=dev)) * h for b in ((0, 0), (1, 0), (1, 1), (0, 1))], 1)
    th = torch.atan2(nd[..., 1], nd[..., 0])
    f = nd.norm(dim=2) - star.r0
    for k in range(2, 7):
        f = f - star.amp[k - 2] * torch.cos(k * th + star.phase[k - 2])
    out = _ms64(nd, f, h)
    out["phi"] = f
    return out


def _gvf64(n, a):
    """The fraction {n . x <= a} of the unit square or cube (Scardovelli and Zaleski 2000)."""
    al, m = a + sum(v.abs() * (v < 0) for v in n), [v.abs() for v in n]
    s = sum(m)
    flat = s == 0
    s = torch.where(flat, 1.0, s)
    al = al / s
    flip = al > 0.5
    b = torch.where(flip, 1 - al, al).clamp(min=0)
    m = torch.sort(torch.stack([v / s for v in m]), 0).values
    if len(n) == 2:
        v = torch.where(b < m[0], b * b / (2 * m[0] * m[1]), (b - 0.5 * m[0]) / m[1])
    else:
        m1, m2, m3 = m
        m12 = m1 + m2
        core = (3 * b * b - 3 * b * m1 + m1 * m1) / (6 * m2 * m3)
        e = 6 * m1 * m2 * m3
        u, w = (b - m2) ** 3, (b - m3) ** 3
        v = torch.where(m3 < m12, core - (u + w) / e, (2 * b - m12) / (2 * m3))
        v = torch.where(b < torch.minimum(m12, m3), core - u / e, v)
        v = torch.where(b < m2, core, v)
        v = torch.where(b < m1, b ** 3 / e, v)
    v = torch.where(flip, 1 - v, v)
    v = torch.where(al <= 0, 0.0, torch.where(al >= 1, 1.0, v))
    return torch.where(flat, (a >= 0).to(v.dtype), v)


def _plic_slabs64(case, seed, dev, layers=8):
    """(first layer, normals, intercept, solid fraction, valid) of the cell planes, a few layers at a time."""
    g = _grid3(case, iso=True)
    prims, k = _prims64(case, seed)
    ax = _axes64(g, dev, 0.5)
    for z in range(0, g.n[2], layers):
        x = torch.meshgrid(ax[2][z:z + layers], ax[1], ax[0], indexing="ij")[::-1]
        v, n = _eval64(prims, k, x)
        a = 0.5 * sum(n) - v / g.d[0]
        ok = ~(torch.isnan(a) | ((n[0] == 0) & (n[1] == 0) & (n[2] == 0)))
        n = [torch.where(ok, w, 0.0) for w in n]
        a = torch.where(ok, a, 0.0)
        yield z, n, a, torch.where(ok, _gvf64(n, a), (v <= 0).to(v.dtype)), ok


def _plic64(case, seed, dev):
    n0, n1, n2 = case["n0"], case["n1"], case["n2"]
    new = lambda *w: torch.empty(n2, n1, n0, *w, dtype=torch.float64, device=dev)  # noqa: E731
    out = {"normals": new(3), "intercepts": new(), "volume_fraction": new(), "face_fraction": new(6)}
    for z, n, a, solid, ok in _plic_slabs64(case, seed, dev):
        at = slice(z, z + a.shape[0])
        out["normals"][at] = torch.stack(n, -1)
        out["intercepts"][at] = a
        out["volume_fraction"][at] = 1 - solid
        for k in range(6):  # the fraction of its face that each cell's own plane leaves open
            c = k // 2
            p, q = [w for w in range(3) if w != c]
            one = 1 - _gvf64([n[p], n[q]], a - (k & 1) * n[c])
            out["face_fraction"][at, ..., k] = torch.where(ok, one, (1 - solid >= 0.5).to(a.dtype))
    ff = out["face_fraction"]
    for axis in range(3):  # a face between two cells takes the mean of what the two say
        d = 2 - axis
        lo = ff.narrow(d, 0, ff.shape[d] - 1).select(-1, 2 * axis + 1)
        hi = ff.narrow(d, 1, ff.shape[d] - 1).select(-1, 2 * axis)
        mean = 0.5 * (lo + hi)
        lo.copy_(mean)
        hi.copy_(mean)
    return {"normals": out["normals"].reshape(-1, 3), "intercepts": out["intercepts"].reshape(-1),
            "volume_fraction": out["volume_fraction"].reshape(-1), "face_fraction": ff.reshape(-1, 6)}


def exact(case, seed):
    path, dev = case["path"], torch.device("cuda")
    if path in ("mesh", "plic_mesh"):
        return None
    if path == "plic":
        return {**dict.fromkeys(PLIC_FIELDS + ("is_valid",)), **_plic64(case, seed, dev)}
    if path == "volume":
        g = _grid3(case, iso=True)
        return {"volume": sum(float(s.sum()) for _, _, _, s, _ in _plic_slabs64(case, seed, dev)) * g.d[0] ** 3}
    if path == "batch":
        each = [_grid_ms64(g, b.center, b.radius, dev) for g, b, _ in _updates(case, seed)]
        flat = {f: [e[f].reshape(-1) for e in each] for f in each[0]}
        pad = torch.nn.functional.pad
        return {**dict.fromkeys(FIELDS), **{f: torch.cat([pad(v, (0, -len(v) % 64)) for v in vs])
                                            for f, vs in flat.items()}}
    if path == "ms":
        return {**dict.fromkeys(FIELDS), **_grid_ms64(*_circle2(case, seed), dev)}
    if path == "tree":
        return {**dict.fromkeys(FIELDS), **_tree64(*_star(case, seed), dev)}
    g = _grid3(case)
    if path == "field":
        phi = _field(case, seed, dev).double()
    else:
        prims, k = _prims64(case, seed)
        ax = _axes64(g, dev, 0.0)
        phi = torch.empty(g.node_shape(), dtype=torch.float64, device=dev)
        for z in range(0, g.n[2] + 1, 8):
            x = torch.meshgrid(ax[2][z:z + 8], ax[1], ax[0], indexing="ij")[::-1]
            phi[z:z + 8] = _eval64(prims, k, x)[0]
    out = dict.fromkeys(FIELDS + ("fallback", "report"))
    out["phi"] = phi.reshape(-1)
    out["face_fraction"], out["face_centroid_local"] = _mc64(out["phi"], g.n, g.d, torch.finfo(_dtype(case)).eps, dev)
    out["face_centroid_local"] = out["face_centroid_local"].reshape(-1, 6, 2)
    return out
