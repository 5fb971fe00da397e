"""The longest tapes in the 3D PLIC passes and calc_volume: a tape and its lists take up to 50 KB of shared
memory beside a kernel's own arrays, more than a launch may take without asking. Bit for bit against
the oracle, at lengths on both sides of where a launch has to ask (217 smooth spheres at Float64 fit)."""
import importlib
import math

import numpy as np
import pytest
import torch

from helpers import assert_cells_bitwise, bits, cc, po

pytestmark = pytest.mark.gpu

G = importlib.import_module("cutcell_b200.geometry")
PREC = [("f64", 1), ("f32", 0), ("mixed", 2)]


def _smooth_spheres(n):
    rng = np.random.default_rng(n)
    return cc.flatten(cc.SmoothUnion(*[cc.Sphere(tuple(rng.uniform(0.0, 0.9, 3)), float(rng.uniform(0.02, 0.09)))
                                       for _ in range(n)], k=0.02), 3)


def _tori(n, mode):
    """n tori from the parameters of 20, as a C caller may share them."""
    rng = np.random.default_rng(n)
    params = []
    for _ in range(20):
        c = rng.uniform(0.0, 0.9, 3)
        params += [*c, *cc.quat_to_matrix(rng.normal(size=4)).ravel(), 0.1, 0.03]
    params.append(0.02)
    ops = np.zeros(n, G.OP_DTYPE)
    ops["opcode"] = G.OP_TORUS
    ops["combine"] = mode
    ops["combine"][0] = G.COMB_PUSH
    ops["poff"] = 14 * (np.arange(n) % 20)
    ops["kparam"] = len(params) - 1
    return cc.Tape(ops, np.array(params), 3)


TAPES = {**{f"smooth_{n}": (lambda n=n: _smooth_spheres(n)) for n in (216, 217, 218, 255)},
         **{f"tori_{n}": (lambda n=n: _tori(n, G.COMB_MIN)) for n in (164, 166, 256)},
         **{f"smooth_tori_{n}": (lambda n=n: _tori(n, G.COMB_SMIN)) for n in (140, 256)}}


@pytest.mark.parametrize("name", sorted(TAPES))
@pytest.mark.parametrize("pname,prec", PREC)
def test_plic_and_volume_of_long_tapes(name, pname, prec):
    dtype, T = (torch.float64, np.float64) if prec == 1 else (torch.float32, np.float32)
    precision = "mixed" if prec == 2 else "plain"
    g = cc.CartesianGrid((-0.07, 0.03, -0.02), (33, 9, 5), (1.0 / 33,) * 3)
    tape = TAPES[name]()
    c = cc.update_cache(cc.allocate_cache(g, cc.PLICCutCell(), dtype=dtype, precision=precision), tape, g)
    ref, rn, ri, rv = po.plic_update(g, tape, prec)
    assert_cells_bitwise(c.to_host(), ref, fields=("kind", "volume_fraction", "face_fraction"), label=name)
    assert np.array_equal(bits(c.normals.cpu().numpy()), bits(rn))
    assert np.array_equal(bits(c.intercepts.cpu().numpy()), bits(ri))
    assert np.array_equal(c.is_valid.cpu().numpy(), rv)
    total = math.fsum(po.plic_fractions(g, tape, prec).tolist())
    h = T(g.d[0])
    v = cc.calc_volume(tape, g, dtype=dtype, precision=precision)
    assert abs(v / float(h * h * h) - total) <= 6 * 2.0 ** -53 * max(1.0, total)


@pytest.mark.parametrize("pname,prec", PREC)
def test_the_longest_2d_tape(pname, prec):
    """256 star curves blended: in 2D the tape, its pruned ops and their bounds take 48 KB exactly."""
    dtype, T = (torch.float64, np.float64) if prec == 1 else (torch.float32, np.float32)
    precision = "mixed" if prec == 2 else "plain"
    params = [0.4, 0.3, 0.2] + [0.0] * 10 + [0.02]  # circles: no angle, so host and device agree to the bit
    ops = np.zeros(256, G.OP_DTYPE)
    ops["opcode"] = G.OP_STAR
    ops["combine"] = G.COMB_SMIN
    ops["combine"][0] = G.COMB_PUSH
    ops["kparam"] = 13
    tape = cc.Tape(ops, np.array(params), 2)
    g = cc.CartesianGrid((0.0, 0.0), (40, 19), (1.0 / 40,) * 2)
    c = cc.update_cache(cc.allocate_cache(g, cc.PLICCutCell(), dtype=dtype, precision=precision), tape, g)
    ref, rn, ri, rv = po.plic_update(g, tape, prec)
    assert_cells_bitwise(c.to_host(), ref, fields=("kind", "volume_fraction", "face_fraction"))
    total = math.fsum(po.plic_fractions(g, tape, prec).tolist())
    h = T(g.d[0])
    v = cc.calc_volume(tape, g, dtype=dtype, precision=precision)
    assert abs(v / float(h * h) - total) <= 6 * 2.0 ** -53 * max(1.0, total)
