"""Dispersive cells of the two-pass step, inside the E pass and in a pass of
their own.

Media of one and two poles run inside the E pass (blocks after those of their
plane), three and four poles in k_tp_ade.  The scatterers start or end on the
32-cell segments the runs are cut at, leave planes without runs above and below
them, and have planes with a single run.  FP64 against the CPU oracle bit for
bit; FP32 against the one-sweep step, whose deferred ADE pass has the same
formulas, to the 1e-4 bar of the FP32 engine.
"""
import math

import numpy as np
import pytest

import xfdtd_cuda_b200 as X
from helpers import bit_equal, compare_fields, fields_of, oracle_of
from xfdtd_cuda_b200 import _lib as L
from xfdtd_cuda_b200 import configs

pytestmark = pytest.mark.gpu

POLES = [X.DrudePole(2e10, 1e9), X.LorentzPole(2.0, 3e10, 5e8), X.LorentzPole(1.0, 5e10, 1e9), X.DrudePole(1e10, 3e9)]


def _sim(prec, poles, shape):
    dl, n = 1e-3, (50, 44, 70)
    s = X.Simulation(dl, dl, dl, 0.9, precision=prec)
    s.addObject(X.Object("domain", X.Cube(X.Vector(0, 0, 0), X.Vector(*(v * dl for v in n))), X.Material.createAir()))
    m = X.DispersiveMaterial("m", 1.5, [POLES[q] for q in poles])
    body = (X.Sphere(X.Vector(25 * dl, 22 * dl, 35 * dl), 11.4 * dl) if shape == "sphere"
            else X.Cube(X.Vector(20 * dl, 15 * dl, 25 * dl), X.Vector(9 * dl, 13 * dl, 32 * dl)))
    s.addObject(X.Object("body", body, m))
    s.addWaveformSource(X.TFSF3D(5, 5, 5, math.pi / 3, 0.4, 0.2, configs._gaussian(dl)))
    for d in range(6):
        s.addBoundary(X.PML(7, d))
    return s


def _run(sim, steps, path):
    h = X.Handle(*sim.lower())
    h.set_kernel_path(path)
    h.init(steps)
    h.step(steps)
    h.sync()
    return h


@pytest.mark.parametrize("shape", ["sphere", "slab"])
@pytest.mark.parametrize("poles", [(0,), (1,), (0, 1), (0, 1, 2), (0, 1, 2, 3)])
def test_runs_inside_and_apart(poles, shape):
    steps = 50
    a = _run(_sim("fp64", poles, shape), steps, L.PATH_AUTO)
    o = oracle_of(_sim("fp64", poles, shape), steps)
    o.run(steps)
    assert a.info().launches_per_step == (2 if len(poles) <= 2 else 3)
    fo = fields_of(o, 3)
    assert all(np.abs(f).max() > 0 for f in fo.values())
    assert bit_equal(fields_of(a, 3), fo)
    a.close()
    b = _run(_sim("fp32", poles, shape), steps, L.PATH_AUTO)
    c = _run(_sim("fp32", poles, shape), steps, L.PATH_FUSED)
    assert compare_fields(fields_of(b, 3), fields_of(c, 3)) <= 1e-4
    b.close()
    c.close()
