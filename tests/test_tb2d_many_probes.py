"""Blocked 2-D step with lines of several hundred probes: many in one lane's
block, several on one node, every component, in every tile.

FP64 series are bit-identical to the CPU oracle's.  A launch finds its tiles'
probes once, so the blocked step stays ahead of one launch per step, which
records them by a kernel of its own (measured with 600 probes on 320 x 220
cells: 17.6 us per step there, 163 when every lane scanned the list)."""
import math

import numpy as np
import pytest

import xfdtd_cuda_b200 as X
from helpers import oracle_of
from xfdtd_cuda_b200 import _lib as L

pytestmark = pytest.mark.gpu

DL = 1e-3
FIELDS = (L.EZ, L.HX, L.HY)


def _scene(nx, ny, nodes, prec):
    s = X.Simulation(DL, DL, 1.0, 0.9, precision=prec)
    s.addObject(X.Object("domain", X.Cube(X.Vector(0, 0, -math.inf), X.Vector(nx * DL, ny * DL, math.inf)),
                         X.Material.createAir()))
    s.addWaveformSource(X.TFSF2D(12, 12, 0.6, X.Waveform.gaussian(6 * DL / 6e8, 12 * DL / 6e8)))
    for d in range(4):
        s.addBoundary(X.PML(7, d))
    for q, (i, j) in enumerate(nodes):
        s.addMonitor(X.PointMonitor(X.Vector(i * DL, j * DL, 0), FIELDS[q % 3]))
    return s


def _lines(nx, ny, n):
    """n nodes: a row and a column of the grid walked cell by cell, every
    seventh node three times over."""
    out = []
    q = 0
    while len(out) < n:
        i, j = (q % nx, ny // 3) if (q // nx) % 2 == 0 else (nx // 3, q % ny)
        out += [(i, j)] * (3 if q % 7 == 0 else 1)
        q += 1
    return out[:n]


@pytest.mark.parametrize("tb", [None, 5])
def test_many_probes_match_oracle(tb):
    nx, ny, steps = 141, 118, 250
    nodes = _lines(nx, ny, 700)
    h = X.Handle(*_scene(nx, ny, nodes, "fp64").lower())
    if tb is not None:
        h.set_temporal_block(tb)
    h.init(steps)
    h.step(steps)
    h.sync()
    assert h.info().launches_per_step == 1
    o = oracle_of(_scene(nx, ny, nodes, "fp64"), steps)
    o.run(steps)
    assert sum(np.abs(o.probe(p)).max() > 0 for p in range(len(nodes))) > len(nodes) // 2
    for p in range(len(nodes)):
        assert np.array_equal(h.read_probe(p), o.probe(p)), (p, h.probe_desc[p])
    h.close()


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_many_probes_cost_less_than_a_launch_per_step(prec):
    nx, ny, steps = 306, 206, 192
    us = []
    for tb in (None, 0):
        h = X.Handle(*_scene(nx, ny, _lines(nx, ny, 600), prec).lower())
        if tb is not None:
            h.set_temporal_block(tb)
        h.init(8 * steps)
        h.step(steps)
        h.sync()
        us.append(min(h.timed_step(steps) for _ in range(4)) / steps * 1e3)
        h.close()
    assert us[0] <= us[1], us
