"""Blocked 2-D step at the edges of its tiles.

A CTA of w warps holds w row blocks of 4 (FP32) or 3 (FP64) rows and 128
columns; S steps eat S rows and columns on each side.  The sizes put one row,
one column or less than a lane's block into the last tile, span several tiles,
and lay TFSF boxes so thin that both their faces fall into one lane's block.

FP64: fields and probes bit-identical to the CPU oracle.  FP32: both paths
compute the same formulas with the same contractions, so they agree to the last
bit; asserted to 1e-6 relative L2, the bound of round-off that reordering one
sum could cause.
"""
import math

import numpy as np
import pytest

import xfdtd_cuda_b200 as X
from conftest import rel_l2
from helpers import oracle_of
from xfdtd_cuda_b200 import _lib as L

pytestmark = pytest.mark.gpu

DL = 1e-3


def _scene(nx, ny, pml, inset, prec, angle=0.0):
    s = X.Simulation(DL, DL, 1.0, 0.9, precision=prec)
    s.addObject(X.Object("domain", X.Cube(X.Vector(0, 0, -math.inf), X.Vector(nx * DL, ny * DL, math.inf)),
                         X.Material.createAir()))
    s.addObject(X.Object("rod", X.Cylinder(X.Vector(0.4 * nx * DL, 0.6 * ny * DL, 0), 0.15 * min(nx, ny) * DL, math.inf, 2),
                         X.Material("m", X.ElectroMagneticProperty(3, 1.5, 0.02, 0.1))))
    tau = 6 * DL / 6e8
    s.addWaveformSource(X.TFSF2D(inset[0], inset[1], angle, X.Waveform.gaussian(tau, 2 * tau)))
    for d in range(4):
        s.addBoundary(X.PML(pml, d))
    for x, y in ((0.1, 0.1), (0.5, 0.5), (0.93, 0.2), (0.3, 0.95)):
        s.addMonitor(X.PointMonitor(X.Vector(x * nx * DL, y * ny * DL, 0), X.EMF.Field.EZ))
    return s


def _run(sim, steps, tb):
    sc, keep = sim.lower()
    h = X.Handle(sc, keep)
    if tb is not None:
        h.set_temporal_block(tb)
    h.init(steps)
    h.step(steps)
    h.sync()
    return h


# (inner nx, ny, CPML, TFSF insets from the outer edge, block steps or None)
CASES = [
    (101, 93, 6, (9, 9), None),     # ragged both ways, the plan's own block
    (97, 118, 8, (11, 58), 7),      # TFSF box two columns wide
    (119, 97, 8, (59, 12), 5),      # TFSF box one row wide
    (33, 225, 5, (8, 8), 11),       # one tile of rows, several of columns
    (257, 40, 5, (8, 8), 3),        # several tiles of rows, part of one of columns
    (96, 112, 4, (7, 7), 25),       # more steps than the registers hold: shorter blocks
    (140, 131, 3, (4, 5), 1),       # one step per launch in registers
]


@pytest.mark.parametrize("nx,ny,pml,inset,tb", CASES)
def test_tile_edges(nx, ny, pml, inset, tb):
    steps = 75
    b = _run(_scene(nx, ny, pml, inset, "fp64", 0.7), steps, tb)
    o = oracle_of(_scene(nx, ny, pml, inset, "fp64", 0.7), steps)
    o.run(steps)
    assert b.info().launches_per_step == 1
    for f in (L.EZ, L.HX, L.HY):
        assert np.abs(o.field(f)).max() > 0
        assert np.array_equal(b.read_field(f), o.field(f)), f
    for p in range(len(b.probe_desc)):
        assert np.array_equal(b.read_probe(p), o.probe(p)), p
    b.close()
    c = _run(_scene(nx, ny, pml, inset, "fp32", 0.7), steps, tb)
    d = _run(_scene(nx, ny, pml, inset, "fp32", 0.7), steps, 0)
    for f in (L.EZ, L.HX, L.HY):
        assert rel_l2(c.read_field(f), d.read_field(f)) <= 1e-6, f
    c.close()
    d.close()
