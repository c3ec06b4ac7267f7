"""Probes on the outer walls of the blocked 2-D step, whose H entries no update
writes: they record the stored field, as one launch per step does, whatever E
the walls hold (random fields everywhere, walls too).  Bit-identical in FP64."""
import math

import numpy as np
import pytest

import xfdtd_cuda_b200 as X
from xfdtd_cuda_b200 import _lib as L

pytestmark = pytest.mark.gpu

DL = 1e-3
FIELDS = (L.EZ, L.HX, L.HY)


def _run(pml, tb):
    nx, ny = 75, 61
    s = X.Simulation(DL, DL, 1.0, 0.9, precision="fp64")
    s.addObject(X.Object("domain", X.Cube(X.Vector(0, 0, -math.inf), X.Vector(nx * DL, ny * DL, math.inf)),
                         X.Material.createAir()))
    for d in range(4):
        if pml:
            s.addBoundary(X.PML(pml, d))
    w, h = (nx + 2 * pml) * DL, (ny + 2 * pml) * DL  # the grid, from -pml cells
    for t in (0.02, 0.3, 0.77):  # upper walls, lower walls, inside
        for x, y in ((w, t * h), (t * w, h), (0, t * h), (t * w, 0), (t * w, 0.5 * h)):
            for f in FIELDS:
                s.addMonitor(X.PointMonitor(X.Vector(x - pml * DL, y - pml * DL, 0), f))
    hd = X.Handle(*s.lower())
    hd.set_temporal_block(tb)
    hd.init(40)
    r = np.random.default_rng(3)
    for f in FIELDS:
        hd.write_field(f, r.standard_normal(hd.shape(f)))
    hd.step(40)
    hd.sync()
    out = [hd.read_probe(q) for q in range(len(hd.probe_desc))], [hd.read_field(f) for f in FIELDS]
    desc, shapes = hd.probe_desc, {f: hd.shape(f) for f in FIELDS}
    hd.close()
    return out, desc, shapes


@pytest.mark.parametrize("pml", [0, 6])
def test_wall_probes_record_the_stored_field(pml):
    (want, wf), desc, shapes = _run(pml, 0)
    (got, gf), _, _ = _run(pml, 9)
    assert any(d[0] == L.HX and d[1] == shapes[L.HX][0] - 1 for d in desc)  # Hx on the upper x wall
    assert any(d[0] == L.HY and d[2] == shapes[L.HY][1] - 1 for d in desc)  # Hy on the upper y wall
    for f, a, b in zip(FIELDS, gf, wf):
        assert np.array_equal(a, b), f
    for d, a, b in zip(desc, got, want):
        assert np.array_equal(a, b), d
