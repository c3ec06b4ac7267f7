"""The records of a step share one launch (time-domain NF2FF chunks, NF2FF
points, probes): every one must be what it is when it is the only one.

260 probes need two blocks, the last nearly empty; the NF2FF boxes have point
counts that are no multiple of a block.  The same field values reach the same
arithmetic in either launch, so the comparison is bit for bit, in both
precisions; the probes also equal the fields read back after the last step.
"""
import math

import numpy as np
import pytest

import xfdtd_cuda_b200 as X
from xfdtd_cuda_b200 import _lib as L
from xfdtd_cuda_b200 import configs

pytestmark = pytest.mark.gpu

DL, N, PML, STEPS = 1e-3, (34, 27, 41), 6, 60


def _run(prec, nf, td, probes):
    s = X.Simulation(DL, DL, DL, 0.9, precision=prec)
    s.addObject(X.Object("domain", X.Cube(X.Vector(0, 0, 0), X.Vector(*(v * DL for v in N))), X.Material.createAir()))
    s.addObject(X.Object("ball", X.Sphere(X.Vector(17 * DL, 13 * DL, 20 * DL), 7 * DL),
                         X.Material("m", X.ElectroMagneticProperty(3, 1, 0.01, 0))))
    s.addWaveformSource(X.TFSF3D(5, 5, 5, math.pi / 3, 0.3, 0.1, configs._gaussian(DL)))
    for d in range(6):
        s.addBoundary(X.PML(PML, d))
    if nf:
        s.addNF2FF(X.NFFFTFrequencyDomain(3, 3, 3, [1e9, 4e9]))
    if td:
        s.addNF2FF(X.NFFFTTimeDomain(2, 2, 2, "", math.pi / 4, 0.5))
    rng = np.random.default_rng(5)
    for _ in range(probes):
        s.addMonitor(X.PointMonitor(X.Vector(*(rng.uniform(0.05, 0.95) * v * DL for v in N)), int(rng.integers(6))))
    h = X.Handle(*s.lower())
    h.init(STEPS)
    h.step(STEPS)
    h.sync()
    out = {"launches": h.info().launches_per_step}
    if nf:
        out["nf"] = [h.read_nf2ff_all(f) for f in range(2)]
    if td:
        out["td"] = [h.read_nf2ff_td(w) for w in range(6)]
    if probes:
        out["probe"] = [h.read_probe(p) for p in range(probes)]
        fields = [h.read_field(f) for f in range(6)]
        assert all(h.read_probe(p)[-1] == fields[d[0]][d[1:]] for p, d in enumerate(h.probe_desc))
    h.close()
    return out


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_records_in_one_launch(prec):
    alone = {**_run(prec, True, False, 0), **_run(prec, False, True, 0), **_run(prec, False, False, 260)}
    assert all(np.abs(a).max() > 0 for k in ("nf", "td") for a in alone[k])
    for nf, td, probes in ((True, True, 260), (True, False, 260), (False, True, 260), (True, True, 0)):
        both = _run(prec, nf, td, probes)
        assert both["launches"] == 3 + td
        for k in both:
            if k != "launches":
                assert all(np.array_equal(a, b) for a, b in zip(both[k], alone[k])), (k, nf, td, probes)
