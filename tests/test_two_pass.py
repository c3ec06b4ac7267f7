"""The two-pass 3-D step (H pass, E pass, in place), which the automatic path
takes for scenes with a CPML: against the CPU restatement at sizes where its
vectors, column groups and corrections have their edges, and its state against
the one-sweep path's.

FP64 evaluates the restatement's operations in its order: bit-identical.  FP32
rounds every operation once more than FP64 does: relative L2 <= 1e-4, the
project's bar for FP32 against FP64.
"""
import math

import numpy as np
import pytest

import xfdtd_cuda_b200 as X
from xfdtd_cuda_b200 import _lib as L
from xfdtd_cuda_b200 import simulation as S

from oracle import OracleSim

pytestmark = pytest.mark.gpu

DL = 2e-3
POLES = {
    "drude": [S.DrudePole(2e10, 1e9)],
    "debye": [S.DebyePole(2.0, 9e-12), S.DebyePole(1.0, 3e-11)],
    "lorentz": [S.DrudePole(2e10, 1e9), S.LorentzPole(2.0, 3e10, 5e8)],
}


def scene(n, pml, prec, ade=None, inset=(3, 3, 3), angles=(1.1, 0.7, 0.4), ball=None, freqs=(2e9,), source=True):
    """n inner cells, pml cells per face; a lossy block, a PEC ball and (ade) a dispersive ball."""
    s = S.Simulation(DL, DL, DL, 0.9, precision=prec)
    lo = [-v * DL / 2 for v in n]
    s.addObject(S.Object("domain", S.Cube(S.Vector(*lo), S.Vector(*(v * DL for v in n))), S.Material.createAir()))
    s.addObject(S.Object("block", S.Cube(S.Vector(lo[0] + 2.3 * DL, lo[1] + 3.6 * DL, lo[2] + 1.2 * DL),
                                         S.Vector(0.45 * n[0] * DL, 0.4 * n[1] * DL, 0.5 * n[2] * DL)),
                         S.Material("m", S.ElectroMagneticProperty(3.0, 2.0, 0.05, 1.0))))
    s.addObject(S.Object("pec", S.Sphere(S.Vector(0.2 * n[0] * DL, 0.1 * n[1] * DL, -0.1 * n[2] * DL), 2.7 * DL),
                         S.Material.createPec()))
    if ade:
        r = ball if ball is not None else 0.15 * min(n)
        s.addObject(S.Object("disp", S.Sphere(S.Vector(-0.4 * DL, 0.3 * DL, 0.6 * DL), r * DL),
                             S.DispersiveMaterial("d", 1.5, POLES[ade])))
    if source:
        s.addWaveformSource(S.TFSF3D(*inset, *angles, S.Waveform.gaussian(20 * DL / 6e8, 30 * DL / 6e8)))
    for d, t in enumerate(pml):
        if t:
            s.addBoundary(S.PML(t, d))
    if freqs:
        s.addNF2FF(S.NFFFTFrequencyDomain(2, 2, 2, list(freqs)))
    for q in range(4):
        s.addMonitor(S.PointMonitor(S.Vector(*(lo[a] + (0.2 + 0.17 * q) * n[a] * DL for a in range(3))), q))
    return s


def start(h, seed):
    """Random initial fields off the walls (the reference applies the CPML
    corrections of a face to the wall entries of its other faces too, where the
    engine keeps tangential E and normal H at zero)."""
    r = np.random.default_rng(seed)
    out = []
    for f in range(6):
        v = np.zeros(h.shape(f))
        inner = tuple(slice(1, m - 1) for m in v.shape)
        v[inner] = r.standard_normal(v[inner].shape) * (1.0 if f < 3 else 2e-3)
        out.append(v)
    return out


def results(h, o, freqs):
    got = [h.read_field(f) for f in range(6)] + [h.read_probe(p) for p in range(4)]
    want = [o.field(f) for f in range(6)] + [o.probe(p) for p in range(4)]
    for q in range(freqs):
        for face in range(6):
            for w in range(4):
                got.append(h.read_nf2ff(q, face, w))
                want.append(o.nf2ff(q, face, w))
    return got, want


CASES = [
    # nz covers every remainder of a 4-cell vector, CPML faces of whole and of
    # odd widths and missing faces (PEC walls); boxes next to the CPML
    dict(n=(17, 19, 20), pml=(6, 6, 6, 6, 6, 6)),
    dict(n=(16, 15, 24), pml=(4, 5, 6, 7, 8, 8)),
    dict(n=(15, 18, 21), pml=(5, 3, 4, 6, 7, 5), inset=(1, 1, 1)),
    dict(n=(18, 14, 22), pml=(0, 5, 5, 0, 5, 6), inset=(2, 1, 3)),
    dict(n=(14, 17, 23), pml=(5, 5, 5, 5, 0, 0), inset=(1, 2, 1)),
    dict(n=(16, 16, 33), pml=(4, 4, 0, 0, 4, 9), inset=(2, 2, 0)),   # TFSF face inside the z slab
    dict(n=(16, 16, 18), pml=(4, 4, 4, 4, 4, 4), inset=(0, 2, 2)),   # ... inside the x slab: one-sweep
    dict(n=(20, 18, 9), pml=(4, 4, 4, 4, 3, 3), inset=(3, 3, 3), freqs=()),  # TFSF lines in one vector
    dict(n=(40, 37, 130), pml=(6, 6, 6, 6, 6, 6), angles=(math.pi / 2, 0.0, 0.0)),  # several CTAs of each column group
    dict(n=(17, 19, 22), pml=(6, 6, 6, 6, 6, 6), source=False),
    dict(n=(22, 23, 25), pml=(5, 5, 5, 5, 5, 5), ade="drude"),
    dict(n=(24, 22, 26), pml=(5, 5, 5, 5, 5, 5), ade="debye"),
    dict(n=(22, 24, 23), pml=(6, 6, 6, 6, 6, 6), ade="lorentz"),
    dict(n=(22, 24, 23), pml=(6, 6, 6, 6, 6, 6), ade="lorentz", ball=9.3),   # reaches the TFSF box: recursion in the E pass
    dict(n=(18, 18, 20), pml=(5, 5, 5, 5, 5, 5), ade="debye", ball=12.0),   # ... and the CPML
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_matches_restatement(case, prec):
    kw = dict(CASES[case])
    steps, freqs = 29, len(kw.get("freqs", (0,)))
    h = X.Handle(*scene(prec=prec, **kw).lower())
    h.init(steps)
    o = OracleSim(X.Handle(*scene(prec="fp64", **kw).lower()), steps)
    for f, a in enumerate(start(h, case)):
        a = a if prec == "fp64" else a.astype(np.float32).astype(np.float64)
        h.write_field(f, a)
        o.set_field(f, a)
    h.step(steps)
    h.sync()
    o.run(steps)
    for q, (a, b) in enumerate(zip(*results(h, o, freqs))):
        if prec == "fp64":
            assert np.array_equal(a, b), q
        else:
            assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b), q
    h.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("first,second", [(L.PATH_AUTO, L.PATH_FUSED), (L.PATH_FUSED, L.PATH_AUTO)])
@pytest.mark.parametrize("cut", [6, 7])
def test_state_moves_between_step_forms(prec, first, second, cut):
    """A checkpoint of one form continues in the other, at even and odd steps."""
    def handle(path):
        h = X.Handle(*scene((20, 22, 21), (5,) * 6, prec, ade="lorentz").lower())
        h.set_kernel_path(path)
        h.init(17)
        return h

    a, b, c = handle(first), handle(second), handle(second)
    a.step(cut)
    b.set_state(a.get_state())
    a.step(17 - cut)  # the form that was saved goes on as well
    b.step(17 - cut)
    c.step(17)
    for h in (a, b, c):
        h.sync()
    for f in range(6):
        if prec == "fp64":
            assert np.array_equal(a.read_field(f), c.read_field(f)) and np.array_equal(b.read_field(f), c.read_field(f)), f
        else:
            want = c.read_field(f)
            assert np.linalg.norm(a.read_field(f) - want) <= 1e-4 * np.linalg.norm(want), f
            assert np.linalg.norm(b.read_field(f) - want) <= 1e-4 * np.linalg.norm(want), f
    for h in (a, b, c):
        h.close()
