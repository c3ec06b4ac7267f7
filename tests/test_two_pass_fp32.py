"""The two-pass step's FP32 kernels, on scenes that it takes: the automatic path
against the one-sweep path, to the last bit, and which of the two each handle
ran.  (In FP32 a scene whose TFSF box has two faces in one tile of the one-sweep
step stays there, so the boxes here are wider than a tile: 16 rows, 32 columns.)
"""
import math

import numpy as np
import pytest

import xfdtd_cuda_b200 as X
from test_two_pass import DL, scene, start
from xfdtd_cuda_b200 import _lib as L
from xfdtd_cuda_b200 import simulation as S

pytestmark = pytest.mark.gpu

CASES = [
    # z slabs in whole vectors (one 16-byte access) and not, every remainder of
    # a 4-cell vector, missing faces
    dict(n=(18, 28, 44), pml=(4, 4, 4, 4, 4, 4)),
    dict(n=(18, 28, 48), pml=(8, 8, 8, 8, 8, 8), inset=(1, 1, 1)),
    dict(n=(17, 27, 45), pml=(5, 3, 4, 6, 7, 5)),
    dict(n=(16, 30, 46), pml=(0, 5, 5, 0, 5, 7), inset=(2, 1, 3)),
    dict(n=(18, 28, 50), pml=(5, 5, 4, 4, 0, 0)),
    dict(n=(18, 28, 50), pml=(5, 5, 4, 4, 4, 9), inset=(2, 2, 0)),   # TFSF face at the z slab
    dict(n=(33, 70, 130), pml=(6, 6, 6, 6, 6, 6), angles=(math.pi / 2, 0.0, 0.0)),
    dict(n=(17, 19, 22), pml=(6, 6, 6, 6, 6, 6), source=False),
    dict(n=(18, 28, 44), pml=(4, 4, 4, 4, 4, 4), layers=True),       # materials mixed in every slab's vectors
    dict(n=(18, 28, 45), pml=(5, 3, 4, 6, 7, 5), layers=True),
    dict(n=(30, 30, 48), pml=(5, 5, 5, 5, 4, 4), ade="drude"),
    dict(n=(30, 32, 47), pml=(5, 5, 5, 5, 5, 5), ade="debye"),
    dict(n=(32, 30, 46), pml=(6, 6, 6, 6, 6, 6), ade="lorentz"),
]


def _sim(layers=False, **kw):
    s = scene(prec="fp32", **kw)
    if layers:  # plates a cell thick along z, through the CPML
        n = kw["n"]
        for k in range(-8, n[2] + 8, 2):
            s.addObject(S.Object(f"plate{k}", S.Cube(
                S.Vector(-n[0] * DL, -n[1] * DL, (k - n[2] / 2) * DL), S.Vector(2 * n[0] * DL, 2 * n[1] * DL, DL)),
                S.Material(f"p{k}", S.ElectroMagneticProperty(1.5 + 0.1 * (k % 5), 1.0 + 0.1 * (k % 3), 0.01, 0.5))))
    return s


def _handle(path, steps, **kw):
    h = X.Handle(*_sim(**kw).lower())
    h.set_kernel_path(path)
    h.init(steps)
    return h


def _took_two_passes(h):
    """Whether a step of `h` is an H pass and an E pass (advances it one step)."""
    _, count = h.profile_kernels(1)
    assert (count[L.K_UPDATE_H] > 0) != (count[L.K_STEP] > 0)
    return count[L.K_UPDATE_H] > 0


def _results(h, freqs):
    out = [h.read_field(f) for f in range(6)] + [h.read_probe(p) for p in range(4)]
    return out + [h.read_nf2ff_all(q) for q in range(freqs)]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_equals_one_sweep(case):
    kw, steps = CASES[case], 43
    res = []
    for path in (L.PATH_AUTO, L.PATH_FUSED):
        h = _handle(path, steps, **kw)
        for f, a in enumerate(start(h, case)):
            h.write_field(f, a)
        h.step(steps - 1)
        h.sync()
        assert _took_two_passes(h) == (path == L.PATH_AUTO)
        res.append(_results(h, 1))
        h.close()
    for q, (a, b) in enumerate(zip(*res)):
        assert np.isfinite(b).all() and (q >= 6 or np.abs(b).max() > 0), q
        assert np.array_equal(a, b), q


@pytest.mark.parametrize("first,second", [(L.PATH_AUTO, L.PATH_FUSED), (L.PATH_FUSED, L.PATH_AUTO)])
@pytest.mark.parametrize("cut", [6, 7])
@pytest.mark.parametrize("case", [0, 2, 12])
def test_state_moves_to_the_last_bit(case, cut, first, second):
    """A checkpoint of one form continues in the other, at even and odd steps."""
    kw, steps = CASES[case], 18
    a, b, c = (_handle(p, steps, **kw) for p in (first, second, second))
    for h in (a, c):
        for f, v in enumerate(start(h, case)):
            h.write_field(f, v)
    a.step(cut)
    b.set_state(a.get_state())
    a.step(steps - cut - 1)
    b.step(steps - cut - 1)
    c.step(steps - 1)
    for h, path in ((a, first), (b, second), (c, second)):
        h.sync()
        assert _took_two_passes(h) == (path == L.PATH_AUTO)
    want = _results(c, 0)  # (a checkpoint adds the NF2FF samples at other steps: round-off)
    for h in (a, b):
        for q, (got, w) in enumerate(zip(_results(h, 0), want)):
            assert np.array_equal(got, w), q
    for h in (a, b, c):
        h.close()
