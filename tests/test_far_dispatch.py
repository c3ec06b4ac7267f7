"""Which far-field kernel a call takes (far_many): on thin boxes, whose rows or
columns leave most of k_far_many idle, a call of 2048 directions costs no more
than two calls of 1024 (20 % for the clock), as it does with k_far; and the two
kernels agree at counts that fill the last warp partly, on sides that are no
multiple of a column chunk."""
import time

import numpy as np
import pytest

import xfdtd_cuda_b200 as X
from xfdtd_cuda_b200 import simulation as S

pytestmark = pytest.mark.gpu

DL = 1e-3


def _run(n, prec="fp32"):
    s = S.Simulation(DL, DL, DL, 0.9, precision=prec)
    lo = [-v * DL / 2 for v in n]
    s.addObject(S.Object("domain", S.Cube(S.Vector(*lo), S.Vector(*(v * DL for v in n))), S.Material.createAir()))
    s.addWaveformSource(S.TFSF3D(2, 2, 2, 1.0, 0.5, 0.3, S.Waveform.gaussian(6 * DL / 6e8, 10 * DL / 6e8)))
    for d in range(6):
        s.addBoundary(S.PML(5, d))
    s.addNF2FF(S.NFFFTFrequencyDomain(1, 1, 1, [5e9]))
    h = X.Handle(*s.lower())
    h.run(60)
    return h


def _angles(count):
    r = np.random.default_rng(count)
    return r.uniform(0, np.pi, count), r.uniform(-np.pi, np.pi, count)


@pytest.mark.parametrize("n", [(6, 6, 300), (6, 200, 6), (300, 6, 6)])
def test_thin_boxes_cost_no_more_per_direction(n):
    h = _run(n)
    us = {}
    for count in (1024, 2048):
        a = _angles(count)
        h.far_field_static(0, *a)
        t = []
        for _ in range(25):
            t0 = time.perf_counter()
            h.far_field_static(0, *a)
            t.append(time.perf_counter() - t0)
        us[count] = min(t) * 1e6
    h.close()
    assert us[2048] <= 1.2 * 2 * us[1024], us


@pytest.mark.parametrize("n", [(20, 23, 37), (36, 9, 21), (52, 52, 40)])
@pytest.mark.parametrize("count", [4736, 4737, 9473])
def test_kernels_agree(n, count):
    h = _run(n, "fp64")
    th, ph = _angles(count)
    many = h.far_field(0, th, ph)
    parts = [h.far_field(0, th[o:o + 500], ph[o:o + 500]) for o in range(0, count, 500)]
    for q in range(2):
        few = np.concatenate([p[q] for p in parts])
        assert np.abs(few).max() > 0
        assert np.linalg.norm(many[q] - few) <= 1e-13 * np.linalg.norm(few)
    h.close()
