"""Far field of many directions (k_far_many) against the numpy integral of the
same surface currents, around the direction count from which it is used and at
counts that leave its last warp partly filled; box sides that are no multiple
of its column chunk."""
import numpy as np
import pytest

import xfdtd_cuda_b200 as X
from xfdtd_cuda_b200 import simulation as S

from oracle import far_field_numpy

pytestmark = pytest.mark.gpu

TOL = 1e-10  # the project's bar for the device far field against numpy


@pytest.fixture(scope="module", params=[(20, 23, 37), (36, 9, 21)])
def run(request):
    n, dl = request.param, 4e-3
    s = S.Simulation(dl, dl, dl, 0.9, precision="fp64")
    lo = [-v * dl / 2 for v in n]
    s.addObject(S.Object("domain", S.Cube(S.Vector(*lo), S.Vector(*(v * dl for v in n))), S.Material.createAir()))
    s.addObject(S.Object("ball", S.Sphere(S.Vector(0.1 * dl, 0.2 * dl, -0.3 * dl), 2.6 * dl),
                         S.Material("m", S.ElectroMagneticProperty(3.0, 1.0, 0.0, 0.0))))
    s.addWaveformSource(S.TFSF3D(3, 3, 3, 1.0, 0.5, 0.3, S.Waveform.gaussian(20 * dl / 6e8, 40 * dl / 6e8)))
    for d in range(6):
        s.addBoundary(S.PML(5, d))
    s.addNF2FF(S.NFFFTFrequencyDomain(1, 1, 1, [1.5e9, 4e9]))
    h = X.Handle(*s.lower())
    h.run(90)
    gi = h.info()
    cur = [[[h.read_nf2ff(f, face, w) for w in range(4)] for face in range(6)] for f in range(2)]
    yield h, cur, list(gi.nf2ff_box), list(gi.origin), (gi.dx, gi.dy, gi.dz)
    h.close()


@pytest.mark.parametrize("count", [2047, 2048, 2049, 2111, 4096])
@pytest.mark.parametrize("freq", [0, 1])
def test_matches_numpy(run, count, freq):
    h, cur, box, origin, d = run
    r = np.random.default_rng(count)
    th, ph = r.uniform(0, np.pi, count), r.uniform(-np.pi, np.pi, count)
    want = far_field_numpy(cur[freq], box, origin, d, (1.5e9, 4e9)[freq], th, ph)
    for got in (h.far_field(freq, th, ph), h.far_field_static(freq, th, ph)):
        for a, b in zip(got, want):
            assert np.linalg.norm(a - b) <= TOL * np.linalg.norm(b)
