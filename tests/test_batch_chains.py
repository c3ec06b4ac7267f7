"""Batches whose scenes step as parallel chains of the two-pass step.

More scenes than chains, scenes with monitors next to scenes without, runs of
odd lengths, a checkpoint read in the middle (which may move a scene's state to
the other field set) and a switch to the one-sweep kernels in the middle: every
scene must end where it ends when it is stepped alone.  Both paths apply the
same formulas with the same contractions, so both precisions are compared bit
for bit.
"""
import numpy as np
import pytest

import xfdtd_cuda_b200 as X
from xfdtd_cuda_b200 import _lib as L
from xfdtd_cuda_b200 import configs

pytestmark = pytest.mark.gpu

FIELDS = (L.EX, L.EY, L.EZ, L.HX, L.HY, L.HZ)


def _sims(prec, n):
    sims = configs.batched_sweep(n=n, seed=7, lo=56, hi=72, pml=6, precision=prec)
    sims.append(configs.dielectric_sphere(cells=60, precision=prec, probes=[((0, 0, 0), L.EZ), ((0.01, 0, 0.02), L.HX)]))
    return sims


def _results(h):
    out = [h.read_field(f) for f in FIELDS] + [h.read_probe(p) for p in range(len(h.probe_desc))]
    if h.info().n_freqs:
        out.append(h.read_nf2ff(0, 1, 2))
    return out


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("scenes,switch", [(17, None), (2, "tile"), (2, "wait")])
def test_chains_equal_alone(prec, scenes, switch):
    n = 61
    sims = _sims(prec, scenes)
    alone = []
    for s in sims:
        h = X.Handle(*s.lower())
        h.init(n)
        h.step(n)
        h.sync()
        alone.append(_results(h))
        h.close()
    hs = [X.Handle(*s.lower()) for s in sims]
    b = X.Batch(hs)
    for _ in range(2):  # and once more after a re-init
        b.init(n)
        b.step(7)
        b.sync()
        assert b.info()["launch"] == "per_step"
        hs[1].get_state()  # after an odd step count
        b.step(21)
        if switch == "tile":
            b._c(b.lib.xfb_batch_set_tile(b.b, 14))
        elif switch == "wait":
            b.set_wait_limit(1 << 20)
        b.step(n - 28)
        b.sync()
        for h, a in zip(hs, alone):
            for x, y in zip(_results(h), a):
                assert np.array_equal(x, y)
        if switch:
            b._c(b.lib.xfb_batch_set_tile(b.b, 0))
    # released in the middle, a scene continues alone
    b.init(n)
    b.step(28)
    b.sync()
    b.close()
    hs[1].step(n - 28)
    hs[1].sync()
    for x, y in zip(_results(hs[1]), alone[1]):
        assert np.array_equal(x, y)
    for h in hs:
        h.close()
