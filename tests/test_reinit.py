"""Re-initialised handles and shared read-back staging.

A handle that is initialised again takes over the device blocks of its
previous run, and all handles read back through one pool of pinned buffers.
A run after a re-init (same length, other length, after random data was
written) must give exactly what a fresh handle gives, and reads from several
threads at once must not see one another's chunks.
"""
import threading

import numpy as np
import pytest

import xfdtd_cuda_b200 as X
from xfdtd_cuda_b200 import _lib as L
from xfdtd_cuda_b200 import configs

pytestmark = pytest.mark.gpu

FIELDS3 = (L.EX, L.EY, L.EZ, L.HX, L.HY, L.HZ)


def _handle(sim):
    return X.Handle(*sim.lower())


def _run(h, steps):
    h.init(steps)
    h.step(steps)
    h.sync()
    n = 6 if h.info().dim == 3 else 3
    fields = FIELDS3 if n == 6 else (L.EZ, L.HX, L.HY)
    return [h.read_field(f) for f in fields] + [h.read_probe(p) for p in range(len(h.probe_desc))]


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("dim", [2, 3])
def test_reinit_equals_fresh(dim, prec):
    def sim():
        return (configs.dielectric_sphere(cells=40, precision=prec, probes=[((0, 0, 0), L.EZ)]) if dim == 3
                else configs.cylinder_2d(cells=90, precision=prec, tfsf_inset=8))

    h = _handle(sim())
    first = _run(h, 50)
    rng = np.random.default_rng(3)
    for f in (L.EZ, L.HX, L.HY):
        h.write_field(f, rng.standard_normal(h.shape(f)))
    again = _run(h, 50)      # the same blocks
    longer = _run(h, 90)     # other table sizes
    h.close()
    g = _handle(sim())
    fresh = _run(g, 90)
    g.close()
    assert all(np.abs(a).max() > 0 for a in first[:3])
    assert all(np.array_equal(a, b) for a, b in zip(first, again))
    assert all(np.array_equal(a, b) for a, b in zip(longer, fresh))


def test_threads_read_through_one_pool():
    # components of about 2 chunks each (4 MB of FP64): the threads' reads overlap
    sims = [configs.dielectric_sphere(cells=c, freqs=()) for c in (84, 88, 92)]
    handles = [_handle(s) for s in sims]
    refs = []
    for h in handles:
        h.init(30)
        h.step(30)
        h.sync()
        refs.append([h.read_field(f) for f in FIELDS3])
    bad = []

    def work(h, ref):
        for _ in range(5):
            for f, a in zip(FIELDS3, ref):
                if not np.array_equal(h.read_field(f), a):
                    bad.append(f)

    ts = [threading.Thread(target=work, args=a) for a in zip(handles, refs)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for h in handles:
        h.close()
    assert not bad
