"""Handles read from threads of their own: the staging pool has buffers for all of
them, so a round of four reads side by side takes no longer than the four one
after another and half as long again.  (Pinning a pair of buffers takes 4 ms, ten
times a small read.)"""
import threading
import time

import numpy as np
import pytest

import xfdtd_cuda_b200 as X

pytestmark = pytest.mark.gpu

THREADS, ROUNDS = 4, 12


def _handle(q):
    n, dl = 56, 1e-3
    s = X.Simulation(dl, dl, dl, 0.9, precision="fp32")
    s.addObject(X.Object("domain", X.Cube(X.Vector(0, 0, 0), X.Vector(n * dl, n * dl, n * dl)), X.Material.createAir()))
    for d in range(6):
        s.addBoundary(X.PML(6, d))
    h = X.Handle(*s.lower())
    h.init(5000)
    h.step(1)
    h.sync()
    want = np.random.default_rng(q).standard_normal(h.shape(2)).astype(np.float32).astype(np.float64)
    h.write_field(2, want)
    return h, want


def test_reads_side_by_side():
    hs, want = zip(*(_handle(q) for q in range(THREADS)))
    got = [h.read_field(2) for h in hs]

    def reads(q):
        for _ in range(ROUNDS):
            hs[q].read_field(2, got[q])

    def timed(side_by_side):
        best = 1e9
        for _ in range(5):
            th = [threading.Thread(target=reads, args=(q,)) for q in range(THREADS)]
            t0 = time.perf_counter()
            for t in th:
                t.start()
                if not side_by_side:
                    t.join()
            for t in th:
                t.join()
            best = min(best, time.perf_counter() - t0)
        return best / ROUNDS

    one_by_one, together = timed(False), timed(True)
    for a, w in zip(got, want):
        assert np.array_equal(a, w)
    for h in hs:
        h.close()
    assert together <= 1.5 * one_by_one, (together, one_by_one)
