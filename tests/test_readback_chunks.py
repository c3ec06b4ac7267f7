"""Chunks of a field's staged read: 16 MB for fields of 32 MB or more, 4 MB below.
A chunk costs some 65 us beside its copy, so 4 MB chunks read a 512 MB field at
27 GB/s where 16 MB ones reach 40.  Counted by the chunks' gather kernels."""
import numpy as np
import pytest

import xfdtd_cuda_b200 as X

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.mark.parametrize("n,prec,chunk", [(90, "fp32", 4), (190, "fp64", 16), (230, "fp32", 16)])
def test_chunk_sizes(n, prec, chunk):
    torch = pytest.importorskip("torch")
    from torch.profiler import ProfilerActivity, profile
    dl = 1e-3
    s = X.Simulation(dl, dl, dl, 0.9, precision=prec)
    s.addObject(X.Object("domain", X.Cube(X.Vector(0, 0, 0), X.Vector(n * dl, n * dl, n * dl)), X.Material.createAir()))
    for d in range(6):
        s.addBoundary(X.PML(6, d))
    torch.zeros(1, device="cuda")
    h = X.Handle(*s.lower())
    h.init(20)
    r = np.random.default_rng(n)
    want = r.standard_normal(h.shape(2)).astype(np.float32).astype(np.float64)
    h.write_field(2, want)
    got = h.read_field(2)
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        h.read_field(2, got)
    h.close()
    assert np.array_equal(got, want)
    gathers = sum("k_gather_field" in e.name for e in p.events())
    nbytes = got.size * (4 if prec == "fp32" else 8)
    assert gathers == -(-nbytes // (chunk * MB)), (gathers, nbytes)
