"""Rounding of the far field: a call for many directions (k_far_many, phases as
row and column products) is as close to the 80-bit integral of the same surface
currents as calls for few (k_far, a phase per point).  FP64 currents of a
scattering run on box shapes whose rows, columns or faces are few or many, from
long waves to ten cells a wave.

The bound: over all shapes, frequencies and both polarisations the root mean
square of the relative errors is no larger than that of the few-direction
calls."""
import math

import numpy as np
import pytest

import xfdtd_cuda_b200 as X
from xfdtd_cuda_b200 import simulation as S

pytestmark = pytest.mark.gpu

DL = 1e-3
FREQS = (1e9, 3e9, 5e9, 12e9, 30e9)
LD, CLD = np.longdouble, np.clongdouble
EPS0, MU0 = 8.854187817e-12, 4.0 * 3.14159265358979323846 * 1e-7


def far_field_80bit(cur, box, origin, d, freq, theta, phi):
    """E_theta, E_phi of the currents [4, points], as far_field_numpy, in long double."""
    k = LD(2 * math.pi * freq / (1.0 / math.sqrt(EPS0 * MU0)))
    eta = LD(math.sqrt(MU0 / EPS0))
    th, ph = theta.astype(LD), phi.astype(LD)
    st, ct, sp, cp = np.sin(th), np.cos(th), np.sin(ph), np.cos(ph)
    r = [st * cp, st * sp, ct]
    N, M = np.zeros((len(th), 3), CLD), np.zeros((len(th), 3), CLD)
    o = 0
    for face in range(6):
        ax, pos = face // 2, face % 2
        n = [box[2 * a + 1] - box[2 * a] if a != ax else 1 for a in range(3)]
        ph3 = []
        ds = LD(1)
        for a in range(3):
            x = LD(origin[a]) + (box[2 * a + (pos if a == ax else 0)] + np.arange(n[a]) + (LD(0.5) if a != ax else 0)) * LD(d[a])
            p = k * np.outer(r[a], x)
            ph3.append(np.cos(p) + 1j * np.sin(p))
            ds = ds * LD(d[a]) if a != ax else ds
        m = n[0] * n[1] * n[2]
        c = cur[:, o:o + m].reshape(4, *n).astype(CLD)
        o += m
        sums = []
        for w in range(4):
            v = np.tensordot(ph3[2], c[w], axes=([1], [2]))
            sums.append(((v * ph3[0][:, :, None]).sum(1) * ph3[1]).sum(1) * ds)
        ca, cb = ((1, 2), (2, 0), (0, 1))[ax]
        N[:, ca] += sums[0]
        N[:, cb] += sums[1]
        M[:, ca] += sums[2]
        M[:, cb] += sums[3]
    n_th, n_ph = N[:, 0] * ct * cp + N[:, 1] * ct * sp - N[:, 2] * st, -N[:, 0] * sp + N[:, 1] * cp
    l_th, l_ph = M[:, 0] * ct * cp + M[:, 1] * ct * sp - M[:, 2] * st, -M[:, 0] * sp + M[:, 1] * cp
    f = k / (4 * LD(math.pi))
    return -1j * f * (l_ph + eta * n_th), 1j * f * (l_th - eta * n_ph)


def test_many_directions_as_close_as_few():
    few_all, many_all = [], []
    for n in ((44, 44, 44), (90, 60, 40), (30, 110, 20), (12, 12, 120)):
        s = S.Simulation(DL, DL, DL, 0.9, precision="fp64")
        lo = [-v * DL / 2 for v in n]
        s.addObject(S.Object("domain", S.Cube(S.Vector(*lo), S.Vector(*(v * DL for v in n))), S.Material.createAir()))
        s.addObject(S.Object("ball", S.Sphere(S.Vector(0.1 * DL, 0, 0), 0.2 * min(n) * DL),
                             S.Material("m", S.ElectroMagneticProperty(3.0, 1.0, 0.0, 0.0))))
        s.addWaveformSource(S.TFSF3D(4, 4, 4, 1.0, 0.5, 0.3, S.Waveform.gaussian(20 * DL / 6e8, 60 * DL / 6e8)))
        for f in range(6):
            s.addBoundary(S.PML(6, f))
        s.addNF2FF(S.NFFFTFrequencyDomain(2, 2, 2, list(FREQS)))
        h = X.Handle(*s.lower())
        h.run(200)
        gi = h.info()
        for q, freq in enumerate(FREQS):
            rng = np.random.default_rng(q)
            th, ph = rng.uniform(0, math.pi, 128), rng.uniform(0, 2 * math.pi, 128)
            want = far_field_80bit(h.read_nf2ff_all(q), list(gi.nf2ff_box), list(gi.origin), (gi.dx, gi.dy, gi.dz), freq, th, ph)
            few = h.far_field(q, th, ph)
            many = [e[:128] for e in h.far_field(q, np.tile(th, 256), np.tile(ph, 256))]
            for out, got in ((few_all, few), (many_all, many)):
                out += [float(np.linalg.norm(g.astype(CLD) - w) / np.linalg.norm(w)) for g, w in zip(got, want)]
        h.close()
    few_rms, many_rms = (math.sqrt(np.mean(np.square(v))) for v in (few_all, many_all))
    assert 0 < few_rms < 1e-13
    assert many_rms <= few_rms, (many_rms, few_rms)
    # and at no wavelength alone
    ratios = np.array(many_all).reshape(-1, len(FREQS), 2) / np.array(few_all).reshape(-1, len(FREQS), 2)
    assert (np.sqrt((ratios ** 2).mean(axis=(0, 2))) <= 1.0).all(), ratios.tolist()
