"""Performance cases of the engine: what a user's program runs, end to end.

Every case is a simulation through the package's public calls: the scene
objects lowered to a ``Handle`` (the scene compiled once, as a program keeps
it), then one pass of ``Handle.run(n)`` -- initialise, n time steps, wait --
and the read-back of the results the program is after.  The far-field case
evaluates a radiation pattern on a finished run, the batch case steps a list
of scenes together.  FP32 engines hand their results out as float64 arrays;
the cases keep them as float32, the precision they were computed in.

A case is a dict of plain values:
  kind       "run", "batch" or "pattern"
  nx ny nz   inner cells (nz = 1: 2-D TMz);   pml  CPML cells on every face
  prec       "fp32" or "fp64";                steps  time steps of a pass
  medium     scatterer: "dielectric", "lossy" (conductor + PEC), "lorentz"
             (Drude + Lorentz poles), "debye" (two poles), "pec"
  oblique    plane wave along x, or from a random direction
  freqs      NF2FF frequencies (0: no NF2FF box);  probes  point monitors
  movie      interval of a movie monitor on the middle x plane (0: none)
  td         time-domain NF2FF box
  fields     field components read back at the end (from Ez on)
  learned    learned absorbing walls instead of a CPML
  scenes, seed0   batch: number of scenes (inner sides drawn up to nx)
  angles     pattern: polar angles (twice as many azimuths)

The seed decides the scatterer (place, size, material constants), the
direction of the wave and the places of the probes.
"""
import math

import numpy as np
import torch

import xfdtd_cuda_b200 as X
from xfdtd_cuda_b200 import labc
from xfdtd_cuda_b200 import simulation as S

EPS0, MU0 = 8.854187817e-12, 4e-7 * math.pi
C0 = 1 / math.sqrt(EPS0 * MU0)
DL = 1e-3
BASE = {"kind": "run", "nx": 64, "ny": 64, "nz": 64, "pml": 8, "prec": "fp32", "steps": 100, "medium": "dielectric",
        "oblique": False, "freqs": 0, "probes": 0, "movie": 0, "td": False, "fields": 6, "learned": False, "scenes": 0,
        "angles": 0}


def _case(name, **kw):
    c = dict(BASE, **kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a first look at a coarse model, the library's default precision: set-up and launches count
        _case("coarse_fp64", nx=24, ny=20, nz=28, pml=6, prec="fp64", steps=200, freqs=1, probes=2),
        # a design sweep's inner loop: a small FP32 model run for its probe series and currents
        _case("small_fp32", nx=64, ny=56, nz=72, pml=8, steps=600, medium="lossy", oblique=True, freqs=1, probes=4),
        # the dielectric-sphere scattering scene (140^3 + 8 CPML), default precision
        _case("sphere_fp64", nx=140, ny=140, nz=140, pml=8, prec="fp64", steps=800, freqs=1, probes=4),
        # the same scene in single precision, for its currents and two components
        _case("sphere_fp32", nx=140, ny=140, nz=140, pml=8, steps=1200, freqs=1, probes=4, fields=2),
        # a box-shaped model with odd sides, lossy and PEC bodies, oblique wave, a movie and probes
        _case("ragged_fp32", nx=211, ny=97, nz=149, pml=10, steps=900, medium="lossy", oblique=True, probes=6, movie=50,
              fields=3),
        # the dispersive-sphere workload (384^3 + 12 CPML, NF2FF at three frequencies)
        _case("dispersive_fp32", nx=384, ny=384, nz=384, pml=12, steps=600, medium="lorentz", freqs=3, probes=2, fields=1),
        # two-pole Debye tissue in double precision, off-axis wave
        _case("debye_fp64", nx=108, ny=132, nz=116, pml=10, prec="fp64", steps=600, medium="debye", oblique=True, freqs=2,
              fields=3),
        # time-domain far field of a double-precision model
        _case("transient_fp64", nx=90, ny=84, nz=101, pml=8, prec="fp64", steps=600, oblique=True, td=True, probes=2,
              fields=3),
        # the 2-D cylinder (1024^2 + 10 CPML)
        _case("cylinder2d_fp32", nx=1024, ny=1024, nz=1, pml=10, steps=1600, medium="pec", probes=8, fields=1),
        # a 2-D grid of odd sides in double precision, oblique wave
        _case("ragged2d_fp64", nx=1501, ny=733, nz=1, pml=9, prec="fp64", steps=2200, medium="dielectric", oblique=True,
              probes=5, fields=3),
        # a sweep of scenes of unlike sizes stepped as one batch
        _case("batch_fp32", kind="batch", nx=160, ny=160, nz=160, pml=8, steps=500, oblique=True, scenes=10, fields=1),
        # a full radiation pattern of a finished run
        _case("pattern_fp64", kind="pattern", nx=140, ny=140, nz=140, pml=8, prec="fp64", steps=400, freqs=1, angles=180),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def steps(n, per_cell):
        """Enough for the wave to cross the model and be scattered everywhere."""
        return int((100 + per_cell * max(n)) * rng.uniform(0.95, 1.1))

    kind = rng.choice(["run"] * 6 + ["run2d"] * 3 + ["walls", "batch", "pattern"])
    prec = rng.choice(["fp32", "fp64"])
    if kind == "run2d":
        n = [side(60, 2000), side(60, 2000)]
        return _case(None, nx=n[0], ny=n[1], nz=1, pml=rng.randint(5, 14), prec=prec, steps=steps(n, 1.45),
                     medium=rng.choice(["dielectric", "pec", "lossy"]), oblique=rng.random() < 0.5,
                     probes=rng.randint(1, 8), movie=rng.choice([0, 0, 0, 50]), fields=rng.choice([1, 3]))
    if kind == "batch":
        n = side(60, 130)
        return _case(None, kind="batch", nx=n, ny=n, nz=n, pml=rng.randint(5, 10), prec=prec, steps=steps([n], 2.0),
                     oblique=rng.random() < 0.5, scenes=rng.randint(3, 10), fields=1)
    if kind == "pattern":
        n = [side(40, 140) for _ in range(3)]
        return _case(None, kind="pattern", nx=n[0], ny=n[1], nz=n[2], pml=8, prec=prec, steps=steps(n, 2.0),
                     freqs=rng.randint(1, 3), angles=rng.randint(7, 100))
    while True:
        n = [side(24, 260) for _ in range(3)]
        count = steps(n, 2.0)
        if n[0] * n[1] * n[2] * count < (8e9 if prec == "fp32" else 4e9):
            break
    walls = kind == "walls"
    medium = "dielectric" if walls else rng.choice(["dielectric", "dielectric", "lossy", "lorentz", "debye"])
    return _case(None, nx=n[0], ny=n[1], nz=n[2], pml=0 if walls else rng.randint(5, 14), prec="fp32" if walls else prec,
                 steps=count, medium=medium, oblique=rng.random() < 0.5, freqs=rng.choice([0, 1, 1, 2, 3]),
                 probes=rng.randint(0, 6), movie=rng.choice([0, 0, 0, 25]), td=rng.random() < 0.15,
                 fields=rng.choice([1, 3, 6]), learned=walls)


# ---- the scene of a case and seed, as plain numbers ---------------------------
def _scene(case, seed):
    rng = np.random.default_rng([seed, 77])
    dim = 2 if case["nz"] == 1 else 3
    n = [case["nx"], case["ny"], case["nz"]]
    size = [v * DL for v in n]
    small = min(size[:dim])
    pml = [case["pml"]] * 6 if dim == 3 else [case["pml"]] * 4 + [0, 0]
    tot = [n[a] + pml[2 * a] + pml[2 * a + 1] for a in range(3)]
    origin = [-size[a] / 2 - pml[2 * a] * DL if a < dim else 0.0 for a in range(3)]
    sc = {"dim": dim, "n": n, "size": size, "pml": pml, "tot": tot, "origin": origin, "objects": []}
    ctr = [float(rng.uniform(-0.04, 0.04)) * small if a < dim else 0.0 for a in range(3)]
    r = float(rng.uniform(0.24, 0.30)) * small
    med = case["medium"]
    plain = {"eps": 1.0, "mu": 1.0, "sig": 0.0, "pec": False, "poles": []}
    if med == "dielectric":
        m = dict(plain, eps=float(rng.uniform(2, 4)), mu=float(rng.uniform(1, 2)))
    elif med == "lossy":
        m = dict(plain, eps=float(rng.uniform(2, 8)), sig=float(rng.uniform(0.01, 0.1)))
    elif med == "lorentz":
        m = dict(plain, poles=[("drude", 2e10 * float(rng.uniform(0.9, 1.1)), 1e9),
                               ("lorentz", 2.0 * float(rng.uniform(0.8, 1.2)), 3e10, 5e8)])
    elif med == "debye":
        m = dict(plain, eps=2.0, poles=[("debye", float(rng.uniform(1, 3)), 9e-12), ("debye", 1.0, 3e-11)])
    else:
        m = dict(plain, pec=True)
    if med == "lossy" and dim == 3:  # a conducting block with a PEC ball in it
        lo = [ctr[a] - float(rng.uniform(0.12, 0.22)) * size[a] for a in range(3)]
        ext = [float(rng.uniform(0.25, 0.40)) * size[a] for a in range(3)]
        sc["objects"].append(("cube", lo + ext, m))
        sc["objects"].append(("ball", ctr + [0.4 * r], dict(plain, pec=True)))
    else:
        sc["objects"].append(("ball", ctr + [r], m))
    tau = 20 * DL / 6e8
    th, ph, ps = math.pi / 2, 0.0, 0.0
    if case["oblique"]:
        th, ph, ps = (float(rng.uniform(0.3, math.pi - 0.3)), float(rng.uniform(0, 2 * math.pi)), float(rng.uniform(0, math.pi)))
    if dim == 2:
        th, ps = math.pi / 2, 0.0
    inset = 15 if min(n[:dim]) >= 90 else 4
    if case["learned"]:
        inset = max(4, min(n) // 8)
    sc["wave"] = {"inset": inset, "theta": th, "phi": ph, "psi": ps, "tau": tau, "t0": 4.5 * tau}
    sc["freqs"] = [1e9, 3e9, 5e9][:case["freqs"]]
    sc["nf_inset"] = 11 if inset == 15 else 2
    sc["td"] = {"theta": 1.1, "phi": 0.7} if case["td"] else None
    sc["probes"] = []
    for q in range(case["probes"]):
        f = 2 if dim == 2 else q % 6
        idx = [int(rng.integers(max(1, pml[2 * a]), tot[a] - max(1, pml[2 * a + 1]))) if a < dim else 0 for a in range(3)]
        sc["probes"].append((f, idx))
    sc["movie"] = None
    if case["movie"]:  # Ez on the middle x plane
        i = tot[0] // 2
        sc["movie"] = (2, [i, 0, 0], [i + 1, tot[1] + 1, tot[2] if dim == 3 else 1], case["movie"])
    sc["fields"] = ([2, 3, 4] if dim == 2 else [2, 4, 0, 3, 1, 5])[:case["fields"]]
    return sc


def _simulation(case, sc):
    """The scene through the package's scene objects."""
    dim, size = sc["dim"], sc["size"]
    inf = math.inf
    s = S.Simulation(DL, DL, DL if dim == 3 else 1.0, 0.9, precision=case["prec"])
    lo = [-v / 2 for v in size]
    s.addObject(S.Object("domain", S.Cube(S.Vector(lo[0], lo[1], lo[2] if dim == 3 else -inf),
                                          S.Vector(size[0], size[1], size[2] if dim == 3 else inf)), S.Material.createAir()))
    for k, (shape, p, m) in enumerate(sc["objects"]):
        poles = [{"drude": S.DrudePole, "lorentz": S.LorentzPole, "debye": S.DebyePole}[q[0]](*q[1:]) for q in m["poles"]]
        mat = S.Material(f"m{k}", S.ElectroMagneticProperty(m["eps"], m["mu"], m["sig"], 0.0), pec=m["pec"], poles=poles)
        if shape == "cube":
            body = S.Cube(S.Vector(*p[:3]), S.Vector(*p[3:]))
        elif dim == 3:
            body = S.Sphere(S.Vector(*p[:3]), p[3])
        else:
            body = S.Cylinder(S.Vector(p[0], p[1], 0.0), p[3], inf, 2)
        s.addObject(S.Object(f"o{k}", body, mat))
    w = sc["wave"]
    form = S.Waveform.gaussian(w["tau"], w["t0"])
    if dim == 3:
        s.addWaveformSource(S.TFSF3D(w["inset"], w["inset"], w["inset"], w["theta"], w["phi"], w["psi"], form))
    else:
        s.addWaveformSource(S.TFSF2D(w["inset"], w["inset"], w["phi"], form))
    for d in range(2 * dim):
        if sc["pml"][d]:
            s.addBoundary(S.PML(sc["pml"][d], d))
    if sc["freqs"]:
        s.addNF2FF(S.NFFFTFrequencyDomain(sc["nf_inset"], sc["nf_inset"], sc["nf_inset"], sc["freqs"]))
    if sc["td"]:
        s.addNF2FF(S.NFFFTTimeDomain(sc["nf_inset"], sc["nf_inset"], sc["nf_inset"], "", sc["td"]["theta"], sc["td"]["phi"]))
    for f, idx in sc["probes"]:
        s.addMonitor(S.PointMonitor(S.Vector(*(sc["origin"][a] + idx[a] * (DL if a < dim else 1.0) for a in range(3))), f))
    if sc["movie"]:
        f, lo_i, hi_i, every = sc["movie"]
        s.addMonitor(S.MovieMonitor(S.FieldMonitor(S.Cube(S.Vector(0, 0, 0), S.Vector(1, 1, 1)), f), every,
                                    index_box=(lo_i, hi_i)))
    return s


def _batch_cases(case, seed):
    rng = np.random.default_rng([seed, 5, case["scenes"]])
    sizes = np.random.default_rng(case["scenes"] * 1009 + case["nx"])  # the sizes belong to the case
    out = []
    for _ in range(case["scenes"]):
        n = [int(sizes.integers(max(24, case["nx"] // 3), case["nx"] + 1)) for _ in range(3)]
        out.append((dict(case, kind="run", nx=n[0], ny=n[1], nz=n[2]), int(rng.integers(1 << 30))))
    return out


def _angles(case):
    """Polar x azimuthal grid of a pattern, the poles and the seam once."""
    th = (np.arange(case["angles"]) + 0.5) * math.pi / case["angles"]
    ph = np.arange(2 * case["angles"]) * math.pi / case["angles"]
    a, b = np.meshgrid(th, ph, indexing="ij")
    return a.ravel(), b.ravel()


def _handle(case, seed):
    sc = _scene(case, seed)
    h = X.Handle(*_simulation(case, sc).lower())
    h.set_device(0)
    return h, sc


def prepare(case, seed):
    if case["kind"] == "batch":
        hs, scs = zip(*(_handle(c, sd) for c, sd in _batch_cases(case, seed)))
        return {"case": case, "handles": hs, "scenes": scs, "batch": X.Batch(hs)}
    h, sc = _handle(case, seed)
    st = {"case": case, "handle": h, "scene": sc}
    if case["learned"]:
        st["weights"] = labc.shipped_weights()
    if case["kind"] == "pattern":
        h.run(case["steps"])
        st["angles"] = _angles(case)
    return st


def _kept(a, prec):
    """A float64 read-back in the precision it was computed in."""
    t = torch.from_numpy(a)
    return t if prec == "fp64" else t.to(torch.complex64 if t.is_complex() else torch.float32)


def run(state):
    case = state["case"]
    prec, n = case["prec"], case["steps"]
    if case["kind"] == "pattern":
        th, ph = state["angles"]
        out = [state["handle"].far_field(f, th, ph) for f in range(case["freqs"])]
        return {"pattern": [[_kept(e, prec) for e in pair] for pair in out]}
    if case["kind"] == "batch":
        b = state["batch"]
        b.init(n)
        b.step(n)
        b.sync()
        return {"fields": [_kept(h.read_field(f), prec) for h, sc in zip(state["handles"], state["scenes"]) for f in sc["fields"]]}
    h, sc = state["handle"], state["scene"]
    if case["learned"]:
        h.init(n)
        h.set_learned_abc(state["weights"])
        h.step(n)
        h.sync()
    else:
        h.run(n)
    out = {"fields": [_kept(h.read_field(f), prec) for f in sc["fields"]]}
    if sc["probes"]:
        out["probes"] = _kept(np.stack([h.read_probe(q) for q in range(len(sc["probes"]))]), prec)
    if sc["freqs"]:
        out["currents"] = [_kept(h.read_nf2ff_all(f), prec) for f in range(len(sc["freqs"]))]
    if sc["td"]:
        out["potentials"] = [_kept(h.read_nf2ff_td(w), prec) for w in range(6)]
    if sc["movie"]:
        out["movie"] = _kept(h.read_movie(0), prec)
    return out


# ---- what a pass cannot do without --------------------------------------------
def _run_work(case, seed=0):
    """Streaming one time step: every field component read and written once
    (3-D: six, 2-D: three) with a one-byte material id, the CPML memory
    variables of the slabs (two components x E and H per slab cell, 2-D one
    each), the polarisation currents of the scatterer, and per step and NF2FF
    face point the four tangential fields; then the results read once."""
    sc = _scene(case, seed)
    T = 4 if case["prec"] == "fp32" else 8
    nx, ny, nz = sc["tot"]
    cells = nx * ny * nz
    dim = sc["dim"]
    slab = sum((sc["pml"][2 * a] + sc["pml"][2 * a + 1]) * cells // sc["tot"][a] for a in range(dim))
    byt = cells * ((12 if dim == 3 else 6) * T + 1) + slab * (4 if dim == 3 else 2) * 2 * T
    flop = cells * (36 if dim == 3 else 14) + slab * (4 if dim == 3 else 2) * 5
    m = sc["objects"][0][2]
    if m["poles"]:
        ball = 4 / 3 * math.pi * (sc["objects"][0][1][3] / DL) ** 3
        state = 4 * len(m["poles"]) + 2 if case["medium"] == "lorentz" else 2 * len(m["poles"])
        byt += ball * 3 * state * T
        flop += ball * 3 * 12 * len(m["poles"])
    pts = 0
    if sc["freqs"] or sc["td"]:
        b = [sc["n"][a] - 2 * sc["nf_inset"] for a in range(3)]
        pts = 2 * (b[0] * b[1] + b[1] * b[2] + b[0] * b[2])
        byt += pts * 4 * T * (bool(sc["freqs"]) + bool(sc["td"]))
        flop += pts * (16 * len(sc["freqs"]) + 20 * bool(sc["td"]))
    byt *= case["steps"]
    flop *= case["steps"]
    byt += len(sc["fields"]) * cells * T + len(sc["freqs"]) * pts * 64
    if sc["movie"]:
        byt += (case["steps"] // case["movie"] + 1) * ny * nz * T
    return byt, flop


def work(case):
    if case["kind"] == "batch":
        parts = [_run_work(c, s) for c, s in _batch_cases(case, 0)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if case["kind"] == "pattern":
        sc = _scene(case, 0)
        b = [sc["n"][a] - 2 * sc["nf_inset"] for a in range(3)]
        pts = 2 * (b[0] * b[1] + b[1] * b[2] + b[0] * b[2])
        ang = 2 * case["angles"] ** 2
        # per frequency: the currents read, the pattern written; per point and
        # angle four complex currents times a phase, added up
        return {"bytes": case["freqs"] * (pts * 64 + ang * 48), "flops": case["freqs"] * float(pts) * ang * 32}
    byt, flop = _run_work(case)
    return {"bytes": byt, "flops": flop}


# ---- the same results in 64 bits, from plain torch -----------------------------
class _Yee:
    """The Yee scheme of a scene in float64 tensors: CPML as memory variables
    on slabs, a plane wave from a 1-D auxiliary grid, auxiliary differential
    equations for the poles.  Component arrays all have the node extents
    (nx+1, ny+1, nz+1); cells (i, j, k) < (nx, ny, nz) are updated."""

    def __init__(self, case, sc, weights=None):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.sc, self.dim, self.tot = sc, sc["dim"], sc["tot"]
        self.steps = case["steps"]
        d2 = self.dim if self.dim == 3 else 2
        self.d = [DL, DL, DL if self.dim == 3 else 1.0]
        self.dt = 0.9 / (C0 * math.sqrt(d2 / DL ** 2))
        self.f = [torch.zeros([n + 1 for n in self.tot], dtype=torch.float64, device=self.dev) for _ in range(6)]
        self.e_on = [0, 1, 2] if self.dim == 3 else [2]
        self.h_on = [3, 4, 5] if self.dim == 3 else [3, 4]
        self._materials()
        self._profiles()
        self._source()
        self.weights = None if weights is None else self._walls(weights)

    def T(self, a):
        return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=self.dev)

    def _materials(self):
        n, o = self.tot, self.sc["origin"]
        x = [(torch.arange(n[a], dtype=torch.float64, device=self.dev) + 0.5) * self.d[a] + o[a] if a < self.dim
             else torch.zeros(1, dtype=torch.float64, device=self.dev) for a in range(3)]
        gx, gy, gz = x[0][:, None, None], x[1][None, :, None], x[2][None, None, :]
        ids = torch.zeros(n, dtype=torch.uint8, device=self.dev)
        for k, (shape, p, _) in enumerate(self.sc["objects"]):
            if shape == "cube":
                inside = ((gx >= p[0]) & (gx < p[0] + p[3]) & (gy >= p[1]) & (gy < p[1] + p[4])
                          & (gz >= p[2]) & (gz < p[2] + p[5]))
            else:
                inside = (gx - p[0]) ** 2 + (gy - p[1]) ** 2 + ((gz - p[2]) ** 2 if self.dim == 3 else 0.0) <= p[3] ** 2
            ids[inside.expand(n)] = k + 1
        mats = [{"eps": 1.0, "mu": 1.0, "sig": 0.0, "pec": False, "poles": []}] + [m for _, _, m in self.sc["objects"]]
        dt = self.dt
        ce, cb, ch, db = [], [], [], []
        self.ade = None
        for k, m in enumerate(mats):
            eps, mu = EPS0 * m["eps"], MU0 * m["mu"]
            if m["pec"]:
                ce.append(0.0), cb.append(0.0)
            elif not m["poles"]:
                ce.append((2 * eps - m["sig"] * dt) / (2 * eps + m["sig"] * dt)), cb.append(2 * dt / (2 * eps + m["sig"] * dt))
            else:
                # J+ = jj J + jp J- + en E+ + e0 E + ep E-
                rec = []
                for q in m["poles"]:
                    if q[0] == "debye":
                        g = q[2] / dt + 0.5
                        b = EPS0 * q[1] / dt / g
                        rec.append(((q[2] / dt - 0.5) / g, 0.0, b, -b, 0.0))
                    else:
                        a0, b0, b1 = (q[1] ** 2, 0.0, q[2]) if q[0] == "drude" else (q[1] * q[2] ** 2, q[2] ** 2, 2 * q[3])
                        A = 1 + b1 * dt / 2
                        g = EPS0 * a0 * dt / 2 / A
                        rec.append(((2 - b0 * dt * dt) / A, (b1 * dt / 2 - 1) / A, g, 0.0, -g))
                D = eps / dt + m["sig"] / 2 + sum(r[2] for r in rec) / 2
                ce.append((eps / dt - m["sig"] / 2 - sum(r[3] for r in rec) / 2) / D), cb.append(1 / D)
                at = torch.nonzero(ids == k)
                st = self.f[0].stride()
                self.ade = {"at": at[:, 0] * st[0] + at[:, 1] * st[1] + at[:, 2], "rec": rec, "D": D,
                            "ep": -sum(r[4] for r in rec) / (2 * D)}
            ch.append(1.0), db.append(dt / mu)
        ids = ids.long()
        self.ce, self.cb, self.ch, self.db = (self.T(v)[ids] for v in (ce, cb, ch, db))
        if self.ade:
            z = torch.zeros(len(self.ade["at"]), dtype=torch.float64, device=self.dev)
            self.ade["J"] = [[[z.clone(), z.clone()] for _ in self.ade["rec"]] for _ in range(3)]
            self.ade["E"] = [z.clone() for _ in range(3)]

    def _profiles(self):
        self.psi = {}
        for a in range(self.dim):
            n, lo, hi = self.tot[a], self.sc["pml"][2 * a], self.sc["pml"][2 * a + 1]
            smax = 0.8 * 4 / (math.sqrt(MU0 / EPS0) * self.d[a])
            for kind, shift in (("e", 0.0), ("h", 0.5)):
                for side, L in ((0, lo), (1, hi)):
                    if not L:
                        continue
                    q = np.arange(0, L) if side == 0 else np.arange(n - L, n)
                    rho = (L - q - shift) / L if side == 0 else (q + shift - (n - L)) / L
                    sg, al = smax * rho ** 3, 0.05 * (1 - rho)
                    b = np.exp(-(sg + al) * self.dt / EPS0)
                    shape = [1, 1, 1]
                    shape[a] = L
                    av = np.where(sg + al > 0, sg / np.where(sg + al > 0, sg + al, 1) * (b - 1), 0.0)
                    self.psi[kind, a, side] = (int(q[0]), L, self.T(av).reshape(shape), self.T(b).reshape(shape), {})

    def _stretch(self, kind, a, comp, diff, first):
        """Adds the CPML memory of the derivative `diff` along axis a (its
        entry 0 along a is node `first`) in place."""
        for side in (0, 1):
            if (kind, a, side) not in self.psi:
                continue
            q0, L, av, bv, mem = self.psi[kind, a, side]
            skip = max(0, first - q0)
            part = diff.narrow(a, q0 + skip - first, L - skip)
            if comp not in mem:
                mem[comp] = torch.zeros_like(part)
            mem[comp].mul_(bv.narrow(a, skip, L - skip)).add_(av.narrow(a, skip, L - skip) * part)
            part.add_(mem[comp])

    def _cells(self, t, lo=(0, 0, 0), up=(0, 0, 0)):
        """View of the cells from index lo, shifted by up."""
        for a in range(3):
            t = t.narrow(a, lo[a] + up[a], self.tot[a] - lo[a])
        return t

    def half_h(self):
        for c in self.h_on:
            c -= 3
            a, b = (c + 1) % 3, (c + 2) % 3
            cur = None
            for ax, comp, sign in ((b, a, 1.0), (a, b, -1.0)):
                if comp not in self.e_on:
                    continue
                up = [int(q == ax) for q in range(3)]
                d = self._cells(self.f[comp], up=up) - self._cells(self.f[comp])
                self._stretch("h", ax, c, d, 0)
                d.mul_(sign / self.d[ax])
                cur = d if cur is None else cur.add_(d)
            self._cells(self.f[3 + c]).mul_(self.ch).add_(cur.mul_(self.db))

    def half_e(self):
        for c in self.e_on:
            a, b = (c + 1) % 3, (c + 2) % 3
            lo = [int(q in (a, b)) for q in range(3)]
            cur = None
            for ax, comp, sign in ((a, b, 1.0), (b, a, -1.0)):
                dn = [-int(q == ax) for q in range(3)]
                d = self._cells(self.f[3 + comp], lo) - self._cells(self.f[3 + comp], lo, dn)
                self._stretch("e", ax, c, d, 1)
                d.mul_(sign / self.d[ax])
                cur = d if cur is None else cur.add_(d)
            sub = [slice(v, None) for v in lo]
            F, flat = self._cells(self.f[c], lo), self.f[c].view(-1)
            if self.ade:
                old = flat[self.ade["at"]]
            F.mul_(self.ce[sub[0], sub[1], sub[2]]).add_(cur.mul_(self.cb[sub[0], sub[1], sub[2]]))
            if self.ade:
                A = self.ade
                new = flat[A["at"]] + A["ep"] * A["E"][c]
                for (jj, jp, _, _, _), (J, Jp) in zip(A["rec"], A["J"][c]):
                    new = new - ((1 + jj) * J + jp * Jp) / (2 * A["D"])
                flat[A["at"]] = new
                for q, (jj, jp, en, e0, ep) in enumerate(A["rec"]):
                    J, Jp = A["J"][c][q]
                    A["J"][c][q] = [en * new + e0 * old + ep * A["E"][c] + jj * J + jp * Jp, J]
                A["E"][c] = old

    def _source(self):
        sc, w, dt = self.sc, self.sc["wave"], self.dt
        box = []
        for a in range(3):
            box += [sc["pml"][2 * a] + w["inset"], self.tot[a] - sc["pml"][2 * a + 1] - w["inset"]] if a < self.dim else [0, 1]
        th, ph, ps = w["theta"], w["phi"], w["psi"]
        k = [math.sin(th) * math.cos(ph), math.sin(th) * math.sin(ph), math.cos(th)]
        k = [0.0 if abs(v) < 1e-6 else v for v in k]
        ratio = 1 / math.sqrt(math.sin(th) ** 4 * (math.cos(ph) ** 4 + math.sin(ph) ** 4) + math.cos(th) ** 4)
        nb = [box[2 * a + 1] - box[2 * a] for a in range(3)]
        pi, pf = [], []
        for a in range(3):
            inc = box[2 * a + (k[a] < 0)] - 2 * k[a] / ratio
            pi.append(self.T((np.arange(nb[a] + 1) + box[2 * a] - inc) * k[a] * ratio))
            pf.append(self.T((np.arange(nb[a] + 2) + box[2 * a] - inc - 0.5) * k[a] * ratio))
        nl = math.ceil(ratio * math.sqrt(float(sum(v * v for v in nb)))) + 5
        dl = DL / ratio
        ct, st, cp, sp, cs, ss = math.cos(th), math.sin(th), math.cos(ph), math.sin(ph), math.cos(ps), math.sin(ps)
        te = [ss * -sp + cs * cp * ct, ss * cp + cs * sp * ct, cs * -st]
        tr = te + [k[1] * te[2] - k[2] * te[1], k[2] * te[0] - k[0] * te[2], k[0] * te[1] - k[1] * te[0]]
        e, h = np.zeros(nl + 1), np.zeros(nl)
        rows = np.zeros((2, self.steps, nl + 1))
        abc = (C0 * dt - dl) / (C0 * dt + dl)
        for t in range(self.steps):
            rows[0, t] = e
            last = e[nl - 1], e[nl]
            h -= dt / (MU0 * dl) * (e[1:] - e[:-1])
            rows[1, t, :nl] = h
            e[1:nl] -= dt / (EPS0 * dl) * (h[1:] - h[:-1])
            e[0] = math.exp(-(((t + 1) * dt - w["t0"]) / w["tau"]) ** 2)
            e[nl] = last[0] + abc * (e[nl - 1] - last[1])
        self.rows = self.T(rows)
        # every face's corrections: (field, view, table, index, weight, scale)
        self.inject = {0: [], 3: []}
        for half in (0, 3):  # corrections of E (from incident H), of H (from incident E)
            for face in range(2 * self.dim):
                c, pos = face // 2, face % 2
                a, b = (c + 1) % 3, (c + 2) % 3
                for mine, dual in ((a, b), (b, a)):
                    if half + mine not in self.e_on + self.h_on or (3 - half) + dual not in self.e_on + self.h_on:
                        continue
                    off = (half == 0 and mine == b) or (half == 3 and mine == a)
                    lo, n = [0] * 3, [1] * 3
                    lo[c] = box[2 * c + pos]
                    for ax in (a, b):
                        lo[ax], n[ax] = box[2 * ax], nb[ax] + int((ax == a) == off)
                    shift = [0] * 3
                    if half == 3 and not pos:
                        shift[c] = -1  # H just outside the low face
                    at = [lo[q] + shift[q] for q in range(3)]
                    view = self.f[half + mine]
                    for q in range(3):
                        view = view.narrow(q, at[q], n[q])
                    proj = 0.0
                    for q in range(3):
                        s = lo[q] - (1 if half == 0 and not pos and q == c else 0) - box[2 * q]
                        halfnode = (q == dual) if half == 3 else (q != dual)
                        line = pf[q][s + 1:s + 1 + n[q]] if halfnode else pi[q][s:s + n[q]]
                        proj = proj + line.reshape([n[q] if r == q else 1 for r in range(3)])
                    if half == 0:
                        proj = proj - 0.5
                    i = proj.long()
                    sign = (1 if half == 0 else -1) * (-1 if mine == a else 1) * (1 if pos else -1)
                    coef = dt / ((EPS0 if half == 0 else MU0) * self.d[c]) * sign * tr[(3 if half == 0 else 0) + dual]
                    self.inject[half].append((view, i, proj - i.double(), coef))

    def add_source(self, half, t):
        row = self.rows[1 if half == 0 else 0, t]
        for view, i, w, coef in self.inject[half]:
            view.add_(((1 - w) * row[i] + w * row[i + 1]) * coef)

    # learned walls: y = w3 . tanh(W2 tanh(W1 x + b1) + b2) + b3 on top of Mur's boundary
    def _walls(self, w):
        w = torch.as_tensor(w).to(torch.bfloat16).double().to(self.dev)
        cut = np.cumsum([0, 512, 64, 4096, 64, 64, 1])
        p = [w[cut[q]:cut[q + 1]] for q in range(6)]
        self.hist = {}
        return p[0].reshape(64, 8), p[1], p[2].reshape(64, 64), p[3], p[4], p[5]

    def _planes(self, face, comp):
        """Wall, first and second inner plane of E's `comp`: (own axis, other axis)."""
        c = face // 2
        n, s = self.tot[c], (-1 if face % 2 else 1)
        at = n if face % 2 else 0
        out = []
        for q in range(3):
            pl = self.f[comp].select(c, at + s * q)
            rest = [v for v in range(3) if v != c]
            out.append(pl if rest[0] == comp else pl.t())
        return out

    def walls(self, old):
        W1, b1, W2, b2, w3, b3 = self.weights
        k = (C0 * self.dt - DL) / (C0 * self.dt + DL)
        todo = []
        for (face, comp), (w0, w1, w2) in old.items():
            new = self._planes(face, comp)
            nu = self.tot[comp]
            mid = slice(1, w0.shape[1] - 1)
            z = torch.zeros_like(w0[:nu, mid])
            h0, h1 = self.hist.get((face, comp), (z, z))
            e1 = w1[:nu]
            up, dn = torch.cat([e1[1:], e1[-1:]]), torch.cat([e1[:1], e1[:-1]])
            lap = up[:, mid] + dn[:, mid] + e1[:, 2:] + e1[:, :-2] - 4 * e1[:, mid]
            x = torch.stack([w0[:nu, mid], e1[:, mid], w2[:nu, mid], new[1][:nu, mid], new[2][:nu, mid], h0, h1, lap], -1)
            scale = x[..., :7].abs().amax(-1)
            y = torch.where((scale > 1e-30)[..., None], x / scale.clamp(min=1e-300)[..., None], torch.zeros_like(x))
            y = torch.tanh(torch.tanh(y @ W1.t() + b1) @ W2.t() + b2) @ w3 + b3
            out = x[..., 1] + k * (x[..., 3] - x[..., 0]) + torch.where(scale > 1e-30, scale * y, torch.zeros_like(y))
            self.hist[face, comp] = (w0[:nu, mid].clone(), e1[:, mid].clone())
            todo.append((new[0], nu, mid, out))
        for wall, nu, mid, out in todo:
            wall[:nu, mid] = out

    def step(self, t):
        old = None
        if self.weights is not None:
            old = {(f, c): [p.clone() for p in self._planes(f, c)] for f in range(6) for c in range(3) if c != f // 2}
        self.half_h()
        self.add_source(3, t)
        self.half_e()
        self.add_source(0, t)
        if old is not None:
            self.walls(old)

    def face(self, box, face):
        """Tangential (E_a, E_b, H_a, H_b) at the cell faces of one side of a box."""
        c, pos = face // 2, face % 2
        a, b = (c + 1) % 3, (c + 2) % 3

        def cut(f, **up):
            t = self.f[f]
            for q in range(3):
                s = up.get("xyz"[q], 0)
                t = t.narrow(q, box[2 * q + pos] + s, 1) if q == c else t.narrow(q, box[2 * q] + s, box[2 * q + 1] - box[2 * q])
            return t

        ax = "xyz"
        e = [0.5 * (cut(f) + cut(f, **{ax[o]: 1})) for f, o in ((a, b), (b, a))]
        h = [0.25 * (cut(3 + f) + cut(3 + f, **{ax[f]: 1}) + cut(3 + f, **{ax[c]: -1}) + cut(3 + f, **{ax[f]: 1, ax[c]: -1}))
             for f in (a, b)]
        return e + h


def _nf_box(sc):
    return [v for a in range(3) for v in (sc["pml"][2 * a] + sc["nf_inset"], sc["tot"][a] - sc["pml"][2 * a + 1] - sc["nf_inset"])]


def _face_points(sc, box, face):
    """Positions of a face's sample points: face node along the normal, cell centres across."""
    c, pos = face // 2, face % 2
    out = []
    for q in range(3):
        n = np.array([box[2 * q + pos]]) if q == c else np.arange(box[2 * q], box[2 * q + 1]) + 0.5
        out.append(sc["origin"][q] + n * DL)
    return out


def _reference(case, seed):
    sc = _scene(case, seed)
    y = _Yee(case, sc, labc.shipped_weights() if case["learned"] else None)
    n, dt, dev = case["steps"], y.dt, y.dev
    box = _nf_box(sc) if sc["freqs"] or sc["td"] else None
    cur = {}
    series = torch.zeros(len(sc["probes"]), n, dtype=torch.float64, device=dev)
    frames, td = [], None
    if sc["td"]:
        th, ph = sc["td"]["theta"], sc["td"]["phi"]
        r = [math.sin(th) * math.cos(ph), math.sin(th) * math.sin(ph), math.cos(th)]
        dist = []
        for face in range(6):
            p = _face_points(sc, box, face)
            dist.append(p[0][:, None, None] * r[0] + p[1][None, :, None] * r[1] + p[2][None, None, :] * r[2])
        far = max(v.max() for v in dist)
        delay = [(far - v) / (299792458.0 * dt) for v in dist]
        span = math.floor(max(v.max() for v in delay) + 0.5) + 3
        td = {"delay": [y.T(v) for v in delay], "pot": torch.zeros(6, n + span, dtype=torch.float64, device=dev), "prev": {}}
    for t in range(n):
        y.step(t)
        for q, (f, idx) in enumerate(sc["probes"]):
            series[q, t] = y.f[f][idx[0], idx[1], idx[2]]
        if sc["movie"] and t % sc["movie"][3] == 0:
            f, lo, hi, _ = sc["movie"]
            frames.append(y.f[f][lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]].clone())
        for face in range(6 if box else 0):
            ea, eb, ha, hb = y.face(box, face)
            s = 1.0 if face % 2 else -1.0
            a, b = (face // 2 + 1) % 3, (face // 2 + 2) % 3
            for q, fr in enumerate(sc["freqs"]):
                w = 2 * math.pi * fr
                kh, ke = (dt * complex(math.cos(w * v), -math.sin(w * v)) for v in ((t + 0.5) * dt, (t + 1.0) * dt))
                for k, (v, z) in enumerate(((-s * hb, kh), (s * ha, kh), (s * eb, ke), (-s * ea, ke))):
                    if (q, k, face) not in cur:
                        cur[q, k, face] = torch.zeros(v.shape + (2,), dtype=torch.float64, device=dev)
                    cur[q, k, face].add_(torch.stack([v * z.real, v * z.imag], -1))
            if td:
                for kind, (va, vb), off in ((3, (ea, eb), 0.5), (0, (ha, hb), 0.0)):
                    pa, pb = td["prev"].get((face, kind), (torch.zeros_like(va), torch.zeros_like(vb)))
                    td["prev"][face, kind] = (va, vb)
                    at = td["delay"][face] + off
                    i = at.floor()
                    w = at - i
                    i = (i.long() + t).reshape(-1)
                    g = (s if kind == 3 else -s) * DL * DL
                    for comp, val in ((a, g * (vb - pb)), (b, -g * (va - pa))):
                        td["pot"][kind + comp].index_add_(0, i, ((1 - w) * val).reshape(-1))
                        td["pot"][kind + comp].index_add_(0, i + 1, (w * val).reshape(-1))
    shapes = []
    for f in sc["fields"]:
        node = [[0, 1, 1], [1, 0, 1], [1, 1, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]][f]
        ext = [sc["tot"][a] + node[a] for a in range(3)]
        if sc["dim"] == 2:
            ext[2] = 1
        shapes.append(y.f[f][:ext[0], :ext[1], :ext[2]].contiguous())
    out = {"fields": shapes}
    if sc["probes"]:
        out["probes"] = series
    if sc["freqs"]:
        out["currents"] = [torch.view_as_complex(torch.stack([torch.cat([cur[q, k, f].reshape(-1, 2) for f in range(6)])
                                                              for k in range(4)])) for q in range(len(sc["freqs"]))]
    if td:
        out["potentials"] = list(td["pot"])
    if sc["movie"]:
        out["movie"] = torch.stack(frames)
    return out, sc


def _pattern(sc, cur, freq, th, ph):
    """r E_theta, r E_phi of the surface currents (e^{+jwt}, e^{-jkr} removed)."""
    box, k, eta = _nf_box(sc), 2 * math.pi * freq / C0, math.sqrt(MU0 / EPS0)
    th, ph = torch.as_tensor(th, device=cur.device), torch.as_tensor(ph, device=cur.device)
    st, ct, sp, cp = torch.sin(th), torch.cos(th), torch.sin(ph), torch.cos(ph)
    r = (st * cp, st * sp, ct)
    NL = torch.zeros(2, 3, len(th), dtype=torch.complex128, device=cur.device)
    o = 0
    for face in range(6):
        c = face // 2
        p = [torch.as_tensor(v, device=cur.device) for v in _face_points(sc, box, face)]
        size = [len(v) for v in p]
        m = size[0] * size[1] * size[2]
        ex = [torch.exp(1j * k * r[q][:, None] * p[q][None, :]) for q in range(3)]
        for w in range(4):
            comp = (c + 1 + w % 2) % 3
            s = torch.einsum("ijk,ai,aj,ak->a", cur[w, o:o + m].reshape(size), *ex)
            NL[w // 2, comp] += s * DL * DL
        o += m
    N, L = NL
    nt, npf = N[0] * ct * cp + N[1] * ct * sp - N[2] * st, -N[0] * sp + N[1] * cp
    lt, lp = L[0] * ct * cp + L[1] * ct * sp - L[2] * st, -L[0] * sp + L[1] * cp
    g = 1j * k / (4 * math.pi)
    return [-g * (lp + eta * nt), g * (lt - eta * npf)]


def exact(case, seed):
    if case["kind"] == "batch":
        return {"fields": [f for c, s in _batch_cases(case, seed) for f in _reference(c, s)[0]["fields"]]}
    out, sc = _reference(case, seed)
    if case["kind"] == "pattern":
        th, ph = _angles(case)
        return {"pattern": [_pattern(sc, out["currents"][q], f, th, ph) for q, f in enumerate(sc["freqs"])]}
    return out
