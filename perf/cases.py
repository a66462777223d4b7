"""Measured cases of the TILD step: what user programs do with this library, through the
Python binding (tild_b200.Box, tild_b200.Batch), over the sizes, boxes and options that its
benchmark workloads and tests use.

A case is one or several boxes and one call sequence on them:

  forces    set_positions, forces: a driver with its own integrator or optimiser
  run       set_positions, step(n), forces: a production run and the forces at its end
  nvt       set_positions, run_nvt(n) with logged energies, forces: a script's `run nvt`
  analysis  set_positions, thermo, structure_factor: an analysis of stored frames
  batch     set_positions of every replica, Batch.step(n), forces of every replica

A pass starts from the case's positions, so every pass steps the same physical system; what
a run leaves behind is read as the forces at its last positions (positions themselves jump
by a box length when a particle on a face rounds to the other side).  Inputs are Gaussian
random-walk chains and uniform solvent and ions at the melts' density, drawn from the seed.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "matilda.ft_b200"))
import tild_b200  # noqa: E402

RHO0 = 5.0          # particles per unit volume (per unit area of a film)
KAPPA = 25.0
SIGMA = 0.7071      # Gaussian pair kernel of two densities smeared by 0.5
DT = 0.005


def listed():
    return [
        # one force evaluation of a few short chains: the smallest call, launches and latency
        dict(name="small_forces", call="forces", system="diblock", particles=2000, chain=20, nx=16, ny=16, nz=16, order=3),
        # the plain diblock melt of 1,000 chains of 20 on 32^3: an ordinary single job
        dict(name="melt20k_run", call="run", system="diblock", particles=20000, chain=20, nx=32, ny=32, nz=32, order=3,
             steps=100),
        # a non-cubic odd box, quadratic splines, EM integrator
        dict(name="odd_box_em_run", call="run", system="diblock", particles=45360, chain=24, nx=45, ny=50, nz=63, order=2,
             steps=50, integrator="EM"),
        # a two-dimensional film with the order-4 weights
        dict(name="film2d_run", call="run", system="diblock", particles=40000, chain=16, nx=160, ny=192, nz=1, order=4,
             steps=50),
        # a replica on a grid of prime size, as the batched sweep has one
        dict(name="prime_grid_run", call="run", system="diblock", particles=124488, chain=24, nx=73, ny=73, nz=73, order=3,
             steps=20),
        # semiflexible homopolymers (one density field, angles), energies, virial and S(k) of a frame
        dict(name="semiflexible_analysis", call="analysis", system="semiflexible", particles=96000, chain=32, nx=70, ny=64,
             nz=66, order=3),
        # three species with all pair interactions, bit-reproducible deposit
        dict(name="ternary_exact_run", call="run", system="ternary", particles=200000, chain=20, nx=84, ny=84, nz=84, order=3,
             steps=20, deterministic=True),
        # a script's run with energies logged every 10 steps
        dict(name="melt300k_nvt", call="nvt", system="diblock", particles=300000, chain=24, nx=100, ny=96, nz=98, order=3,
             steps=40, log=10),
        # a served coacervate job: charges, implicit ordinary size
        dict(name="coacervate140k_run", call="run", system="coacervate", particles=140000, chain=32, nx=75, ny=75, nz=75,
             order=3, steps=50),
        # uneven diblock replicas in one batch
        dict(name="replicas_batch", call="batch", system="diblock", replicas=12, least=10000, most=300000, chain=24, order=3,
             steps=20),
        # the one-million-particle melt of the precision study, Gaussian and Erf potentials
        dict(name="melt1m_erf_run", call="run", system="erf", particles=1048576, chain=32, nx=160, ny=160, nz=160, order=3,
             steps=30),
        # the two-million-particle coacervate on 192^3, tiles from the autotuner: the largest job
        dict(name="coacervate2m_run", call="run", system="coacervate", particles=2097152, chain=32, nx=192, ny=192, nz=192,
             order=3, steps=50, autotune=True),
    ]


def draw(rng):
    call = rng.choice(["forces", "run", "run", "run", "nvt", "analysis", "batch"])
    system = rng.choice(["diblock", "diblock", "coacervate", "erf", "semiflexible", "ternary"])
    chain = rng.choice([16, 20, 24, 32])
    order = rng.choice([3, 3, 3, 2, 4, 1])
    if call == "batch":
        least = int(10.0 ** rng.uniform(4.0, 4.6))
        return dict(call=call, system="diblock", replicas=rng.randint(2, 10), least=least,
                    most=int(least * 10.0 ** rng.uniform(0.3, 1.0)), chain=chain, order=order, steps=rng.randint(5, 20))
    n = int(10.0 ** rng.uniform(3.5, 5.9 if call != "nvt" else 5.5))
    if system == "semiflexible":
        n = min(n, 300000)
    flat = system == "diblock" and rng.random() < 0.15
    side = (n / RHO0) ** (1.0 / 2.0 if flat else 1.0 / 3.0) / rng.uniform(0.36, 0.48)
    g = [max(8, int(round(side * rng.uniform(0.85, 1.18)))) for _ in range(3)]
    if flat:
        g[2] = 1
    c = dict(call=call, system=system, particles=n, chain=chain, nx=g[0], ny=g[1], nz=g[2], order=order)
    if flat and call == "analysis":
        c["call"] = "run"
    if c["call"] in ("run", "nvt"):
        c["steps"] = rng.randint(5, 40)
        if c["call"] == "nvt":
            c["log"] = rng.choice([5, 10, 20])
        if rng.random() < 0.2:
            c["integrator"] = "EM"
    if rng.random() < 0.2:
        c["deterministic"] = True
    return c


# ---- inputs ----------------------------------------------------------------------------
def smooth_size(v):
    """The nearest integer >= 8 to v whose prime factors are 2, 3, 5 and 7."""
    def ok(m):
        for f in (2, 3, 5, 7):
            while m % f == 0:
                m //= f
        return m == 1
    d = 0
    while True:
        for m in (int(round(v)) - d, int(round(v)) + d):
            if m >= 8 and ok(m):
                return m
        d += 1


def boxes_of(case):
    """The single boxes of a case: a batch's replicas have sizes spread over their range by
    the logarithm, cubic 2,3,5,7-smooth grids at a spacing of 0.4, the last one an odd grid."""
    if case["call"] != "batch":
        return [case]
    out, R = [], case["replicas"]
    for r in range(R):
        n = int(case["least"] * (case["most"] / case["least"]) ** ((r + 0.5) / R))
        g = smooth_size((n / RHO0) ** (1.0 / 3.0) / 0.4)
        if r == R - 1:
            g |= 1
        out.append(dict(case, particles=n, nx=g, ny=g, nz=g))
    return out


def gaussian(a, b, amp):
    return dict(kind="gaussian", I=a, J=b, A=float("%.9g" % amp), sigma=SIGMA)


def make_system(c, seed, replica=0):
    rng = np.random.default_rng([int(seed), replica, 7])
    dim = 2 if c["nz"] == 1 else 3
    grid = [c["nx"], c["ny"], c["nz"]][:dim]
    n, nper = c["particles"], c["chain"]
    h = (n / RHO0 / float(np.prod(grid, dtype=np.float64))) ** (1.0 / dim)
    L = np.array([float("%.9g" % np.float32(h * g)) for g in grid], np.float32)
    kind = c["system"]
    chained = {"coacervate": n // 4, "ternary": 2 * n // 3}.get(kind, n)
    nch = max(2, chained // nper)
    if kind == "coacervate":
        nch -= nch % 2
    npoly = nch * nper
    n = max(n, npoly) if kind in ("coacervate", "ternary") else npoly
    pos = rng.random((nch, nper, dim), np.float32)
    step = rng.standard_normal((nch, nper, dim), np.float32) * np.float32(1.0 / np.sqrt(3.0))
    step[:, 0] = pos[:, 0] * L
    x = np.cumsum(step, axis=1, dtype=np.float64).reshape(-1, dim)
    if n > npoly:
        x = np.concatenate([x, rng.random((n - npoly, dim)) * L.astype(np.float64)])
    x = np.mod(x, L.astype(np.float64)).astype(np.float32)
    x[x >= L] = 0.0
    i = (np.arange(nch)[:, None] * nper + np.arange(nper - 1)[None, :]).reshape(-1)
    s = dict(dim=dim, grid=grid, L=L, x=x, bonds=np.stack([i, i + 1], 1), seed=int(seed) % 100003 + 17 * replica + 1,
             order=c["order"], bond_k=1.5, q=None, angles=None, angle_k=0.0, integrator=c.get("integrator", "GJF"))
    aa = KAPPA / RHO0
    types = np.zeros(n, np.int32)
    if kind in ("diblock", "erf"):
        types = np.tile((np.arange(nper) >= nper // 2).astype(np.int32), nch)
        s["species"] = ["A", "B"]
        s["pots"] = [gaussian("A", "A", aa), gaussian("B", "B", aa), gaussian("A", "B", (KAPPA + 1.0) / RHO0)]
        if kind == "erf":
            s["pots"].append(dict(kind="erf2", I="A", J="B", A=0.01, Rp=1.0, sigma=0.5))
    elif kind == "coacervate":   # polycations and polyanions, as many counterions, neutral solvent
        q = np.zeros(n, np.float32)
        half = npoly // 2
        q[:half], q[half:npoly] = 1.0, -1.0
        ions = min(half, (n - npoly) // 2)
        q[npoly:npoly + ions], q[npoly + ions:npoly + 2 * ions] = -1.0, 1.0
        types[npoly:npoly + 2 * ions] = 1
        types[npoly + 2 * ions:] = 2
        s.update(q=q, species=["P", "C", "S"],
                 pots=[gaussian("all", "all", aa), dict(kind="charges", lB=1.0, sigma=0.5)])
        keep = np.isin([0, 1, 2], types)
        if not keep.all():   # a tiny box may lack solvent: fold the missing species away
            types = np.zeros(n, np.int32)
            s["species"] = ["P"]
    elif kind == "ternary":      # AB diblocks in a third species, every pair interacting
        types[:npoly] = np.tile((np.arange(nper) >= nper // 2).astype(np.int32), nch)
        types[npoly:] = 2
        s["species"] = ["A", "B", "C"]
        s["pots"] = [gaussian(a, b, aa if a == b else (KAPPA + 1.0) / RHO0)
                     for a, b in (("A", "A"), ("B", "B"), ("C", "C"), ("A", "B"), ("A", "C"), ("B", "C"))]
    else:                        # semiflexible homopolymers: worm-like-chain angles
        s["species"] = ["A"]
        s["pots"] = [gaussian("A", "A", aa)]
        j = (np.arange(nch)[:, None] * nper + np.arange(1, nper - 1)[None, :]).reshape(-1)
        s["angles"], s["angle_k"] = np.stack([j - 1, j, j + 1], 1), 2.0
    s["types"] = types
    return s


def make_box(s, c):
    options = {"write_files": 0}
    if c.get("deterministic"):
        options["deterministic"] = 1
    if c.get("autotune"):
        options["autotune"] = 1
    b = tild_b200.Box(0, options=options)
    b.command("Dim %d" % s["dim"])
    b.command("boxLengths " + " ".join("%.9g" % v for v in s["L"]))
    b.command("grid " + " ".join("%d" % v for v in s["grid"]))
    b.command("pmeorder %d" % s["order"])
    b.command("randSeed %d" % s["seed"])
    if s["q"] is not None:
        b.command("doCharges")
    for name in s["species"]:
        b.command("species %s mass 1 mobility 1" % name)
    b.set_particles(s["x"], s["types"], None, s["q"])
    b.command("bond 1 harmonic %.9g 0" % s["bond_k"])
    b.set_bonds(s["bonds"])
    if s["angles"] is not None:
        b.command("angle 1 wlc %.9g" % s["angle_k"])
        b.set_angles(s["angles"])
    for p in s["pots"]:
        if p["kind"] == "gaussian":
            b.command("potential gaussian %s %s %.9g %.9g" % (p["I"], p["J"], p["A"], p["sigma"]))
        elif p["kind"] == "erf2":
            b.command("potential erf2 %s %s %.9g %.9g %.9g" % (p["I"], p["J"], p["A"], p["Rp"], p["sigma"]))
        else:
            b.command("potential charges %.9g %.9g" % (p["lB"], p["sigma"]))
    b.command("integrator all %s delt %.9g" % (s["integrator"], DT))
    b.command("logFreq %d" % c.get("log", 100))
    b.command("endBox")
    return b


class State:
    def __init__(self, case, seed):
        self.case = case
        self.boxes, self.x = [], []
        for r, c in enumerate(boxes_of(case)):
            s = make_system(c, seed, r)
            self.boxes.append(make_box(s, c))
            self.x.append(s["x"])
        self.batch = None
        if case["call"] == "batch":
            self.batch = tild_b200.Batch(0)
            for b in self.boxes:
                self.batch.add(b)
        self.kmax = 0.9 * float(np.pi * min(g / l for g, l in zip(s["grid"], s["L"])))

    def __del__(self):
        if getattr(self, "batch", None) is not None:
            self.batch.close()
        for b in getattr(self, "boxes", ()):
            b.close()


SK_BINS = 48


def prepare(case, seed):
    return State(case, seed)


def run(state):
    c, call = state.case, state.case["call"]
    for b, x in zip(state.boxes, state.x):
        b.set_positions(x)
    if call == "batch":
        state.batch.step(c["steps"])
        return {"forces": [b.forces() for b in state.boxes]}
    b = state.boxes[0]
    if call == "analysis":
        thermo = b.thermo_raw()
        k, sk, count = b.structure_factor("A" if c["system"] != "coacervate" else "P", SK_BINS, state.kmax)
        return {"thermo": thermo, "k": k, "sk": sk, "count": count}
    if call == "nvt":
        b.run_nvt(c["steps"])
        rows = (c["steps"] + c["log"] - 1) // c["log"] + 2
        return {"log": b.log()[-rows:, 1:], "forces": b.forces()}
    if call == "run":
        b.step(c["steps"])
    return {"forces": b.forces()}


def work(case):
    """Bytes: a run's steps each read and write the particle state (positions, old positions,
    noise, ids, flags, bonds) once and each grid field once: the densities, and the grid
    forces of every force group; flops: the transforms, the spreading and the gather."""
    byt = flops = 0.0
    for c in boxes_of(case):
        n, m = float(c["particles"]), float(c["nx"]) * c["ny"] * c["nz"]
        d = {"semiflexible": 1, "ternary": 3}.get(c["system"], 2)
        evals = c["steps"] + (c["steps"] // c.get("log", 10 ** 9)) + 1 if "steps" in c else 1
        if c["call"] == "analysis":
            byt += n * 12 + m * 4 * (d + 1)
            flops += (d + 1) * 2.5 * m * np.log2(m) + 2.0 * n * (c["order"] + 1) ** 3
            continue
        dim = 2 if c["nz"] == 1 else 3
        byt += evals * (n * 88.0 + m * (12.0 * d + 36.0 * d)) + n * 24
        flops += evals * ((1 + dim) * d * 2.5 * m * np.log2(m) + 2.0 * n * (c["order"] + 1) ** dim * (1 + dim) * 1.5)
    return {"bytes": byt, "flops": flops}


def tolerance(case):
    # forces of one evaluation: 32-bit sums in another order; after steps: the same rounding
    # carried through the trajectory's positions (which are rounded at the box length)
    if case["call"] in ("forces", "analysis"):
        return {"rel": 4e-6, "max": 1e-4, "differ": 0.0}
    return {"rel": 1e-4, "max": 1e-2, "differ": 0.0}


# ---- the same calls in 64 bits (torch) --------------------------------------------------
def splines(x, L, n, order, dim_flat):
    """First stencil index and the order + 1 weights along one axis."""
    if dim_flat:
        return torch.zeros_like(x, dtype=torch.int64), [torch.ones_like(x)]
    d = L / n
    t = x / d
    if order % 2 == 0:
        g = torch.floor(t + 0.5)
        s = t - g
    else:
        g = torch.floor(t)
        s = t - g - 0.5
    s2 = s * s
    if order == 1:
        w = [0.5 - s, 0.5 + s]
    elif order == 2:
        w = [0.125 - 0.5 * s + 0.5 * s2, 0.75 - s2, 0.125 + 0.5 * s + 0.5 * s2]
    elif order == 3:
        s3 = s2 * s
        w = [(1 - 6 * s + 12 * s2 - 8 * s3) / 48, (23 - 30 * s - 12 * s2 + 24 * s3) / 48,
             (23 + 30 * s - 12 * s2 - 24 * s3) / 48, (1 + 6 * s + 12 * s2 + 8 * s3) / 48]
    else:   # the order-4 weights take s^4 where a quartic spline has s^3
        s4 = s2 * s2
        s3 = s4
        w = [(1 - 8 * s + 24 * s2 - 32 * s3 + 16 * s4) / 384, (19 - 44 * s + 24 * s2 + 16 * s3 - 16 * s4) / 96,
             (115 - 120 * s2 + 48 * s4) / 192, (19 + 44 * s + 24 * s2 - 16 * s3 - 16 * s4) / 96,
             (1 + 8 * s + 24 * s2 + 32 * s3 + 16 * s4) / 384]
    return g.to(torch.int64) - order // 2, w


class Exact:
    def __init__(self, s):
        self.s = s
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        f64 = dict(dtype=torch.float64, device=self.dev)
        self.dim = s["dim"]
        self.n3 = list(s["grid"]) + [1] * (3 - self.dim)
        self.L = [float(v) for v in s["L"]] + [1.0] * (3 - self.dim)
        Lf = [np.float32(v) for v in self.L]
        dx = [float(l) / n for l, n in zip(Lf, self.n3)]
        self.gvol = float(np.prod(dx))
        dxf = [np.float32(v) for v in dx]
        self.gvf = float(np.float32(np.float32(dxf[0] * dxf[1]) * dxf[2]))
        self.M = int(np.prod(self.n3))
        self.types = torch.as_tensor(s["types"], device=self.dev)
        self.q = None if s["q"] is None else torch.as_tensor(s["q"], **f64)
        self.bonds = torch.as_tensor(s["bonds"], device=self.dev)
        k = []
        for j, (n, l) in enumerate(zip(self.n3, self.L)):
            i = torch.arange(n, device=self.dev)
            i = torch.where(i < n - i, i, i - n).to(torch.float64) * (2.0 * np.pi / l)
            k.append(i.reshape([n if 2 - j == a else 1 for a in range(3)]))
        self.k = k
        self.k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
        self.groups = ["all"] + s["species"] + (["charges"] if s["q"] is not None else [])

    def member(self, name):
        if name == "all":
            return torch.ones(len(self.types), dtype=torch.float64, device=self.dev)
        if name == "charges":
            return self.q
        return (self.types == self.s["species"].index(name)).to(torch.float64)

    def shape_of(self, p):
        """u(k) and (du/dk)/k."""
        k2, f32 = self.k2, lambda v: float(np.float32(v))
        s2 = float(np.float32(np.float32(p["sigma"]) * np.float32(p["sigma"])))
        if p["kind"] == "gaussian":
            u = f32(p["A"]) * torch.exp(-0.5 * k2 * s2)
            return u, -s2 * u
        safe = torch.where(k2 > 0, k2, torch.ones_like(k2))
        if p["kind"] == "charges":
            u = torch.where(k2 > 0, 4 * np.pi * f32(p["lB"]) * torch.exp(-k2 * s2) / safe, torch.zeros_like(k2))
            return u, torch.where(k2 > 0, u * (-2.0 * s2 - 2.0 / safe), torch.zeros_like(k2))
        R, kk, A = f32(p["Rp"]), torch.sqrt(safe), f32(p["A"])
        f = torch.sin(R * kk) - R * kk * torch.cos(R * kk)
        t = 4 * np.pi * f / (safe * kk)
        dt = 4 * np.pi * (R * R * torch.sin(R * kk) / (safe * kk) - 3.0 * f / (safe * safe * kk))
        g = torch.exp(-0.5 * k2 * s2)
        u = torch.where(k2 > 0, A * g * t * t, torch.full_like(k2, A * (4 * np.pi * R ** 3 / 3) ** 2))
        return u, torch.where(k2 > 0, A * g * t * (-s2 * t + 2.0 * dt), torch.zeros_like(k2))

    def stencil(self, x):
        o = [splines(x[:, j] if j < self.dim else torch.zeros_like(x[:, 0]), self.L[j], self.n3[j], self.s["order"],
                     j >= self.dim) for j in range(3)]
        idx = [[torch.remainder(o[j][0] + a, self.n3[j]) for a in range(len(o[j][1]))] for j in range(3)]
        for e, wz in enumerate(o[2][1]):
            for b, wy in enumerate(o[1][1]):
                row, wyz = (idx[2][e] * self.n3[1] + idx[1][b]) * self.n3[0], wy * wz
                for a, wx in enumerate(o[0][1]):
                    yield row + idx[0][a], wx * wyz

    def densities(self, x, names):
        rho = {n: torch.zeros(self.M, dtype=torch.float64, device=self.dev) for n in names}
        mem = {n: self.member(n) for n in names}
        for m, w in self.stencil(x):
            for n in names:
                rho[n].index_add_(0, m, w * mem[n])
        return {n: r.reshape(self.n3[::-1]) / self.gvf for n, r in rho.items()}

    def fields(self):
        names = []
        for p in self.s["pots"]:
            for n in (("charges",) if p["kind"] == "charges" else (p["I"], p["J"])):
                if n not in names:
                    names.append(n)
        return names

    def bond_vectors(self, x, half):
        d = x[self.bonds[:, 0]] - x[self.bonds[:, 1]]
        L = torch.tensor(self.L[:self.dim], dtype=torch.float64, device=self.dev)
        return torch.where(d > half * L, d - L, torch.where(d < -half * L, d + L, d))

    def forces(self, x):
        names = self.fields()
        hat = {n: torch.fft.fftn(r) for n, r in self.densities(x, names).items()}
        phi = {n: 0.0 for n in names}
        for p in self.s["pots"]:
            u, _ = self.shape_of(p)
            if p["kind"] == "charges":
                phi["charges"] = phi["charges"] + u * hat["charges"]
            elif p["I"] == p["J"]:
                phi[p["I"]] = phi[p["I"]] + 2.0 * u * hat[p["I"]]
            else:
                phi[p["I"]] = phi[p["I"]] + u * hat[p["J"]]
                phi[p["J"]] = phi[p["J"]] + u * hat[p["I"]]
        del hat
        f = torch.zeros_like(x)
        dr = self.bond_vectors(x, 0.5)
        r2 = (dr * dr).sum(1, keepdim=True)
        fb = torch.where(r2 > 1e-4, -2.0 * self.s["bond_k"] * dr, torch.zeros_like(dr))
        f.index_add_(0, self.bonds[:, 0], fb)
        f.index_add_(0, self.bonds[:, 1], -fb)
        if self.s["angles"] is not None:
            f += self.angle_forces(x)
        grid = {n: [torch.fft.ifftn(-1j * self.k[j] * phi[n]).real.reshape(-1) * (self.gvol / self.gvf)
                    for j in range(self.dim)] for n in names}
        del phi
        mem = {n: self.member(n) for n in names}
        for m, w in self.stencil(x):
            for n in names:
                wm = w * mem[n]
                for j in range(self.dim):
                    f[:, j] += wm * grid[n][j][m]
        return f

    def angle_parts(self, x):
        a = torch.as_tensor(self.s["angles"], device=self.dev)
        L = torch.tensor(self.L[:self.dim], dtype=torch.float64, device=self.dev)
        def mi(d):
            return torch.where(d > 0.5 * L, d - L, torch.where(d < -0.5 * L, d + L, d))
        rij, rkj = mi(x[a[:, 0]] - x[a[:, 1]]), mi(x[a[:, 2]] - x[a[:, 1]])
        i2, k2 = (rij * rij).sum(1, keepdim=True), (rkj * rkj).sum(1, keepdim=True)
        ok = (i2 >= 1e-4) & (k2 >= 1e-4)
        i2, k2 = torch.where(ok, i2, torch.ones_like(i2)), torch.where(ok, k2, torch.ones_like(k2))
        m = torch.sqrt(i2 * k2)
        cos = (rij * rkj).sum(1, keepdim=True) / m
        fi = torch.where(ok, -self.s["angle_k"] * (rkj / m - cos * rij / i2), torch.zeros_like(rij))
        fk = torch.where(ok, -self.s["angle_k"] * (rij / m - cos * rkj / k2), torch.zeros_like(rij))
        return a, rij, rkj, fi, fk, torch.where(ok, self.s["angle_k"] * (1.0 + cos), torch.zeros_like(cos)).sum()

    def angle_forces(self, x):
        a, _, _, fi, fk, _ = self.angle_parts(x)
        f = torch.zeros_like(x)
        f.index_add_(0, a[:, 0], fi)
        f.index_add_(0, a[:, 1], -(fi + fk))
        f.index_add_(0, a[:, 2], fk)
        return f

    def normals(self, step):
        """Philox4x32-10 with counter (step, particle, 0, 0), Box-Muller pairs."""
        n, mask = len(self.types), 0xFFFFFFFF
        c = [torch.full((n,), step, dtype=torch.int64, device=self.dev), torch.arange(n, device=self.dev),
             torch.zeros(n, dtype=torch.int64, device=self.dev), torch.zeros(n, dtype=torch.int64, device=self.dev)]
        k0, k1 = self.s["seed"] & mask, self.s["seed"] >> 32
        for _ in range(10):
            p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
            c = [((p1 >> 32) & mask) ^ c[1] ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c[3] ^ k1, p0 & mask]
            k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
        u = [(v.to(torch.float64) + 0.5) * 2.0 ** -32 for v in c]
        r0, r1 = torch.sqrt(-2.0 * torch.log(u[0])), torch.sqrt(-2.0 * torch.log(u[2]))
        z = [r0 * torch.cos(2 * np.pi * u[1]), r0 * torch.sin(2 * np.pi * u[1]), r1 * torch.cos(2 * np.pi * u[3])]
        return torch.stack(z[:self.dim], 1)

    def walk(self, x, steps):
        """GJF (xold = x, no old noise at the start) or EM, coefficients in the 32 bits the
        integrators state them in."""
        f1 = np.float32
        dt = f1(DT)
        L = torch.tensor(self.L[:self.dim], dtype=torch.float64, device=self.dev)
        h = f1(dt / f1(f1(2) * f1(1)))
        b, a = float(f1(f1(1) / f1(f1(1) + h))), float(f1(f1(f1(1) - h) / f1(f1(1) + h)))
        mag = float(np.sqrt(f1(f1(2) * dt)))
        bd, bd2 = float(f1(f1(b) * f1(dt * dt))), float(f1(f1(f1(b) * dt) / f1(2)))
        old, n0 = x.clone(), torch.zeros_like(x)
        for t in range(steps):
            f, z = self.forces(x), self.normals(t)
            if self.s["integrator"] == "EM":
                new = x + float(dt) * f + float(f1(np.sqrt(2.0 * float(dt)))) * z
            else:
                o = torch.where(old - x > 0.5 * L, old - L, torch.where(old - x < -0.5 * L, old + L, old))
                nn = mag * z
                new = 2.0 * b * x - a * o + bd * f + bd2 * (nn + n0)
                n0 = nn
            old, x = x, torch.where(new > L, new - L, torch.where(new < 0, new + L, new))
        return x

    def thermo(self, x):
        """The values of tild_box_thermo."""
        pairs = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))
        hat = {n: torch.fft.fftn(r) / self.M for n, r in self.densities(x, self.fields()).items()}
        U, W = [], [0.0] * 6
        for p in self.s["pots"]:
            u, du = self.shape_of(p)
            I, J, fac = ("charges", "charges", 0.5) if p["kind"] == "charges" else (p["I"], p["J"], 1.0)
            re = (hat[I].conj() * hat[J]).real * (fac * self.gvol * self.M)
            U.append(float((u * re).sum()))
            for i, (a, b) in enumerate(pairs):
                W[i] += float((du * re * self.k[a] * self.k[b]).sum())
        for i in range(3):
            W[i] += sum(U)
        dr = self.bond_vectors(x, 0.25)
        r2 = (dr * dr).sum(1)
        on = r2 > 1e-4
        ub = float(torch.where(on, self.s["bond_k"] * r2, torch.zeros_like(r2)).sum())
        mf = torch.where(on, torch.full_like(r2, -2.0 * self.s["bond_k"]), torch.zeros_like(r2))
        B = [float((mf * dr[:, a] * dr[:, b]).sum()) for a, b in pairs]
        ua = 0.0
        if self.s["angles"] is not None:
            _, rij, rkj, fi, fk, e = self.angle_parts(x)
            ua = float(e)
            B = [v + float((fi[:, a] * rij[:, b] + fk[:, a] * rkj[:, b]).sum()) for v, (a, b) in zip(B, pairs)]
        V = self.L[0] * self.L[1] * self.L[2]
        P = [((len(self.types) if i < 3 else 0) + W[i] + B[i]) / V for i in range(6)]
        return np.array([ub + ua + sum(U), ub] + U + B + W + P + [ua])

    def structure(self, x, name, kmax):
        s = torch.fft.fftn(self.densities(x, [name])[name]) / self.M
        s = (s.real ** 2 + s.imag ** 2).reshape(-1)
        k = torch.sqrt(self.k2).expand(self.n3[::-1]).reshape(-1)
        bin_ = torch.floor(k * (SK_BINS / kmax)).to(torch.int64)
        on = bin_ < SK_BINS
        tot = [torch.bincount(bin_[on], weights=v, minlength=SK_BINS).cpu().numpy()
               for v in (k[on], s[on], torch.ones_like(k[on]))]
        some = tot[2] > 0
        cnt = np.maximum(tot[2], 1.0)
        mid = (np.arange(SK_BINS) + 0.5) * kmax / SK_BINS
        return np.where(some, tot[0] / cnt, mid), np.where(some, tot[1] / cnt, 0.0), tot[2]


def exact(case, seed):
    cost = sum(float(c["particles"]) * c.get("steps", 1) for c in boxes_of(case))
    if cost > 4.0e7:
        return None
    got = []
    for r, c in enumerate(boxes_of(case)):
        s = make_system(c, seed, r)
        e = Exact(s)
        x = torch.as_tensor(s["x"], dtype=torch.float64, device=e.dev)
        if case["call"] == "analysis":
            kmax = 0.9 * float(np.pi * min(g / l for g, l in zip(s["grid"], s["L"])))
            k, sk, _ = e.structure(x, "A" if case["system"] != "coacervate" else "P", kmax)
            # the shells' counts may differ by a k-vector on a shell's edge
            return {"thermo": e.thermo(x), "k": k, "sk": sk, "count": None}
        if case["call"] != "forces":
            x = e.walk(x, case["steps"])
        got.append(e.forces(x).cpu().numpy())
    if case["call"] == "batch":
        return {"forces": got}
    return {"log": None, "forces": got[0]} if case["call"] == "nvt" else {"forces": got[0]}
