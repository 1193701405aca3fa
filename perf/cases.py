"""What a program asks of this package, as cases that can be timed: the time
loop of the reference's small configurations and of full 6D fields in both
precisions, the host-array drop-in call, the energy budget, the set-up of a
field, and the batched ensemble.  Each case goes through the public entry
points (Model, Batch); the inputs are made from the seed alone.
"""
import math

import numpy as np
import torch

PAD = 2                  # ghost cells on both sides of every axis
AXES = "xyzklm"
CFL = 0.4


def _case(name, use, form, schedule, n, steps, **more):
    c = {"name": name, "use": use, "form": form, "schedule": schedule, "steps": steps,
         "grid": "uniform", "walls": "reflect", "force": "none", "start": "packet"}
    c.update(zip(("nx", "ny", "nz", "nk", "nl", "nm"), n))
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: one step of a test-sized field through the literal drop-in for the module-state
        # subroutine (upload, step, download)
        _case("tiny_host_step", "host", "fp64", "default", (6, 5, 6, 4, 4, 6), 1),
        # the reference's 1D set-up (test1D, fac = 2: a column of z and m), stepped between two looks at the state
        _case("column_1d", "integrate", "fp64", "default", (1, 1, 40, 1, 1, 120), 50),
        # its forced column (critical_gm1, fac = 1): the bottom plane relaxes to a spectrum before every step
        _case("forced_column", "integrate", "fp64", "default", (1, 1, 160, 1, 1, 300), 20, force="relax",
              walls="open"),
        # its 2D section (test2D, fac = 1)
        _case("section_2d", "integrate", "fp64", "default", (1, 10, 20, 1, 60, 60), 20),
        # the 6D packet 8x8x16 x 16^3 as it runs without any tuning: the reference's arithmetic bit for bit
        _case("packet_exact", "integrate", "fp64", "default", (8, 8, 16, 16, 16, 16), 10),
        # the same packet at a snapshot: one step, then the budget and the wavenumber integrals
        _case("packet_budget", "diagnose", "fp64", "default", (8, 8, 16, 16, 16, 16), 1),
        # a field whose extents divide nothing, on stretched grids, with the fast binary64 schedule
        _case("ragged_fp64", "integrate", "fp64", "fast", (18, 14, 20, 10, 12, 14), 10, grid="stretched",
              walls="open"),
        # the headline workload's physics (32 x 32 x 32 in space, log-normal spectrum, mean flow) in binary64
        _case("jet_fp64", "integrate", "fp64", "fast", (32, 32, 32, 12, 12, 12), 10, start="spectrum"),
        # and in binary32
        _case("jet_fp32", "integrate", "fp32", "w2q", (32, 32, 32, 12, 16, 12), 20, start="spectrum"),
        # a binary32 field of ragged extents as it runs without any tuning
        _case("ragged_fp32", "integrate", "fp32", "default", (30, 18, 20, 14, 10, 12), 10, grid="stretched"),
        # an ensemble of independent binary32 fields of different sizes, batched
        _case("ensemble_fp32", "ensemble", "fp32", "default", (0, 0, 0, 0, 0, 0), 32, members=10, shapes=5),
        # a request arrives: coefficients, time step and state of a binary32 member, and its first step
        _case("admission_fp32", "setup", "fp32", "default", (24, 24, 24, 12, 12, 16), 1),
    ]


def _even(rng, lo, hi):
    return 2 * max(1, round(0.5 * math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _any(rng, lo, hi):
    return round(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["host", "column", "section", "exact", "budget", "fast", "fp32", "fp32", "ensemble", "setup"])
    grid = rng.choice(["uniform", "stretched"])
    walls = rng.choice(["reflect", "open"])
    start = rng.choice(["packet", "packet", "spectrum"])
    more = dict(grid=grid, walls=walls, start=start)

    def six(lo, hi, klo, khi, cells):
        while True:
            n = tuple(_any(rng, lo, hi) for _ in range(3)) + tuple(_even(rng, klo, khi) for _ in range(3))
            if np.prod(n) <= cells:
                return n
    if kind == "host":
        c = _case("", "host", "fp64", "default", six(5, 12, 4, 10, 2e5), 1, **more)
    elif kind == "column":
        more["force"] = rng.choice(["none", "flux", "relax"])
        c = _case("", "integrate", "fp64", "default", (1, 1, _any(rng, 20, 200), 1, 1, _even(rng, 40, 300)),
                  rng.randint(10, 60), **more)
    elif kind == "section":
        c = _case("", "integrate", "fp64", "default",
                  (1, _any(rng, 6, 24), _any(rng, 10, 40), 1, _even(rng, 16, 64), _even(rng, 16, 64)),
                  rng.randint(5, 20), **more)
    elif kind == "exact":
        c = _case("", "integrate", "fp64", "default", six(5, 20, 4, 18, 6e6), rng.randint(4, 10), **more)
    elif kind == "budget":
        c = _case("", "diagnose", "fp64", "default", six(5, 20, 4, 18, 6e6), 1, **more)
    elif kind == "fast":
        c = _case("", "integrate", "fp64", "fast", six(8, 32, 6, 16, 3e7), rng.randint(4, 10), **more)
    elif kind == "fp32":
        n = six(8, 32, 6, 18, 4e7)
        n = (n[0] // 2 * 2,) + n[1:]
        sched = "w2q" if n[0] * n[1] % 4 == 0 and n[0] * n[1] >= 256 and rng.random() < 0.6 else "default"
        c = _case("", "integrate", "fp32", sched, n, rng.randint(8, 20), **more)
    elif kind == "ensemble":
        c = _case("", "ensemble", "fp32", "default", (0,) * 6, rng.randint(16, 28), members=rng.randint(4, 8),
                  shapes=rng.randint(0, 10 ** 6))
    else:
        c = _case("", "setup", "fp32", "default", six(8, 28, 6, 16, 3e7), 1, **more)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs: plain arrays, from the case and the seed
# ---------------------------------------------------------------------------
def _shapes(case):
    """the extents of the case's fields (an ensemble has several)"""
    if case["use"] != "ensemble":
        return [tuple(int(case["n" + a]) for a in AXES)]
    g = np.random.Generator(np.random.PCG64(case["shapes"]))
    return [tuple(int(g.choice((8, 16, 24, 32))) for _ in range(3)) + tuple(int(g.choice((8, 12, 16))) for _ in range(3))
            for _ in range(case["members"])]


def _spacings(n, stretched):
    """interior spacings; uniform ones are exact in binary so that the sums of the grid set-up are too"""
    d = []
    for a, k in enumerate(n):
        base = (5000.0, 5000.0, math.floor(8 * 4000.0 / k) / 8, 4e-3 / k, 4e-3 / k, 0.1 / k)[a]
        w = np.ones(k)
        if stretched and k >= 8:
            i = np.arange(k)
            if a in (0, 1):
                w = 1.0 + 0.3 * np.sin(1.7 * i + 0.4)
            elif a == 2:                                  # refined upwards
                w = 1.0 - 0.5 * (i / (k - 1)) ** 2
            else:                                         # refined towards zero and mirrored
                j = np.arange(k // 2) / (k // 2 - 1)
                h = 1.0 - 0.5 * j ** 2
                w = np.concatenate([h, h[::-1]])
        d.append(base * w)
    return d


def _padded(v):
    return np.concatenate([np.full(PAD, v[0]), v, np.full(PAD, v[-1])])


def _centres(d, fixed):
    """padded cell centres of a spectral axis: the reference's recursion, centred on the middle face"""
    if len(d) == 1:
        return np.full(1 + 2 * PAD, fixed)
    p = _padded(d)
    u = np.concatenate([[0.0], np.cumsum(p[1:])])
    t = np.empty_like(p)
    t[0] = u[0] - 0.5 * p[0]
    for i in range(1, len(p)):
        t[i] = 2 * u[i - 1] - t[i - 1]
    return t - u[len(d) // 2 + PAD - 1]


FIXED = (1e-3, 0.0, 0.0)   # wavenumbers of collapsed spectral axes


def _inputs(case, n, rng):
    """grid, background (padded 3D), state (interior) and forcing of one field"""
    d = _spacings(n, case["grid"] == "stretched")
    x, y, z = (np.cumsum(_padded(d[a])) - np.sum(d[a][:1]) * 2.5 for a in range(3))
    X, Y, Z = np.meshgrid(x, y, z - np.sum(d[2]), indexing="ij")
    Lx, Ly = np.sum(d[0]), np.sum(d[1])
    amp = 0.08 + 0.08 * rng.random()
    Nsqr = (5e-3 * np.exp(Z / 2000.0)) ** 2 * (1 + 0.05 * rng.random() * np.cos(2 * np.pi * X / Lx))
    U = amp * (0.4 + np.sin(2 * np.pi * Y / Ly)) * np.exp(Z / 800.0)
    V = 0.3 * amp * np.cos(2 * np.pi * X / Lx) * np.exp(Z / 1200.0)
    # a spatial times a spectral factor, Fortran order: (x,y,z) fastest
    space, spec = np.ones(1), np.full(1, 1e-3)
    if case["start"] == "spectrum":                       # log-normal in (k,l,m), uniform in space
        space = np.ones(np.prod(n[:3]))
        spec = spec * np.exp(0.5 * rng.standard_normal(np.prod(n[3:])))
    else:                                                 # Gaussian packet over a little noise
        for a in range(6):
            c = (0.5 if a < 3 else 0.6) * n[a] + rng.random()
            g = np.exp(-0.5 * ((np.arange(n[a]) - c) / max(2.0, 0.12 * n[a])) ** 2) if n[a] > 1 else np.ones(1)
            if a < 3:
                space = np.outer(g, space).ravel()
            else:
                spec = np.outer(g, spec).ravel()
    dtype = np.float32 if case["form"] == "fp32" else np.float64
    E = np.multiply.outer(spec.astype(dtype), space.astype(dtype))
    if case["start"] != "spectrum":
        for q in range(len(spec)):
            E[q] += dtype(1e-6 * rng.random()) * (dtype(1) + np.roll(space, 7 * q).astype(dtype))
    E = E.reshape(n[::-1]).T
    force = None
    if case["force"] != "none":
        F = np.zeros(tuple(n[a] + 2 * PAD for a in (0, 1, 3, 4, 5)), order="F")
        F[(slice(PAD, -PAD),) * 5] = (1e-3 if case["force"] == "relax" else 1e-7) * (0.5 + rng.random((n[0], n[1]) + n[3:]))
        force = (case["force"], F)
    return {"n": n, "d": d, "Nsqr": Nsqr, "U": U, "V": V, "E": E, "force": force, "f0": 1e-4,
            "reflect": case["walls"] == "reflect"}


def _fields(case, seed):
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    return [_inputs(case, n, rng) for n in _shapes(case)]


# ---------------------------------------------------------------------------
# the program
# ---------------------------------------------------------------------------
def _model(case, i):
    from raytracer_3d_gb300.model import Model
    # binary32 callers keep no padded module array: the state moves as the interior in the form's precision
    m = Model(*i["n"], dt=1.0, f0=i["f0"], enable_upper_reflection=i["reflect"], enable_lower_reflection=i["reflect"],
              precision=case["form"], k_fixed=FIXED[0], l_fixed=FIXED[1], m_fixed=FIXED[2], padded=case["form"] == "fp64")
    m.calc_grid(i["d"])
    m.Nsqr[:], m.U[:], m.V[:] = i["Nsqr"], i["U"], i["V"]
    if m.padded:
        m.E[(slice(PAD, -PAD),) * 6] = i["E"]
    else:
        m.E = np.asfortranarray(i["E"])
    m.calc_parameter()
    m.set_dt(CFL / m.max_rate())
    if i["force"]:
        m.set_forcing(*i["force"])
    if case["schedule"] == "fast":
        m.set_tuning("fast", 8, 256)
    elif case["schedule"] == "w2q":
        m.set_tuning("w2q", 4, 512, 1)
    m.set_state()
    return m


def prepare(case, seed):
    models = [_model(case, i) for i in _fields(case, seed)]
    if case["use"] == "ensemble":
        from raytracer_3d_gb300.batch import Batch
        return {"case": case, "models": models, "batch": Batch(models)}
    return {"case": case, "models": models}


def run(state):
    case, m = state["case"], state["models"][0]
    inner = (slice(PAD, -PAD),) * 6
    if case["use"] == "host":
        m.integrate_host()
        return m.E[inner]
    if case["use"] == "integrate":
        m.integrate(case["steps"])
        E = m.get_state()
        return E[inner] if m.padded else E
    if case["use"] == "diagnose":
        m.integrate(case["steps"])
        b, fields = m.diagnose()
        return {"sums": np.array([b["eint"], b["mflint"]]), "mfl_max": b["mfl_max"],
                "bfl": np.array([b["bfl_%s%s" % (a, e)] for a in AXES for e in "se"]),
                "vmax": [b[k] for k in ("umax", "vmax", "wmax", "kmax", "lmax", "mmax")],
                "cfl": np.array([b["cfl_" + a] for a in AXES]),
                "fields": {k: v[inner[:3]] for k, v in fields.items()}}
    if case["use"] == "setup":
        m.calc_parameter()
        rate = m.max_rate()
        m.set_dt(CFL / rate)
        m.set_state()
        m.integrate(case["steps"])
        return {"rate": rate, "E": m.get_state()}
    state["batch"].integrate(case["steps"])
    return [x.get_state() for x in state["models"]]


def work(case):
    size = 8 if case["form"] == "fp64" else 4
    b = f = 0.0
    for n in _shapes(case):
        cells = float(np.prod(n))
        act = sum(k > 1 for k in n)
        # a step reads and writes E and reads a velocity per active axis and the growth rate; then the state goes out
        b += cells * size * (case["steps"] * (3 + act) + 1)
        f += cells * case["steps"] * (14.0 * act + 4)
        if case["use"] == "host":
            b += cells * 8
        if case["use"] == "diagnose":                     # the step's inputs and its result once more
            b += cells * size * (3 + act) - cells * size
            f += cells * (14.0 * act + 20)
        if case["use"] == "setup":                        # velocities and rate written, the state read
            b += cells * size * (act + 2)
            f += cells * 60.0
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same, as the scheme's formulas in 64 bits
# ---------------------------------------------------------------------------
class _Plain:
    """Dispersion relation, velocities, limited fluxes and budget on plain
    tensors; axis a of the field is dimension 5 - a."""

    def __init__(self, i):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.n, self.reflect = i["n"], i["reflect"]
        self.d = [self.t(_padded(v)) for v in i["d"]]
        self.E = self.t(np.asarray(i["E"], dtype=np.float64).T)
        self.force = i["force"]
        kw = [self.t(_centres(i["d"][3 + c], FIXED[c])) for c in range(3)]
        bg = [self.t(i[k].T) for k in ("Nsqr", "U", "V")]
        f2 = i["f0"] * i["f0"]
        n = self.n

        def spec(v, a):
            return v.reshape([-1 if b == a else 1 for b in (5, 4, 3, 2, 1, 0)])

        def cut(v, a, lo, hi):
            """Fortran indices lo..hi of axis a of a padded tensor (broadcast axes stay)"""
            dim = v.dim() - 1 - a
            return v if v.shape[dim] == 1 else v.narrow(dim, lo + PAD - 1, hi - lo + 1)

        k, l, m = (spec(kw[c], 3 + c) for c in range(3))
        N2, U, V = (v.reshape((1, 1, 1) + tuple(v.shape)) for v in bg)

        def omega(ranges):
            """(omega_i, omega_e) on the given Fortran index range of every axis"""
            K, L, M = (cut(v, a, *ranges[a]) for v, a in ((k, 3), (l, 4), (m, 5)))
            c = [v for v in (N2, U, V)]
            for a in range(3):
                c = [cut(v, a, *ranges[a]) for v in c]
            kh2, m2 = L * L + K * K, M * M
            oi = torch.sqrt((c[0] * kh2 + f2 * m2) / (m2 + kh2))
            return oi, oi + K * c[1] + L * c[2]

        inside = [(1, q) for q in n]
        self.v = []
        for a in range(6):
            s, w = a % 3, a % 3 + 3
            shape = [n[b] + (b == a) for b in (5, 4, 3, 2, 1, 0)]
            if s < 2 and not (n[s] > 1 and n[w] > 1):
                v = torch.zeros(shape, dtype=torch.float64, device=self.dev)
                if a < 3:
                    oi, _ = omega(inside)
                    K, L, M = (cut(q, b, 1, n[b]) for q, b in ((k, 3), (l, 4), (m, 5)))
                    c = [N2, U, V]
                    for b in range(3):
                        c = [cut(q, b, 1, n[b]) for q in c]
                    kh2, m2 = L * L + K * K, M * M
                    g = (c[0] - f2) / oi * m2 / (m2 + kh2) ** 2
                    v.narrow(5 - a, 1, n[a]).copy_(c[1 + s] + g * (K if s == 0 else L))
                self.v.append(v)
                continue
            r = list(inside)
            r[a] = (0, n[a])
            if a < 3:                                     # centred difference over the wavenumber
                hi, lo = list(r), list(r)
                hi[w], lo[w] = (2, n[w] + 1), (0, n[w] - 1)
                v = 0.5 * (omega(hi)[1] - omega(lo)[1]) / spec(self.d[w][PAD:-PAD], w)
            else:                                         # refraction: difference over the spatial partner
                hi, lo = list(r), list(r)
                hi[a], lo[a] = (1, n[a] + 1), (1, n[a] + 1)
                h1, l1 = list(r), list(r)
                h0, l0 = list(r), list(r)
                h1[a], h0[a] = (1, n[a] + 1), (0, n[a])
                l1[a], l0[a] = (1, n[a] + 1), (0, n[a])
                l1[s] = l0[s] = (0, n[s] - 1)
                v = -0.5 * ((omega(h1)[1] + omega(h0)[1]) - (omega(l1)[1] + omega(l0)[1])) / spec(self.d[s][PAD:-PAD], s)
            v = v.expand(shape).contiguous()
            first, last = v.narrow(5 - a, 0, 1), v.narrow(5 - a, n[a], 1)
            if a != 2 or not self.reflect:                # open ends let energy out only
                last.clamp_(min=0.0)
                first.clamp_(max=0.0)
            self.v.append(v)
        oi, _ = omega(inside)
        right = [self.v[a].narrow(5 - a, 1, n[a]) for a in range(3)]
        Ui, Vi = U, V
        for b in range(3):
            Ui, Vi = cut(Ui, b, 1, n[b]), cut(Vi, b, 1, n[b])

        def slope(F, a):
            for b in range(3):
                F = F if b == a else cut(F, b, 1, n[b])
            return (cut(F, a, 2, n[a] + 1) - cut(F, a, 0, n[a] - 1)) / (2 * spec(self.d[a][PAD:-PAD], a))

        K, L = cut(k, 3, 1, n[3]), cut(l, 4, 1, n[4])
        rate = 0.0
        for a, wn in ((0, K), (1, L)):
            if n[a] > 1:
                rate = rate + wn / oi * ((right[0] - Ui) * slope(U, a) + (right[1] - Vi) * slope(V, a))
        if n[2] > 1:
            rate = rate + right[2] / oi * (K * slope(U, 2) + L * slope(V, 2))
        self.rate = rate
        total = 0.0
        for a in range(6):
            if n[a] > 1:
                v = self.v[a].abs()
                total = total + torch.maximum(v.narrow(5 - a, 0, n[a]), v.narrow(5 - a, 1, n[a])) / spec(
                    self.d[a][PAD:-PAD], a)
        self.max_rate = float(total.max())
        self.dt = CFL / self.max_rate
        self.spec = spec

    def t(self, v):
        return torch.from_numpy(np.ascontiguousarray(v)).to(self.dev)

    def flux(self, a):
        """faces 0..n of axis a"""
        n, E, dim = self.n[a], self.E, 5 - a
        if a == 2 and self.reflect:                       # mirrored in z and m
            low = E.narrow(dim, 0, 2).flip(dim, 0)
            top = E.narrow(dim, n - 2, 2).flip(dim, 0)
        else:
            low, top = E.narrow(dim, 0, 1), E.narrow(dim, n - 1, 1)
            low, top = torch.cat([low, low], dim), torch.cat([top, top], dim)
        P = torch.cat([low, E, top], dim)
        Ea, Eb, Ec, Ed = (P.narrow(dim, q, n + 1) for q in range(4))
        v = self.v[a]
        u = (v * self.dt).abs() / self.spec(self.d[a][PAD - 1:-PAD], a)
        Rj = Ec - Eb
        r = torch.where(v > 0, Eb - Ea, Ed - Ec)
        r = torch.where(Rj != 0, r / torch.where(Rj != 0, Rj, torch.ones_like(Rj)), r * 1e20)
        r = torch.maximum(torch.minimum(2 * r, torch.ones_like(r)), r.clamp(max=2.0)).clamp(min=0.0)
        return v * (Ec + Eb) * 0.5 - v.abs() * ((1 - r) + u * r) * Rj * 0.5

    def step(self, keep=None):
        if self.force:
            kind, F = self.force
            F = self.t(F[(slice(PAD, -PAD),) * 5].T)
            bottom, dz = self.E.select(3, 0), self.d[2][PAD]
            if kind == "flux":
                bottom += self.dt * F / dz
            else:
                bottom -= self.dt * self.v[2].select(3, 1).clamp(min=0.0) * (bottom - F) / dz
        mf = self.E * self.rate
        dE = -mf
        for a in range(6):
            n = self.n[a]
            if n > 1:
                f = self.flux(a)
                dE = dE - (f.narrow(5 - a, 1, n) - f.narrow(5 - a, 0, n)) / self.spec(self.d[a][PAD:-PAD], a)
                if keep is not None:
                    keep[a] = (f.narrow(5 - a, 0, 1), f.narrow(5 - a, n, 1))
        self.E = self.E + self.dt * dE
        if keep is not None:
            keep["mf"], keep["dE"] = mf, dE

    def state(self):
        return self.E.cpu().numpy().T

    def budget(self, keep):
        n = self.n
        w = [self.spec(self.d[a][PAD:-PAD], a) for a in range(6)]
        vol = w[0] * w[1] * w[2] * w[3] * w[4] * w[5]
        dk, sp = w[3] * w[4] * w[5], (0, 1, 2)
        out = {"sums": np.array([float((keep["dE"] * vol).sum()), float((keep["mf"] * vol).sum())]),
               "mfl_max": float((keep["mf"].abs() / self.E.clamp(min=float(np.float32(1e-12)))).max())}
        vmax = [float(self.v[a].narrow(5 - a, 1, n[a]).abs().max()) for a in range(6)]
        bfl = []
        fields = {"E_int": (self.E * dk).sum(sp), "meanfl_int": (keep["mf"] * dk).sum(sp)}
        for a in range(6):
            for e in (0, 1):
                f = keep[a][e] if a in keep else torch.zeros((1,) * 6, dtype=torch.float64, device=self.dev)
                area = 1.0
                for b in range(6):
                    area = area * w[b] if b != a else area
                bfl.append(float((f * area).sum()) if a in keep else 0.0)
                if a >= 3:
                    part = 1.0
                    for b in (3, 4, 5):
                        part = part * w[b] if b != a else part
                    fields["diss_%s%s" % (AXES[a], "se"[e])] = (f * part).sum(sp).expand(n[2], n[1], n[0])
        out.update(bfl=np.array(bfl), vmax=vmax, fields={k: v.cpu().numpy().T for k, v in fields.items()},
                   cfl=np.array([vmax[a] * self.dt / float(w[a].min()) for a in range(6)]))
        return out


def exact(case, seed):
    out = []
    for i in _fields(case, seed):
        p = _Plain(i)
        keep = {} if case["use"] == "diagnose" else None
        for _ in range(case["steps"]):
            p.step(keep)
        if keep is not None:
            return p.budget(keep)
        if case["use"] == "setup":
            return {"rate": p.max_rate, "E": p.state()}
        out.append(p.state())
    return out if case["use"] == "ensemble" else out[0]
