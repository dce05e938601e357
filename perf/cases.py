"""Workloads of the stepper, for timing it through its public entry points.

A case is one of two kinds of work that a user of the package has it do:

  solve  a handle (Solver) that is advanced by `steps` time steps and then read, again and
         again: the reference's time loop with its probe and DFT monitor, plus the fields a
         program looks at between runs.  The handle is kept, as a driver of a long run keeps it.
  batch  a set of independent jobs handed to the packed engine (Batch), run to their end and
         collected: the serving form.  The engine is kept for the process, as a server does
         (a device holds one at a time); the jobs are new every time.

Set-up data (mesh lines, CPML profiles, material rows, gain regions) is made here in FP64 and
passed as the plain-data view of the C ABI, so that nothing but the stepper is timed, and so
that `exact` can step the same data with plain torch in 64 bits.  The seed sets the initial
field, the sources' amplitudes and the pump.

Sizes come from the shipped configurations (80^3 sphere, 201 x 201 x 69 gain slab, 280^3 and
536^3 gain slabs, the 96 x 96 x 65 sweep cavities, the serving stream's 32 .. 192 cell cores).
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("3d_fdtd_version008_b200")

C0 = 299792458.0
EPS0 = 8.8541878128e-12
MU0 = 4e-7 * math.pi
HBAR = 1.054571817e-34
ETA0 = 376.730313668
PRECISION = {"fp32": pkg.PREC_FP32, "fp64": pkg.PREC_FP64, "fp16": pkg.PREC_FP16, "bf16": pkg.PREC_BF16}
WORD = {"fp32": 4, "fp64": 8, "fp16": 2, "bf16": 2}
FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
FREQS = np.linspace(168e12, 218e12, 21)


def _solve(name, n, npml, precision, steps, scene="vacuum", mesh="uniform", boundary="cpml", sheets=0, reads="fields",
           ds=20e-9):
    """nx, ny, nz count all cells, CPML included.  reads: "fields" all six, "ez" that component."""
    return {"name": name, "kind": "solve", "nx": n[0], "ny": n[1], "nz": n[2], "npml": npml, "precision": precision,
            "steps": steps, "scene": scene, "mesh": mesh, "boundary": boundary, "sheets": sheets, "reads": reads, "ds": ds}


def _batch(name, n, npml, precision, steps, jobs, spread, mesh="uniform", ds=20e-9):
    """spread 1: every job has the case's grid; else the jobs' edges lie between the grid's and
    that many times it, evenly over the logarithm."""
    return {"name": name, "kind": "batch", "nx": n[0], "ny": n[1], "nz": n[2], "npml": npml, "precision": precision,
            "steps": steps, "jobs": jobs, "spread": spread, "scene": "gain", "mesh": mesh, "boundary": "cpml",
            "sheets": 0, "reads": "none", "ds": ds}


def listed():
    return [
        # the smallest grid of the serving stream, advanced a few steps at a time by a program
        # that looks at one component in between: launches and latency count
        _solve("48^3 fp32, 10 steps", (48, 48, 48), 8, "fp32", 10, scene="sphere", reads="ez"),
        # the 64^3 + CPML dielectric sphere with a dipole, probe and DFT
        _solve("80^3 fp32 sphere", (80, 80, 80), 8, "fp32", 400, scene="sphere", ds=25e-9),
        # the graded-mesh gain slab: odd sizes, 10-cell CPML, two-level medium
        _solve("201x201x69 fp32 gain", (201, 201, 69), 10, "fp32", 400, scene="gain", mesh="graded", ds=12.5e-9),
        # two plane waves onto a sphere, in the accuracy mode, ragged
        _solve("173x131x97 fp64 waves", (173, 131, 97), 10, "fp64", 200, scene="sphere", sheets=2),
        # a metal box with a dielectric in it (no CPML): cavity modes
        _solve("157x121x93 fp32 metal box", (157, 121, 93), 0, "fp32", 300, scene="sphere", boundary="pec", sheets=1),
        # the gain-laser sweep: graded cavities, 16-bit storage, packed
        _batch("32 cavities 96x96x65 bf16", (96, 96, 65), 10, "bf16", 300, 32, 1.0, mesh="graded", ds=12.5e-9),
        # the serving stream: microcavities with core edges of 32 .. 192 cells, packed
        _batch("12 cavities fp32", (48, 48, 48), 8, "fp32", 300, 12, 3.5),
        # the 256^3 + CPML gain slab
        _solve("280^3 fp32 gain", (280, 280, 280), 12, "fp32", 300, scene="gain", reads="ez"),
        _solve("280^3 fp16 gain", (280, 280, 280), 12, "fp16", 300, scene="gain", reads="ez"),
        # the large solve: 512^3 + CPML gain slab, in the reference's own arithmetic and below it
        _solve("536^3 fp64 gain", (536, 536, 536), 12, "fp64", 120, scene="gain", reads="ez"),
        _solve("536^3 fp32 gain", (536, 536, 536), 12, "fp32", 200, scene="gain", reads="ez"),
        _solve("536^3 bf16 gain", (536, 536, 536), 12, "bf16", 200, scene="gain", reads="ez"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    if rng.random() < 0.25:
        n = tuple(int(_log(rng, 44, 110)) for _ in range(3))
        graded = rng.random() < 0.5
        case = _batch("", n, rng.choice((6, 8, 10)), rng.choice(("fp32", "bf16", "fp16")), 100 + rng.randrange(200),
                      2 + rng.randrange(15), 1.0 if rng.random() < 0.5 else 1.0 + rng.random(),
                      mesh="graded" if graded else "uniform")
    else:
        edge = _log(rng, 44, 400)
        n = tuple(max(40, int(edge * _log(rng, 0.7, 1.4))) for _ in range(3))
        cells = n[0] * n[1] * n[2]
        steps = int(min(400, max(10, 6e9 / cells)))
        scene = rng.choice(("vacuum", "sphere", "gain", "gain"))
        pec = scene != "gain" and rng.random() < 0.25
        precision = rng.choice(("fp32", "fp32", "fp64", "bf16", "fp16"))
        case = _solve("", n, 0 if pec else rng.choice((6, 8, 9, 10, 12)), precision,
                      10 + rng.randrange(steps), scene=scene, mesh=rng.choice(("uniform", "graded")),
                      boundary="pec" if pec else "cpml", sheets=rng.choice((0, 0, 0, 1, 2)),
                      # 16-bit storage: the driven component (the weak ones are its rounding noise)
                      reads="fields" if cells < 4e6 and WORD[precision] > 2 else "ez")
    case.pop("name")
    return case


# ------------------------------------------------------------------ set-up data, FP64
def _lines(n, npml, mesh, ds):
    """Cell sizes along one axis: uniform, or ds in the middle half growing by 1.15 to 3 ds."""
    d = np.full(n, ds)
    if mesh == "graded":
        dist = np.maximum(np.abs(np.arange(n) - 0.5 * (n - 1)) - 0.25 * n, 0.0)
        d = ds * np.minimum(1.15 ** np.minimum(dist, 20.0), 3.0)
    return d


def _cpml(d, npml, dt):
    """kappa, bE, cE, bH, cH of the polynomially graded CPML."""
    n = len(d)
    kappa, sigma, alpha = np.ones(n), np.zeros(n), np.zeros(n)
    if npml:
        at = np.minimum(np.arange(n), n - 1 - np.arange(n))
        inside = at < npml
        r = (npml - (at[inside] + 0.5)) / npml
        smax = 4.0 * math.log(1e6) * EPS0 * C0 / (2.0 * npml * float(np.mean(d[inside])))
        kappa[inside] = 1.0 + 4.0 * r**3
        sigma[inside] = smax * kappa[inside] * r**3
        alpha[inside] = 0.05 * (C0 / d[inside]) * (1.0 - r)
    out = [kappa]
    for norm in (EPS0, MU0):
        s = sigma / norm
        b = np.maximum(np.exp(-(s / kappa + alpha) * dt), 1e-30)
        den = kappa * (s + kappa * alpha)
        c = np.where(den > 1e-30, s * (b - 1.0) / np.where(den > 1e-30, den, 1.0), 0.0)
        out += [b, c]
    return out


class _Problem:
    """One solve's inputs, from a case's numbers and a seed."""

    def __init__(self, case, seed, shape=None, field=True):
        self.shape = n = tuple(shape or (case["nx"], case["ny"], case["nz"]))
        self.npml, self.precision, self.steps = case["npml"], case["precision"], case["steps"]
        self.pec = case["boundary"] == "pec"
        rng = np.random.default_rng(seed)
        self.d = [_lines(m, self.npml, case["mesh"], case["ds"]) for m in n]
        self.inv = [1.0 / d for d in self.d]
        self.dt = 0.99 / (C0 * math.sqrt(sum(1.0 / float(d.min()) ** 2 for d in self.d)))
        self.cpml = [_cpml(d, self.npml, self.dt) for d in self.d]
        c = [m // 2 for m in n]
        # material: rows 0 background, 1 .. 4 interface averages, 5 the dielectric
        eps = 1.0 + (11.56 - 1.0) * np.linspace(0.0, 1.0, 6)
        self.rows = np.repeat((self.dt / (EPS0 * eps))[:, None], 3, axis=1).copy()
        self.index = np.zeros(n, dtype=np.uint16)
        self.region = None
        core = [slice(self.npml + max(2, (m - 2 * self.npml) // 10), m - self.npml - max(2, (m - 2 * self.npml) // 10)) for m in n]
        if case["scene"] == "gain":
            # a slab normal to z, 22 cells thick at most, whose middle is the two-level medium
            half = min(11, (n[2] - 2 * self.npml) // 4)
            for r, h in ((2, half + 1), (5, half)):
                self.index[core[0], core[1], c[2] - h:c[2] + h] = r
            self.box = (core[0], core[1], slice(c[2] - half + 1, c[2] + half - 1))
            self.region = np.full(n, -1, dtype=np.int32)
            self.region[self.box] = 0
            self.N0 = 5e23
        elif case["scene"] == "sphere":
            rad = 0.16 * min(n)
            g = np.meshgrid(*[np.arange(m) - k for m, k in zip(n, c)], indexing="ij", sparse=True)
            dist = np.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2)
            self.index[:] = np.clip(np.rint(5 * (rad + 0.5 - dist)), 0, 5).astype(np.uint16)
        self.pump = float(10 ** rng.uniform(7, 11))
        w, gamma, tau = 2 * math.pi * 193.4e12, 2 * math.pi * 5e12, 1e-9
        beta = 2.0 + gamma * self.dt
        mu2 = 3 * math.pi * EPS0 * HBAR * C0**3 / (w**3 * tau)
        self.gain = dict(kapa_coeff=(2 * self.dt**2 / beta) * (2 * w / HBAR) * mu2, pa2=2 * (2 - w**2 * self.dt**2) / beta,
                         pa3=(gamma * self.dt - 2) / beta, inv_dt=1 / self.dt, tau=tau, hbar=HBAR, omega_a=w, N0=5e23,
                         pump_rate=self.pump, enable_population_clamp=0)
        # a z dipole off the centre, a continuous wave (it keeps the fields alive over long runs)
        at = (c[0] - n[0] // 8, c[1], c[2])
        self.dipole = dict(i=at[0], j=at[1], k=at[2], polarization=2, waveform=3,
                           cell_area=float(self.d[0][at[0]] * self.d[1][at[1]]), I0=1e-7 * float(rng.uniform(0.5, 2.0)),
                           f0=193.4e12, tau=1.06e-14, t0=3.18e-14, t_shift=3.18e-14)
        self.sheets = []
        for q in range(case["sheets"]):
            ax = 2 if q == 0 else 0
            comp = 0 if q == 0 else 1
            plane = self.npml + 3 if q == 0 else n[ax] - self.npml - 4
            rest = [a for a in range(3) if a != ax]
            lo = [self.npml + 1 for _ in rest]
            hi = [n[a] - self.npml - 2 for a in rest]
            self.sheets.append(dict(axis=ax, comp=comp, plane=plane, lo0=lo[0], hi0=hi[0], lo1=lo[1], hi1=hi[1],
                                    d=float(self.d[ax][plane]), sign=1.0 if q == 0 else -1.0, waveform=3,
                                    E0=float(rng.uniform(0.5, 2.0)), f0=193.4e12, tau=1.06e-14, t0=3.18e-14, t_shift=0.0))
        self.probe = (min(n[0] - 2, c[0] + n[0] // 8), c[1], c[2])
        self.amp = 1.0  # V/m of the seeded initial field
        self.seed = seed
        self.field = field

    def initial_ez(self):
        """Seeded Ez away from the outer faces, as a GPU tensor in idx3 order."""
        g = torch.Generator(device="cuda").manual_seed(int(self.seed))
        e = torch.zeros(self.shape, dtype=torch.float64, device="cuda")
        s = tuple(slice(2, m - 2) for m in self.shape)
        v = e[s]
        v.copy_(torch.randn(v.shape, generator=g, device="cuda", dtype=torch.float32))
        return e.mul_(self.amp)

    def view(self):
        """The C ABI's setup view and what it points to (kept until the handle exists)."""
        import ctypes as ct
        keep = []

        def ptr(a, kind=ct.c_double):
            a = np.ascontiguousarray(a)
            keep.append(a)
            return a.ctypes.data_as(ct.POINTER(kind))

        v = pkg.SetupV1()
        v.struct_size = ct.sizeof(pkg.SetupV1)
        v.precision = PRECISION[self.precision]
        v.NxT, v.NyT, v.NzT = self.shape
        v.npml, v.save_every, v.dt = self.npml, 1, self.dt
        v.dx, v.dy, v.dz = (ptr(d) for d in self.d)
        v.inv_dx, v.inv_dy, v.inv_dz = (ptr(d) for d in self.inv)
        for a in range(3):
            for name, arr in zip(("cpml_kappa", "cpml_bE", "cpml_cE", "cpml_bH", "cpml_cH"), self.cpml[a]):
                getattr(v, name)[a] = ptr(arr)
        v.bH_uniform = self.dt / MU0
        v.n_bE_rows = len(self.rows)
        v.bE_rows = ptr(self.rows)
        v.bE_index = ptr(self.index, ct.c_uint16)
        flat = ptr(np.zeros(1))
        for a in range(3):  # the rows and the index stand for the three arrays
            v.bE[a] = flat
        dip = (pkg.DipoleV1 * 1)(pkg.DipoleV1(**self.dipole))
        prb = (pkg.ProbeV1 * 1)(pkg.ProbeV1(*self.probe, pkg.COMPONENTS["Ez"], 0))
        keep += [dip, prb]
        v.n_dipoles, v.dipoles = 1, dip
        v.n_probes, v.probes = 1, prb
        v.n_dft_freqs, v.dft_freqs = len(FREQS), ptr(FREQS)
        if self.region is not None:
            reg = (pkg.TlsRegionV1 * 1)(pkg.TlsRegionV1(**self.gain))
            keep.append(reg)
            v.n_tls_regions, v.tls_regions = 1, reg
            v.tls_region_map = ptr(self.region, ct.c_int32)
            nu, ng = np.zeros(self.shape), np.zeros(self.shape)
            ng[self.box] = self.N0
            v.tls_Nu, v.tls_Ng = ptr(nu), ptr(ng)
        if self.sheets:
            sh = (pkg.SheetV1 * len(self.sheets))(*[pkg.SheetV1(**s) for s in self.sheets])
            keep.append(sh)
            v.n_sheets, v.sheets = len(self.sheets), sh
        v.pec_boundary = int(self.pec)
        v.monitor_interval, v.max_E, v.max_P, v.conservation_err, v.growth_rate = 10, 1e10, 1e5, 1e-2, 10.0
        return v, keep


def _grids(case):
    """The grids of a case: one, or the batch's jobs spread evenly over the logarithm of the
    edge, some of them a cell or two short along x or y."""
    n = (case["nx"], case["ny"], case["nz"])
    if case["kind"] == "solve":
        return [n]
    out = []
    for q in range(case["jobs"]):
        f = case["spread"] ** (q / max(1, case["jobs"] - 1))
        short = q % 3 if case["spread"] > 1 else 0
        out.append(tuple(int(round(m * f)) - (short if a == q % 2 else 0) for a, m in enumerate(n)))
    return out


def _jobs(case, seed):
    return [_Problem(case, seed + 1000 * q, shape=n, field=False) for q, n in enumerate(_grids(case))]


_ENGINE = []


def _engine():
    if not _ENGINE:
        _ENGINE.append(pkg.Batch(0, 100 << 30))
    return _ENGINE[0]


def prepare(case, seed):
    if case["kind"] == "batch":
        jobs = [p.view() + (p,) for p in _jobs(case, seed)]
        return {"case": case, "jobs": jobs, "engine": _engine()}
    p = _Problem(case, seed)
    v, keep = p.view()
    sol = pkg.Solver(None, view=v)
    del keep
    sol.set_field("Ez", p.initial_ez().cpu().numpy())
    return {"case": case, "solver": sol}


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        eng = state["engine"]
        tickets = [eng.submit(None, case["steps"], view=v) for v, _, _ in state["jobs"]]
        left = (1, 1)
        while left != (0, 0):
            left = eng.run(case["steps"])
        out = {"series": [], "dft": []}
        for t in tickets:
            out["series"].append(eng.probe_series(t))
            out["dft"].append(eng.dft(t))
            eng.release(t)
        # the jobs' series and spectra, one array each (the jobs take the same number of steps)
        return {"series": np.stack(out["series"]), "dft": np.stack(out["dft"])}
    sol = state["solver"]
    sol.run(case["steps"])
    out = {"dft": sol.dft(0)}
    for c in (FIELDS if case["reads"] == "fields" else ("Ez",)):
        out[c] = sol.field(c)
    if case["scene"] == "gain" and case["reads"] == "fields":
        out["Nu"] = sol.tls_state("Nu")
        out["Pz"] = sol.tls_state("Pz")
    return out


def work(case):
    """Per time step: E and H read and written once, the material's row number read, psi of
    each CPML cell and the two-level state of each gain cell read and written once; once per
    pass the fields that are read back.  36 operations per cell, 12 more per CPML slab and 20
    per gain cell."""
    w, m = WORD[case["precision"]], case["npml"]
    g = 8 if case["precision"] == "fp64" else 4
    total_b = total_f = 0.0
    for n in _grids(case):
        cells = n[0] * n[1] * n[2]
        slab = sum(2 * m * cells / n[a] for a in range(3))
        gain = 0.0
        if case["scene"] == "gain":
            gain = 0.8 * (n[0] - 2 * m) * 0.8 * (n[1] - 2 * m) * min(20, (n[2] - 2 * m) / 2)
        total_b += case["steps"] * (cells * (12 * w + 2) + slab * 8 * w + gain * 7 * g)
        total_f += case["steps"] * (36.0 * cells + 12.0 * slab + 20.0 * gain)
        total_b += 8.0 * cells * {"fields": 6, "ez": 1, "none": 0}[case["reads"]]
    return {"bytes": total_b, "flops": total_f}


# ------------------------------------------------------------------ the same in plain torch, 64 bits
def _waveform_cw(t, amp, f0, tau):
    env = 0.5 * (1 - math.cos(math.pi * t / tau)) if t < tau else 1.0
    return amp * env * math.sin(2 * math.pi * f0 * t)


def _step_exact(p, fields=True):
    """p.steps steps of the Yee loop on problem p: H, E with CPML, two-level medium, sources."""
    dev, f64 = "cuda", torch.float64
    n, np_, dt = p.shape, p.npml, p.dt
    E = [torch.zeros(n, dtype=f64, device=dev) for _ in range(3)]
    H = [torch.zeros(n, dtype=f64, device=dev) for _ in range(3)]
    if p.field:
        E[2] = p.initial_ez()
    tab = torch.from_numpy(p.rows[:, 0].copy()).to(dev)
    bE = tab[torch.from_numpy(p.index.astype(np.int32)).to(dev).long()] if np.prod(n) < 2e7 else None
    if bE is None:  # by row, without a full-grid 64-bit index
        idx = torch.from_numpy(p.index.astype(np.uint8)).to(dev)
        bE = torch.full(n, float(tab[0]), dtype=f64, device=dev)
        for r in range(1, len(tab)):
            bE.masked_fill_(idx == r, float(tab[r]))
        del idx
    bH = dt / MU0

    def line(a, ax):
        s = [1, 1, 1]
        s[ax] = len(a)
        return torch.from_numpy(np.ascontiguousarray(a)).to(dev).reshape(s)

    inv = [line(p.inv[a], a) for a in range(3)]
    ik = [line(1.0 / p.cpml[a][0], a) for a in range(3)]
    co = {"E": [(line(p.cpml[a][1], a), line(p.cpml[a][2], a)) for a in range(3)],
          "H": [(line(p.cpml[a][3], a), line(p.cpml[a][4], a)) for a in range(3)]}
    psi = {}

    def cut(t, ax, s):
        k = [slice(None)] * 3
        k[ax] = s
        return t[tuple(k)]

    # H holds cells [0, n-1) of each axis, E cells [1, n)
    rng_ = {"H": slice(0, -1), "E": slice(1, None)}

    def diff(f, ax, side):
        """One-sided difference along ax over the side's cells, with the CPML."""
        s = rng_[side]
        k1, k0 = [s] * 3, [s] * 3
        k1[ax], k0[ax] = slice(1, None), slice(0, -1)
        d = (f[tuple(k1)] - f[tuple(k0)]).mul_(cut(inv[ax], ax, s))
        return d

    def cpml(d, key, ax, side):
        if not np_:
            return d
        b, c = co[side][ax]
        m = n[ax]
        raw = [cut(d, ax, slice(0, np_ - (side == "E"))).clone(), cut(d, ax, slice(m - np_ - (side == "E"), m - 1)).clone()]
        d.mul_(cut(ik[ax], ax, rng_[side]))
        for q, part in enumerate((slice(1 if side == "E" else 0, np_), slice(m - np_, m if side == "E" else m - 1))):
            bb, cc = cut(b, ax, part), cut(c, ax, part)
            if (key, q) not in psi:
                psi[key, q] = torch.zeros_like(raw[q])
            psi[key, q].mul_(bb).add_(raw[q].mul_(cc))
            cut(d, ax, slice(0, np_ - 1) if side == "E" and q == 0 else slice(0, np_) if q == 0 else
                slice(m - np_ - (side == "E"), m - 1)).add_(psi[key, q])
        return d

    hs, es = (slice(0, -1),) * 3, (slice(1, None),) * 3
    if p.region is not None:
        P = torch.zeros([s.stop - s.start for s in p.box], dtype=f64, device=dev)
        Pp, Nu, Ng = torch.zeros_like(P), torch.zeros_like(P), torch.full_like(P, p.N0)
        g = p.gain
    series = torch.zeros(p.steps, dtype=f64, device=dev)
    for s in range(p.steps):
        # H
        a = cpml(diff(E[2], 1, "H"), "Hxy", 1, "H").sub_(cpml(diff(E[1], 2, "H"), "Hxz", 2, "H"))
        H[0][hs].sub_(a.mul_(bH))
        a = cpml(diff(E[0], 2, "H"), "Hyz", 2, "H").sub_(cpml(diff(E[2], 0, "H"), "Hyx", 0, "H"))
        H[1][hs].sub_(a.mul_(bH))
        a = cpml(diff(E[1], 0, "H"), "Hzx", 0, "H").sub_(cpml(diff(E[0], 1, "H"), "Hzy", 1, "H"))
        H[2][hs].sub_(a.mul_(bH))
        # the medium's polarization from E^n
        if p.region is not None:
            ez_old = E[2][p.box].clone()
            Pn = g["kapa_coeff"] * p.N0 * ((Ng - Nu) / p.N0) * ez_old + g["pa2"] * P + g["pa3"] * Pp
            dP = (Pn - P) / dt
        t_half = (s + 0.5) * dt
        # E
        curl = [cpml(diff(H[2], 1, "E"), "Exy", 1, "E").sub_(cpml(diff(H[1], 2, "E"), "Exz", 2, "E")),
                cpml(diff(H[0], 2, "E"), "Eyz", 2, "E").sub_(cpml(diff(H[2], 0, "E"), "Eyx", 0, "E")),
                cpml(diff(H[1], 0, "E"), "Ezx", 0, "E").sub_(cpml(diff(H[0], 1, "E"), "Ezy", 1, "E"))]
        d = p.dipole
        curl[2][d["i"] - 1, d["j"] - 1, d["k"] - 1] -= _waveform_cw(t_half, d["I0"], d["f0"], d["tau"]) / d["cell_area"]
        for w in p.sheets:
            J = 2.0 * _waveform_cw(t_half, w["E0"], w["f0"], w["tau"]) / (ETA0 * w["d"]) * w["sign"]
            rest = [a for a in range(3) if a != w["axis"]]
            k = [None] * 3
            k[w["axis"]] = w["plane"] - 1
            k[rest[0]] = slice(w["lo0"] - 1, w["hi0"])
            k[rest[1]] = slice(w["lo1"] - 1, w["hi1"])
            curl[w["comp"]][tuple(k)] -= J
        if p.region is not None:
            curl[2][tuple(slice(b.start - 1, b.stop - 1) for b in p.box)] -= dP
        for c in range(3):
            E[c][es].addcmul_(bE[es], curl[c])
        del curl
        if p.pec:
            for c in range(3):
                for ax in range(3):
                    cut(E[c], ax, slice(0, 1)).zero_()
                    cut(E[c], ax, slice(n[ax] - 1, n[ax])).zero_()
        if p.region is not None:
            avg = 0.5 * (E[2][p.box] + ez_old)
            stim = avg * dP / (g["hbar"] * g["omega_a"])
            dNu = stim - Nu / g["tau"] + g["pump_rate"] * Ng
            dNg = Nu / g["tau"] - stim - g["pump_rate"] * Ng
            Nu, Ng = (Nu + dt * dNu).clamp_(min=0), (Ng + dt * dNg).clamp_(min=0)
            Pp, P = P, Pn
        series[s] = E[2][p.probe]
    v = series.cpu().numpy()
    t = (np.arange(p.steps) + 1) * dt
    dft = (v[None, :] * np.exp(-2j * np.pi * FREQS[:, None] * t[None, :])).sum(axis=1) * dt
    out = {"series": v, "dft": dft}
    for name, f in zip(FIELDS, E + H):
        out[name] = f
    if p.region is not None:
        out["Nu"], out["Pz"] = torch.zeros(n, dtype=f64, device=dev), torch.zeros(n, dtype=f64, device=dev)
        out["Nu"][p.box], out["Pz"][p.box] = Nu, P
    return out


def exact(case, seed):
    if case["kind"] == "batch":
        if case["steps"] * case["jobs"] > 4000:  # launch by launch it would take too long
            return None
        r = [_step_exact(p) for p in _jobs(case, seed)]
        return {"series": np.stack([x["series"][:, None] for x in r]), "dft": np.stack([x["dft"] for x in r])}
    r = _step_exact(_Problem(case, seed))
    out = {"dft": r["dft"]}
    for c in (FIELDS if case["reads"] == "fields" else ("Ez",)):
        out[c] = r[c].cpu().numpy()
    if case["scene"] == "gain" and case["reads"] == "fields":
        out["Nu"], out["Pz"] = r["Nu"].cpu().numpy(), r["Pz"].cpu().numpy()
    return out
