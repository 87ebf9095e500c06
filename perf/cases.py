"""Performance cases of the FDTD framework: the work its users have it do.

A case is a dict of plain values.  `prepare` makes what a user's program holds
before the call (a simulation or a batch, its parameters made from the seed),
`run` is one pass through the public entry points, `work` what the pass cannot
do without, and `exact` the same outputs from a 64-bit solver written here
with dense torch operations.

Kinds of pass:

* solve      fdtd_reset, fdtd_run to Tend, the spectra and the probe record: a
             parameter sweep that keeps one simulation, and the reference
             program's own run
* view       single fdtd_step calls with one field plane read back: a live
             view or a host loop that looks at the field as it steps (the
             smallest calls)
* split      the four per-half entry points in the reference's launch order,
             as a port of its time loop calls them
* periodic   a solve with periodic x and y, reflectance and transmittance
* batch      a step block of many uneven simulations, spectra of all members
* snapshots  a solve that records snapshots in the stepper and drains them
* gradient   set_design, forward, backward: one iteration of an inverse design

Sizes come from the benchmark's configurations and the parity tests (34^3 to
384 x 384 x 256 cells); the pulses are short enough for a pass of a few
hundred steps to see them.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fdtd-cuda_b200"))

STEPS_BEFORE_VIEW = 220  # a view or split pass starts on fields the pulse has reached


def listed():
    return [
        # the smallest calls: a host loop that steps and looks (parity-test size)
        dict(name="view_52_fp32", kind="view", particle="sphere", nx=52, ny=52, nz=52, ncpml=10, fp=32,
             steps=8, freqs=9),
        # the benchmark's small plain configuration, whole
        dict(name="solve_64_fp32", kind="solve", particle="sphere", nx=64, ny=64, nz=64, ncpml=10, fp=32,
             steps=2000, freqs=101),
        # the FP64 build on a ragged grid, silver cube
        dict(name="solve_97x89x93_fp64", kind="solve", particle="cube", nx=97, ny=89, nz=93, ncpml=6, fp=64,
             steps=421, freqs=17),
        # the reference's time loop over the split entry points
        dict(name="split_128_fp32", kind="split", particle="sphere", nx=128, ny=128, nz=128, ncpml=10, fp=32,
             steps=16, freqs=51),
        # a metasurface cell: gold spheres on a film, periodic x and y
        dict(name="periodic_64x64x161_fp32", kind="periodic", particle="film", nx=64, ny=64, nz=161, ncpml=10,
             fp=32, steps=1200, freqs=41),
        # a sweep over particle sizes as one batch, edges 48 to 128
        dict(name="batch_16_fp32", kind="batch", particle="sphere", members=16, lo=48, hi=128, ncpml=10, fp=32,
             steps=256, freqs=51),
        # one inverse-design iteration, local metal (the gradient configuration's grid and design box)
        dict(name="gradient_96_fp32", kind="gradient", particle="none", nx=96, ny=96, nz=96, ncpml=10, fp=32,
             steps=600, freqs=48, design="32x32x16", every=200),
        # the same with the hydrodynamic current and recorded and recomputed shapes that are no multiple of a tile
        dict(name="gradient_hydro_184x168x129_fp32", kind="gradient", particle="disks", nx=184, ny=168, nz=129,
             ncpml=10, fp=32, steps=300, freqs=5, design="30x26x8", every=100),
        # field movies out of the stepper
        dict(name="snapshots_160x144x176_fp32", kind="snapshots", particle="cube", nx=160, ny=144, nz=176,
             ncpml=10, fp=32, steps=400, freqs=21, t_skip=50),
        # the headline: nonlocal rod dimer, both precisions
        dict(name="dimer_256_fp32", kind="solve", particle="dimer", nx=256, ny=256, nz=256, ncpml=12, fp=32,
             steps=512, freqs=201),
        dict(name="dimer_256_fp64", kind="solve", particle="dimer", nx=256, ny=256, nz=256, ncpml=12, fp=64,
             steps=256, freqs=201),
        # the large nonlocal configuration
        dict(name="disks_384x384x256_fp32", kind="solve", particle="disks", nx=384, ny=384, nz=256, ncpml=12,
             fp=32, steps=384, freqs=5),
    ]


def draw(rng):
    def log_uniform(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["view", "solve", "solve", "solve", "split", "periodic", "batch", "gradient", "snapshots"])
    fp = 64 if rng.random() < 0.3 else 32
    edge = log_uniform(40, 210)
    if kind == "gradient":
        edge = log_uniform(64, 160)
    elif kind == "view":
        edge = log_uniform(40, 96)
    n = [max(40, min(224, int(edge * rng.uniform(0.85, 1.18)))) for _ in range(3)]
    ncpml = 6 if min(n) < 64 else rng.choice([8, 10, 12])
    freqs = log_uniform(5, 150)
    cells = n[0] * n[1] * n[2]
    # steps of a pass: enough for the pulse to cross the grid, else at most a thousand and about 3e9 cell steps
    least = 270 + n[2]
    most = max(least + 40, min(1000, int(3e9 / cells / (fp / 32))))
    steps = rng.randrange(least, most) | 1
    case = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], ncpml=ncpml, fp=fp, freqs=freqs, steps=steps)
    if kind == "view":
        case.update(particle=rng.choice(["sphere", "cube", "hydro_sphere"]), steps=rng.randrange(1, 16))
    elif kind == "solve":
        case.update(particle=rng.choice(["sphere", "cube", "hydro_sphere", "disks"]))
        if min(n) < 100 and case["particle"] == "disks":
            case["particle"] = "sphere"
    elif kind == "split":
        case.update(particle=rng.choice(["sphere", "hydro_sphere"]), steps=rng.randrange(4, 32))
    elif kind == "periodic":
        case.update(particle="film", nx=max(2, n[0] // 16) * 8, ny=n[1] // 2, nz=max(n[2], 96), ncpml=10)
    elif kind == "batch":
        lo = log_uniform(40, 90)
        hi = min(144, lo + log_uniform(8, 64))
        case = dict(kind=kind, particle="sphere", members=rng.randrange(3, 16), lo=lo, hi=hi, fp=fp,
                    ncpml=6 if lo < 64 else 10, freqs=min(freqs, 64), steps=rng.randrange(100, 260))
    elif kind == "gradient":
        box = [max(4, min(32, (a - 2 * (ncpml + 16)) // 2)) for a in n]
        case.update(particle=rng.choice(["none", "hydro_sphere"]), design="%dx%dx%d" % tuple(box),
                    steps=min(steps, least + 60), every=rng.randrange(40, 160), fp=32)
    else:
        case.update(particle=rng.choice(["sphere", "cube"]), t_skip=max(10, steps // 9))
    return case


# ----------------------------------------------------------------------
# parameters: everything that the seed decides is decided here


def _params(case, seed):
    """The fdtd_params fields of a case (a list of dicts for a batch)."""
    rng = np.random.default_rng([int(seed), 20261205])
    if case["kind"] == "batch":
        # edges spread over the range, the inner ones moved by a cell at most: the same work for every seed, nearly
        edges = [int(e) for e in np.linspace(case["lo"], case["hi"], case["members"])]
        edges[1:-1] = [e + int(rng.integers(-1, 2)) for e in edges[1:-1]]
        return [_one(case, rng, (e, e, e)) for e in edges]
    return _one(case, rng, (case["nx"], case["ny"], case["nz"]))


def _one(case, rng, n):
    nc = case["ncpml"]
    small = min(n) < 64 or case["kind"] == "batch"
    inset, offset = (4, 2) if small else (10, 5)
    h = 1e-9 if case["particle"] in ("dimer", "disks", "hydro_sphere") else 2e-9
    periodic = case["kind"] == "periodic"
    p = dict(dx=h, dy=h, dz=h, NCELLX=n[0] - 2 * nc - 1, NCELLY=n[1] - 2 * nc - 1, NCELLZ=n[2] - 2 * nc - 1,
             NcpmlX=nc, NcpmlY=nc, NcpmlZ=nc, tfsf_inset=inset, box_offset=offset, material=3, first_medium=1,
             NUM_freq=case["freqs"], WL_or_freq=1, lam_min=450e-9, lam_max=850e-9, nano_sphere=0,
             BandWidth=8e15 * (2e-9 / h), lam_0=float(rng.uniform(560e-9, 640e-9)),
             MAX_AMP=float(rng.uniform(0.5, 2.0)), inc_phi_deg=0.0 if case["kind"] == "solve" and h > 1e-9 else 90.0,
             Tend=case["steps"] - 1, precision=0 if case["fp"] == 32 else 1)
    if case["kind"] in ("view", "split", "batch"):
        p["Tend"] = 4000  # these passes go on stepping
    room = (min(n) - 2 * (nc + inset + offset)) // 2 - 2  # cells from the centre to the absorption box
    if case["particle"] in ("sphere", "cube", "hydro_sphere"):
        most = max(2, min(room, 12))
        r = int(rng.integers(max(2, most - 2), most + 1))
        p.update(nano_sphere=3 if case["particle"] == "cube" else 1, nano_sphere_radius=(r + 0.25) * h)
        if case["particle"] == "cube":
            p.update(material=2, WL_or_freq=0)
        if case["particle"] == "hydro_sphere":
            p.update(NONLOCAL=3)
    elif case["particle"] == "dimer":
        p.update(NONLOCAL=3, hydro_D=3.0, geometry=1, axis=0, gap=2e-9, rod_diameter=10e-9,
                 rod_length=float(rng.integers(36, 41)) * 1e-9)
    elif case["particle"] == "disks":
        pitch = min(60, (min(n[0], n[1]) - 2 * (nc + inset + offset + 2)) // 3)
        p.update(NONLOCAL=3, hydro_D=3.0, geometry=2, disk_nx=3, disk_ny=3, pitch=pitch * h,
                 disk_diameter=(pitch // 2 - 1 + float(rng.uniform(0, 1))) * h, disk_height=min(10, room) * h,
                 slab_eps=2.25, slab_thickness=min(20, room) * h)
    elif case["particle"] == "film":
        p.update(NCELLX=n[0], NCELLY=n[1], NcpmlX=0, NcpmlY=0, tfsf_inset=8, periodic_xy=1, nano_sphere=1,
                 inf_disp_slab=2, dispersive_slab=n[2] // 2, inc_phi_deg=30.0,
                 nano_sphere_radius=(min(8, n[0] // 2 - 1, n[1] // 2 - 1) - 2 + int(rng.integers(0, 3)) + 0.25) * h)
    if case["kind"] == "gradient":
        box = [int(v) for v in case["design"].split("x")]
        lo = [a // 2 - b // 2 for a, b in zip(n, box)]
        p["design_box"] = [v for a, b in zip(lo, box) for v in (a, a + b)]
    if case["kind"] == "snapshots":
        p.update(t_skip=case["t_skip"], y_skip=1, z_skip=1)
    return p


def _rho(case, seed):
    bx, by, bz = (int(v) for v in case["design"].split("x"))
    return np.random.default_rng([int(seed), 7]).uniform(0, 1, (bz, by, bx)).astype(np.float32)


def _objective_freqs(case):
    m = case["freqs"]
    return sorted({0, m // 3, m - 1})


# ----------------------------------------------------------------------
# the pass


def prepare(case, seed):
    import fdtd_b200 as F
    p = _params(case, seed)
    if case["kind"] == "batch":
        batch = F.Batch([F.default_params(**q) for q in p])
        return dict(case=case, batch=batch)
    sim = F.Sim(F.default_params(**p))
    state = dict(case=case, sim=sim)
    if case["kind"] in ("view", "split"):
        sim.step(STEPS_BEFORE_VIEW)
    if case["kind"] == "gradient":
        state["rho"] = _rho(case, seed)
    if case["kind"] == "snapshots":
        sim.enable_snapshots(3, capacity=16)
    return state


def _table(t):
    """The ScatAbs table, its columns apart by what they hold (cross sections,
    face fluxes, incident field), since their scales differ."""
    return dict(lam=t[:, 0], cross_sections=t[:, 1:4], face_fluxes=t[:, 4:16], incident=t[:, 16:19])


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.step(case["steps"])
        return _tables([b.spectra(i) for i in range(b.n)])
    sim = state["sim"]
    if case["kind"] == "view":
        for _ in range(case["steps"]):
            sim.step(1)
        return sim.plane(0 if sim.params.inc_phi_deg else 1, 0, sim.shape[0] // 2)
    if case["kind"] == "split":
        for _ in range(case["steps"]):
            sim.update_h()
            sim.update_line()
            sim.update_e()
            sim.spectral_accumulate()
        return sim.plane(0, 1, sim.shape[1] // 2)
    if case["kind"] == "gradient":
        sim.set_design(state["rho"])
        value = sim.forward(_objective_freqs(case), case["every"])
        grad, grad_params = sim.backward()
        return dict(objective=value, grad=grad, grad_omega_D=grad_params[0], grad_gamma=grad_params[1])
    sim.reset()
    sim.run()
    if case["kind"] == "periodic":
        t = sim.reflectance()
        return dict(lam=t[:, 0], rt=t[:, 1:4], incident=t[:, 4:7], probe=sim.probe())
    out = dict(_table(sim.spectra()), probe=sim.probe())
    if case["kind"] == "snapshots":
        out["records"] = sim.drain_snapshots()
    return out


def _tables(tables):
    parts = [_table(t) for t in tables]
    return {k: np.stack([q[k] for q in parts]) for k in parts[0]}


# ----------------------------------------------------------------------
# what a pass cannot do without


def work(case):
    """Per step every field value read and written once per half step (three
    values updated from three others: 9 values a cell and pass), every CPML
    psi value read and written once, the dispersive cells' state once, the
    flux faces' DFT sums as one product per run; a gradient's reverse sweep
    moves what its forward moves."""
    es = case["fp"] // 8
    if case["kind"] == "batch":
        edges = np.linspace(case["lo"], case["hi"], case["members"])
        shapes = [(int(e),) * 3 for e in edges]
    else:
        shapes = [(case["nx"], case["ny"], case["nz"])]
    total_b = total_f = 0.0
    for n in shapes:
        cells = float(n[0]) * n[1] * n[2]
        nc = case["ncpml"]
        periodic = case["kind"] == "periodic"
        axes = (2,) if periodic else (0, 1, 2)
        psi = sum(2 * 2 * (2 * nc + 1) * cells / n[a] for a in axes)
        step_b = (18 * cells + 2 * psi) * es
        step_f = 36 * cells + 6 * psi
        if periodic:
            rows = 2 * 4.0 * n[0] * n[1]
        else:
            inset = 4 if min(n) < 64 or case["kind"] == "batch" else 10
            side = [a - 2 * (nc + inset) for a in n]
            rows = 2 * 2 * 4.0 * (side[0] * side[1] + side[1] * side[2] + side[0] * side[2])
        steps = case["steps"]
        run_b, run_f = steps * step_b, steps * step_f
        if case["kind"] != "view":
            samples = steps / 4.0
            run_b += samples * rows * es + rows * case["freqs"] * 16
            run_f += samples * rows * case["freqs"] * 4
        if case["kind"] == "gradient":
            run_b, run_f = 2 * run_b, 2 * run_f
        total_b += run_b
        total_f += run_f
    return {"bytes": total_b, "flops": total_f}


# ----------------------------------------------------------------------
# the same in 64 bits


def exact(case, seed):
    p = _params(case, seed)
    if case["kind"] == "batch":
        tables = []
        for q in p:
            s = _Solver(q)
            s.steps(case["steps"])
            tables.append(s.spectra())
        return _tables(tables)
    s = _Solver(p, rho=_rho(case, seed) if case["kind"] == "gradient" else None)
    if case["kind"] in ("view", "split"):
        s.steps(STEPS_BEFORE_VIEW + case["steps"])
        if case["kind"] == "view":
            return s.E[0 if p["inc_phi_deg"] else 1][:, :, s.n[0] // 2].T.contiguous()
        return s.E[0][:, s.n[1] // 2, :].T.contiguous()
    records = []
    if case["kind"] == "snapshots":
        done = 0
        while done < case["steps"]:
            s.steps(1 if done % case["t_skip"] == 0 else min(case["t_skip"] - done % case["t_skip"],
                                                             case["steps"] - done))
            if done % case["t_skip"] == 0:
                E = [e[:, :, s.n[0] // 2].T for e in s.E]
                # the aux line lies in the absorbing corner, where the field is all rounding, and before the
                # pulse has come in from the source the plane is
                plane = torch.sqrt(E[0] ** 2 + E[1] ** 2 + E[2] ** 2)
                records.append(dict(t=done, plane=plane if done >= 140 else None, aux=None, line=s.e_line.clone()))
            done = s.t
    else:
        s.steps(case["steps"])
    if case["kind"] == "gradient":
        t = s.spectra()
        w = torch.tensor([1.0, -1.0] * 3, dtype=torch.float64)
        return dict(objective=float(sum((t[m, 10:16].cpu() * w).sum() for m in _objective_freqs(case))), grad=None,
                    grad_omega_D=None, grad_gamma=None)
    if case["kind"] == "periodic":
        t = s.reflectance()
        return dict(lam=t[:, 0], rt=t[:, 1:4], incident=t[:, 4:7], probe=s.probe_record())
    out = dict(_table(s.spectra().cpu()), probe=s.probe_record())
    if records:
        out["records"] = records
    return out


class _Solver:
    """The scheme in FP64 with dense torch arrays [z, y, x]: Yee with CPML,
    total-field / scattered-field plane wave from a 1D line (normal
    incidence), Drude with two critical points or the hydrodynamic current,
    running DFT on the faces of the two flux boxes."""

    PI = 3.1415926535897932384626433832795
    EP0, MU0, C0, Z0 = 8.85418782e-12, 1.25663706e-06, 2.99792458e08, 376.730313462
    QE, ME = 1.60217662e-19, 9.10938356e-31
    GOLD = (1.1431, 1.3202e16, 1.0805e14, ((0.26698, -1.2371, 3.8711e15, 4.4642e14),
                                           (3.0834, -1.0968, 4.1684e15, 2.3555e15)), 5.476415562682574e28)
    SILVER = (1.4447, 1.3280e16, 9.1269e13, ((-1.5951, 3.1288, 8.2749e15, 5.1770e15),
                                             (0.25261, -1.5066, 6.1998e15, 5.4126e14)), 5.541318196761572e28)
    AX = (2, 1, 0)  # tensor dimension of x, y, z

    def __init__(self, p, rho=None):
        self.p, self.t = p, 0
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.per = bool(p.get("periodic_xy"))
        self.d = (p["dx"], p["dy"], p["dz"])
        self.dt = 0.5 * p["dy"] / self.C0
        ncell = (p["NCELLX"], p["NCELLY"], p["NCELLZ"])
        self.nc = (p["NcpmlX"], p["NcpmlY"], p["NcpmlZ"])
        self.n = tuple(c if self.per and a < 2 else c + 2 * q + 1 for a, (c, q) in enumerate(zip(ncell, self.nc)))
        self.nt = tuple(0 if self.per and a < 2 else p["tfsf_inset"] + self.nc[a] for a in range(3))
        shape = (self.n[2], self.n[1], self.n[0])
        self.E = [self._zeros(shape) for _ in range(3)]
        self.H = [self._zeros(shape) for _ in range(3)]
        self._cpml(shape)
        self._line()
        self.cee_h = self.dt / (self.Z0 * self.EP0)
        self.che = self.Z0 * self.dt / self.MU0
        self._material(shape, rho)
        self._dft()
        self.probe = []

    def _zeros(self, shape):
        return torch.zeros(shape, dtype=torch.float64, device=self.dev)

    def _tensor(self, a):
        return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=self.dev)

    def _along(self, a, axis):
        return self._tensor(a).reshape([-1 if self.AX[axis] == q else 1 for q in range(3)])

    # -- tables ---------------------------------------------------------
    def _cpml(self, shape):
        self.ke, self.kh, self.be, self.ce, self.bh, self.ch, self.ce_ey = [], [], [], [], [], [], None
        tables = []
        for a in range(3):
            n, nc, d = self.n[a], self.nc[a], self.d[a]
            ke, kh = np.full(n, d), np.full(n, d)
            be, ce, bh, ch = (np.zeros(n) for _ in range(4))
            far = n - 1 - nc

            def grade(xs, xa, d=d):
                kappa_max = self.p.get("cpml_kappa_max", 5.0)
                s = xs ** 3 * 0.8 * 4 / (self.Z0 * d)
                al = 0.05 * xa
                k = 1 + (kappa_max - 1) * xs ** 3
                b = math.exp(-(s / k + al) * (self.dt / self.EP0))
                c = 0.0 if k * al + s == 0.0 else s * (b - 1) / (k * (s + k * al))
                return b, c, k
            if nc > 0 and not (self.per and a < 2):
                for i in range(nc + 1):
                    be[i], ce[i], k = grade((nc - i) / nc, i / nc)
                    ke[i] *= k
                    be[far + i], ce[far + i], k = grade(i / nc, (nc - i) / nc)
                    ke[far + i] *= k
                for i in range(nc):
                    bh[i], ch[i], k = grade((nc - i - 0.5) / nc, (i + 0.5) / nc)
                    kh[i] *= k
                    bh[far + i], ch[far + i], k = grade((i + 0.5) / nc, (nc - i - 0.5) / nc)
                    kh[far + i] *= k
                    if a == 0:
                        bh[far + i] = 0.0  # the reference's far x slab of H runs with b = 0
            tables.append((ke, kh, be, ce, bh, ch))
        for a, (ke, kh, be, ce, bh, ch) in enumerate(tables):
            self.ke.append(self._along(ke, a))
            self.kh.append(self._along(kh, a))
            self.be.append(self._along(be, a))
            self.ce.append(self._along(ce / self.d[a], a))
            self.bh.append(self._along(bh, a))
            self.ch.append(self._along(ch / self.d[a], a))
        # the reference's near x slab of Ey takes the y axis's c
        ce = tables[0][3].copy()
        if not self.per:
            k = self.nc[0] + 1
            ce[:k] = np.resize(np.pad(tables[1][3][:self.nc[1] + 1], (0, k)), k)
        self.ce_ey = self._along(ce / self.d[0], 0)
        z = self._zeros
        self.psiE = {(c, a): z(shape) for c in range(3) for a in range(3) if a != c}
        self.psiH = {(c, a): z(shape) for c in range(3) for a in range(3) if a != c}

    def _line(self):
        p = self.p
        self.L = 6 * p["NCELLZ"]
        self.m0 = self.L // 2
        self.e_line, self.h_line = self._zeros(self.L), self._zeros(self.L)
        self.cl_h = self.Z0 * self.dt / (self.MU0 * self.d[0])
        self.cl_e = self.dt / (self.Z0 * self.EP0 * self.d[0])
        self.mur = (self.C0 * self.dt - self.d[0]) / (self.C0 * self.dt + self.d[0])
        self.end = [torch.zeros((), dtype=torch.float64, device=self.dev)] * 2
        phi = np.float32(np.float64(p["inc_phi_deg"]) * (self.PI / 180.0))
        sp, cp = float(np.sin(phi)), float(np.cos(phi))
        self.fe, self.fh = (sp, -cp, 0.0), (cp, sp, -0.0)
        width = math.ceil((6 / (p["BandWidth"] * 2 * self.PI)) / self.dt)
        t = np.arange(p["Tend"] + 1)
        u = ((t - 6 * width) / width).astype(np.float32)
        pulse = p["MAX_AMP"] * np.exp(-(u ** 2).astype(np.float64) / 2.0) * np.sin(
            2 * self.PI * (self.C0 / p["lam_0"]) * t * self.dt)
        self.pulse = self._tensor(pulse)
        nf = p["NUM_freq"]
        i = np.arange(nf) / (nf - 1.0)
        if p["WL_or_freq"] == 1:
            self.freq = self.C0 / (p["lam_min"] + i * (p["lam_max"] - p["lam_min"]))
        else:
            self.freq = self.C0 / p["lam_max"] + i * (self.C0 / p["lam_min"] - self.C0 / p["lam_max"])
        ph = 2 * self.PI * t[:-1, None] * self.dt * self.freq[None, :]
        self.einc = (pulse[:-1, None] * np.exp(1j * ph)).sum(0)

    def _shapes(self):
        """Cells of the metal per component and of the dielectric slab, [z, y, x] masks."""
        p, n = self.p, self.n
        x, y, z = (np.arange(n[a]).reshape([-1 if self.AX[a] == q else 1 for q in range(3)]) for a in range(3))
        cx, cy, cz = n[0] // 2, n[1] // 2, n[2] // 2
        off = ((0.5, 0, 0), (0, 0.5, 0), (0, 0, 0.5))
        metal = [np.zeros((n[2], n[1], n[0]), bool) for _ in range(3)]
        slab = np.zeros((n[2], n[1], n[0]), bool)
        geometry = p.get("geometry", 0)
        if geometry == 0:
            r = int(p.get("nano_sphere_radius", 0.0) / self.d[0])
            if p.get("inf_disp_slab") == 2:
                k0 = p["dispersive_slab"] + self.nt[1]
                for c in range(3):
                    metal[c] |= (z >= k0) & (z < k0 + int(p["nano_sphere_radius"] / self.d[2])) & (x >= 0) & (y >= 0)
                if self.per:
                    cz = k0 - r
            for c in range(3):
                X, Y, Z = x + off[c][0] - cx, y + off[c][1] - cy, z + off[c][2] - cz
                if p["nano_sphere"] == 1:
                    metal[c] |= np.sqrt(X * X + Y * Y + Z * Z) < r
                elif p["nano_sphere"] == 3:
                    metal[c] |= (X * X < r * r) & (Y * Y < r * r) & (Z * Z < r * r)
            return metal, slab
        for c in range(3):
            X, Y, Z = ((v + off[c][a] - m) * self.d[a] for a, (v, m) in enumerate(((x, cx), (y, cy), (z, cz))))
            if geometry == 1:
                R, length = 0.5 * p["rod_diameter"], p["rod_length"]
                rr, half = Y * Y + Z * Z, 0.5 * length - R
                for sg in (-1, 1):
                    t = np.abs(X - sg * (0.5 * p["gap"] + 0.5 * length))
                    e = np.maximum(t - half, 0.0)
                    metal[c] |= np.where(t <= half, rr < R * R, rr + e * e < R * R)
            else:
                R = 0.5 * p["disk_diameter"]
                for a in range(p["disk_nx"]):
                    for b in range(p["disk_ny"]):
                        U = X - (a - 0.5 * (p["disk_nx"] - 1)) * p["pitch"]
                        V = Y - (b - 0.5 * (p["disk_ny"] - 1)) * p["pitch"]
                        metal[c] |= (Z >= 0) & (Z < p["disk_height"]) & (U * U + V * V < R * R)
        if geometry == 2:
            Z = (z - cz) * self.d[2]
            t = self.nt[0]
            slab |= ((Z >= -p["slab_thickness"]) & (Z < 0) & (x > t) & (x < n[0] - t - 1) & (y > t) & (y < n[1] - t - 1))
        return metal, slab

    def _material(self, shape, rho):
        p, dt = self.p, self.dt
        metal, slab = self._shapes()
        blend = None
        if rho is not None:
            b = p["design_box"]
            blend = np.ones(shape)
            blend[b[4]:b[5], b[2]:b[3], b[0]:b[1]] = rho
            for c in range(3):
                metal[c][b[4]:b[5], b[2]:b[3], b[0]:b[1]] = True
        self.hydro = p.get("NONLOCAL") == 3
        any_metal = metal[0] | metal[1] | metal[2]
        self.ceh = torch.full(shape, self.cee_h, dtype=torch.float64, device=self.dev)
        if slab.any():
            # a cell is of the slab's class where one of its components is (a component in the metal leaves it)
            s = torch.as_tensor(slab & ~(metal[0] & metal[1] & metal[2]), device=self.dev)
            self.ceh[s] = dt / (self.Z0 * self.EP0 * p["slab_eps"])
        self.keep = []  # 1 where the Yee update writes, per component
        self.cells = []
        n = self.n
        for c in range(3):
            ok = np.ones(shape, bool)
            for a in range(3):
                if self.per and a < 2:
                    continue
                i = np.arange(n[a]).reshape([-1 if self.AX[a] == q else 1 for q in range(3)])
                ok &= (i < n[a] - 1) & ((i > 0) if a != c else (i >= 0))
            self.keep.append(self._tensor(ok & ~metal[c]))
            self.cells.append(torch.as_tensor(np.flatnonzero(metal[c] & ok), device=self.dev))
        eps_inf, wd, gam, poles, neq = self.GOLD if p["material"] == 3 else self.SILVER
        self.neq = neq
        C = []
        for A, phi, om, ga in poles:
            a0 = 2.0 * self.EP0 * A * om * (om * math.cos(phi) - ga * math.sin(phi))
            a1 = -2.0 * self.EP0 * A * om * math.sin(phi)
            b0, b1 = ga * ga + om * om, 2.0 * ga
            cc = 1 / dt ** 2 + b1 / (2 * dt) + b0 / 4
            C.append(((2 / dt ** 2 - b0 / 2) / cc, (b1 / (2 * dt) - 1 / dt ** 2 - b0 / 4) / cc,
                      (a0 / 4 + a1 / (2 * dt)) / cc, a0 / (2 * cc), (a0 / 4 - a1 / (2 * dt)) / cc))
        self.C = C
        dd = 1 / dt ** 2 + gam / (2 * dt)
        self.d1, self.d2 = 2 / (dd * dt * dt), (gam / (2 * dt) - 1 / dt ** 2) / dd
        if self.hydro:
            D = p.get("hydro_D", 2.0)
            beta = 1.39e6 * math.sqrt((3 * D / (D + 2)) / D)
            self.d3, self.d4, self.d5 = -self.QE / self.ME / dd / dt, self.QE / self.ME / dd / dt, 0.0
            self.dnl = neq ** (1 / 3) * beta * beta / dd
            drude = (0.0, 0.0, 0.0)
        else:
            self.d3 = self.d5 = self.EP0 * wd * wd / (4 * dd)
            self.d4 = self.EP0 * wd * wd / (2 * dd)
            drude = (self.d3, self.d4, self.d5)
        CE = self.EP0 * eps_inf + drude[0] + C[0][2] + C[1][2]
        CE1 = self.EP0 * eps_inf - (drude[1] + C[0][3] + C[1][3])
        CE2 = drude[2] + C[0][4] + C[1][4]
        self.m = []
        for c in range(3):
            k = self.cells[c].numel()
            r = torch.ones(k, dtype=torch.float64, device=self.dev)
            if blend is not None:
                r = self._tensor(blend).reshape(-1)[self.cells[c]]
            z = self._zeros(k)
            self.m.append(dict(r=r, CE=self.EP0 + r * (CE - self.EP0), CE1=self.EP0 + r * (CE1 - self.EP0), CE2=r * CE2,
                               en=z.clone(), cp=[z.clone(), z.clone()], cp1=[z.clone(), z.clone()], pd=z.clone(),
                               pd1=z.clone()))
        if self.hydro and any_metal.any():
            # a padded box around the metal for the currents and densities
            w = np.argwhere(any_metal)
            self.lo, self.hi = w.min(0) - 2, w.max(0) + 3
            box = tuple(int(b - a) for a, b in zip(self.lo, self.hi))
            self.bmask, self.br = [], []
            ones = np.ones(shape) if blend is None else blend
            s = tuple(slice(int(a), int(b)) for a, b in zip(self.lo, self.hi))
            self.box = s
            for c in range(3):
                self.bmask.append(self._tensor(metal[c][s]))
                self.br.append(self._tensor(ones[s]))
            self.J = [self._zeros(box) for _ in range(3)]
            self.J1 = [self._zeros(box) for _ in range(3)]
            self.N = [self._zeros(box) for _ in range(3)]
            self.N1 = [self._zeros(box) for _ in range(3)]

    # -- a time step ----------------------------------------------------
    def _next(self, a, axis):
        return torch.roll(a, -1, self.AX[axis])

    def _prev(self, a, axis):
        return torch.roll(a, 1, self.AX[axis])

    def _update_h(self):
        n = self.n
        for c in range(3):
            u, v = (c + 1) % 3, (c + 2) % 3
            # H_c += che (dE_u/dv - dE_v/du)
            du = self._next(self.E[u], v) - self.E[u]
            dv = self._next(self.E[v], u) - self.E[v]
            self.psiH[c, v] = self.bh[v] * self.psiH[c, v] + self.ch[v] * du
            self.psiH[c, u] = self.bh[u] * self.psiH[c, u] + self.ch[u] * dv
            add = self.che * (du / self.kh[v] - dv / self.kh[u] + self.psiH[c, v] - self.psiH[c, u])
            for a in (u, v):
                if not (self.per and a < 2):
                    add.narrow(self.AX[a], n[a] - 1, 1).zero_()
            self.H[c] += add

    def _curl_h(self, c):
        """curl H of component c without and with the CPML terms' psi, and the two differences."""
        u, v = (c + 1) % 3, (c + 2) % 3
        return self.H[v] - self._prev(self.H[v], u), self.H[u] - self._prev(self.H[u], v)

    def _faces(self, hfield):
        """(component, sign, axis, incident component, index along x, y, z) of the TFSF corrections."""
        n, t = self.n, self.nt
        out = []
        for axis in ((2,) if self.per else (0, 1, 2)):
            a, b = (axis + 1) % 3, (axis + 2) % 3
            for c, other, sg in ((a, b, -1), (b, a, 1)):
                for side in (0, 1):
                    if self.per and side == 1:
                        continue
                    i = [None] * 3
                    if hfield:
                        i[axis] = t[axis] - 1 if side == 0 else n[axis] - t[axis]
                        at = t[axis] if side == 0 else n[axis] - t[axis]  # the E cell that the correction takes
                    else:
                        i[axis] = t[axis] if side == 0 else n[axis] - t[axis]
                        at = t[axis] - 1 if side == 0 else n[axis] - t[axis]  # the H cell
                    # tangential ranges: a staggered axis ends one cell earlier
                    for q in (a, b):
                        half = (q == other) if hfield else (q == c)
                        hi = n[q] - t[q] + (0 if half else 1)
                        i[q] = slice(t[q], min(hi, n[q]))
                    # H_c takes E_other, E_c takes H_other with the other sign
                    s = sg if (side == 0) == hfield else -sg
                    out.append((c, s, axis, other, i, at))
        return out

    def _tfsf(self, hfield):
        fields = self.H if hfield else self.E
        line = self.e_line if hfield else self.h_line
        fac = self.fe if hfield else self.fh
        for c, s, axis, other, i, at in self._faces(hfield):
            f = fac[other]
            if f == 0.0:
                continue
            # distance from the line's origin along z, in cells
            if axis == 2:
                z = torch.tensor([at], device=self.dev)
            else:
                z = torch.arange(i[2].start, i[2].stop, device=self.dev)
            k = z - self.nt[2] + self.m0
            # the transverse components of the line: e[k] at k, h[k] at k + 1/2, where the grid's are too
            w = line[k]
            coef = self.che if hfield else self.cee_h
            val = s * coef * w * f / self.d[axis]
            view = fields[c][i[2] if axis != 2 else slice(i[2], i[2] + 1),
                             i[1] if axis != 1 else slice(i[1], i[1] + 1),
                             i[0] if axis != 0 else slice(i[0], i[0] + 1)]
            view += val.reshape(-1, 1, 1)

    def _update_line(self):
        e, h = self.e_line, self.h_line
        h[:-1] -= self.cl_h * (e[1:] - e[:-1])
        new = e.clone()
        new[1:-1] = e[1:-1] - self.cl_e * (h[1:-1] - h[:-2])
        new[0] = self.end[0] + self.mur * (new[1] - e[0])
        new[-1] = self.end[1] + self.mur * (new[-2] - e[-1])
        self.end = [new[1].clone(), new[-2].clone()]
        if self.t < self.pulse.numel():
            new[self.m0 - self.p.get("source_offset", 50)] += self.pulse[self.t]
        self.e_line = new

    def _shift(self, a, *moves):
        """a at the cell moved by each (axis, step); the box's pad is zero."""
        for axis, step in moves:
            a = torch.roll(a, -step, self.AX[axis])
        return a

    def _hydro_currents(self):
        inv = [1.0 / d for d in self.d]
        new = []
        for c in range(3):
            total = [0.0, 0.0]
            for a in range(3):
                for q, f in enumerate((self.J[a], self.J[a] * self.N[a])):
                    if a == c:
                        total[q] = total[q] + inv[c] ** 2 * (self._shift(f, (c, 1)) - 2 * f + self._shift(f, (c, -1)))
                    else:
                        total[q] = total[q] + inv[c] * inv[a] * (
                            self._shift(f, (c, 1)) - f - self._shift(f, (c, 1), (a, -1)) + self._shift(f, (a, -1)))
            cb = (self.neq + self.N[c]) ** (1.0 / 3.0)
            en = self._zeros(self.E[c].numel())
            en[self.cells[c]] = self.m[c]["en"]
            en = en.reshape(self.E[c].shape)[self.box]
            j = (self.d1 * self.J[c] + self.d2 * self.J1[c] + self.d3 * self.E[c][self.box] + self.d4 * en +
                 self.dnl * ((total[0] + total[1] / self.neq) / cb))
            new.append(j * self.br[c] * self.bmask[c])
        return new

    def _hydro_density(self, c, J, N):
        """The density of component c after its continuity update, from currents and densities of this phase."""
        k2 = 2.0 * self.dt / self.d[0]
        s = 0.0
        for a in range(3):
            if a == c:
                v1, v2 = self._shift(J[a], (c, 1)), self._shift(J[a], (c, -1))
                n1, n2 = self._shift(N[a], (c, 1)), self._shift(N[a], (c, -1))
            else:
                v1, v2 = 0.5 * (self._shift(J[a], (c, 1)) + J[a]), 0.5 * (self._shift(J[a], (c, 1), (a, -1)) +
                                                                          self._shift(J[a], (a, -1)))
                n1, n2 = 0.5 * (self._shift(N[a], (c, 1)) + N[a]), 0.5 * (self._shift(N[a], (c, 1), (a, -1)) +
                                                                          self._shift(N[a], (a, -1)))
            w = 0.5 if a == c else 1.0
            if a == 2 and c == 2:
                s = s + 0.5 * (v1 - v2)  # the reference's Ez update leaves the density out of its own term
            else:
                s = s + w * (n1 * v1 - n2 * v2)
            s = s + w * (v1 - v2) * self.neq
        return (self.N1[c] - k2 * s) * self.br[c] * self.bmask[c]

    def _update_e(self):
        curls = []
        new = []
        metal = any(c.numel() for c in self.cells)
        for c in range(3):
            u, v = (c + 1) % 3, (c + 2) % 3
            du, dv = self._curl_h(c)
            curl = du / self.ke[u] - dv / self.ke[v]
            curls.append(curl.reshape(-1)[self.cells[c]])
            cu = self.ce[u]
            cv = self.ce[v]
            if c == 1:
                cv = self.ce_ey  # v is x for Ey
            self.psiE[c, u] = (self.be[u] * self.psiE[c, u] + cu * du) * self.keep[c]
            self.psiE[c, v] = (self.be[v] * self.psiE[c, v] + cv * dv) * self.keep[c]
            new.append(self.ceh * (curl + self.psiE[c, u] - self.psiE[c, v]) * self.keep[c])
        J = N = None
        if metal and self.hydro:
            J = self._hydro_currents()
            Jp, Np = list(self.J), list(self.N)
            newN = []
            for c in range(3):
                newN.append(self._hydro_density(c, Jp, Np))
                Jp[c], Np[c] = J[c], newN[c]
            N = newN
        for c in range(3):
            E = self.E[c]
            if not self.cells[c].numel():
                E += new[c]
                continue
            m = self.m[c]
            en = E.reshape(-1)[self.cells[c]]
            rhs = self.dt * curls[c] / self.Z0 + m["CE1"] * en - m["CE2"] * m["en"]
            for q in range(2):
                rhs = rhs - (self.C[q][0] - 1) * m["cp"][q] - self.C[q][1] * m["cp1"][q]
            if self.hydro:
                src = self._zeros(E.shape)
                src[self.box] = J[c] * (self.neq + N[c])
                rhs = rhs + self.dt * self.QE * src.reshape(-1)[self.cells[c]]
            else:
                rhs = rhs - (self.d1 - 1) * m["pd"] - self.d2 * m["pd1"]
            val = rhs / m["CE"]
            for q in range(2):
                C = self.C[q]
                cp = C[0] * m["cp"][q] + C[1] * m["cp1"][q] + m["r"] * (C[2] * val + C[3] * en + C[4] * m["en"])
                m["cp1"][q], m["cp"][q] = m["cp"][q], cp
            if not self.hydro:
                pd = self.d1 * m["pd"] + self.d2 * m["pd1"] + m["r"] * (self.d3 * val + self.d4 * en + self.d5 * m["en"])
                m["pd1"], m["pd"] = m["pd"], pd
            m["en"] = en
            E += new[c]
            E.reshape(-1)[self.cells[c]] = val
        if J is not None:
            self.J1, self.J = self.J, J
            self.N1, self.N = self.N, N

    def steps(self, count):
        for _ in range(count):
            self._update_h()
            self._tfsf(True)
            self._update_line()
            self._tfsf(False)
            self._update_e()
            if self.t % 4 == 0:
                self._sample()
            i = [q // 2 for q in self.n]
            self.probe.append(torch.stack([e[i[2], i[1], i[0]] for e in self.E]))
            self.t += 1

    # -- spectra --------------------------------------------------------
    def _dft(self):
        """Flux faces: (normal axis, index, ranges of the other two); the absorption box's six, then the scattering box's."""
        n, t, o = self.n, self.nt, self.p["box_offset"]
        self.flux_faces = []
        if self.per:
            for k in (t[2] - 5, n[2] - t[2] - 5):
                self.flux_faces.append((2, k, (0, n[0]), (0, n[1])))
        else:
            for d in (o, -o):
                s, e = [q + d for q in t], [a - q - d for a, q in zip(n, t)]
                for axis in range(3):
                    u, v = [a for a in range(3) if a != axis]
                    for at in (s[axis], e[axis] - 1):
                        self.flux_faces.append((axis, at, (s[u], e[u]), (s[v], e[v])))
        self.samples, self.times, self.acc = [], [], None

    def _face(self, a, axis, at, ru, rv):
        i = [slice(*ru), slice(*rv)]
        i.insert(axis, at)
        return a[i[2], i[1], i[0]].reshape(-1)

    def _sample(self):
        row = [torch.cat([torch.cat([self._face(f, axis, at, ru, rv) for q, f in enumerate(F) if q != axis])
                          for axis, at, ru, rv in self.flux_faces]) for F in (self.E, self.H)]
        self.samples.append(torch.stack(row))
        self.times.append(self.t)
        if len(self.samples) == 32:
            self._contract()

    def _contract(self):
        if not self.samples:
            return
        x = torch.stack(self.samples)  # [sample, field, row]
        t = torch.tensor(self.times, dtype=torch.float64, device=self.dev)
        f = self._tensor(self.freq)
        if self.acc is None:
            self.acc = [[self._zeros((f.numel(), x.shape[2])) for _ in range(2)] for _ in range(2)]
        for h, delta in ((0, 1.0), (1, 0.5)):
            ph = 2 * self.PI * self.dt * f[:, None] * (t[None, :] + delta)
            self.acc[h][0].addmm_(torch.cos(ph), x[:, h])
            self.acc[h][1].addmm_(torch.sin(ph), x[:, h])
        self.samples, self.times = [], []

    def _fluxes(self):
        """[face, frequency]: sum over the face of Re(E_u conj H_v - E_v conj H_u) with (u, v, normal) right-handed."""
        self._contract()
        out, r = [], 0
        for axis, _, ru, rv in self.flux_faces:
            k = (ru[1] - ru[0]) * (rv[1] - rv[0])
            p = [[self.acc[h][c][:, r + q * k:r + (q + 1) * k] for q in range(2)] for h in range(2) for c in range(2)]
            er, ei, hr, hi = p
            s = (er[0] * hr[1] + ei[0] * hi[1] - er[1] * hr[0] - ei[1] * hi[0]).sum(1)
            out.append(-s if axis == 1 else s)
            r += 2 * k
        return torch.stack(out).cpu()

    def spectra(self):
        q = self._fluxes() * self.d[0] * self.d[1] / torch.as_tensor(np.abs(self.einc) ** 2)
        s = torch.tensor([-1.0, 1.0] * 3, dtype=torch.float64)
        ab, sca = (q[:6] * s[:, None]).sum(0), (q[6:] * s[:, None]).sum(0)
        if self.p.get("geometry", 0) == 0 and self.p["nano_sphere"] == 1:
            area = self.PI * self.p["nano_sphere_radius"] ** 2
            sca, ab = sca / area, -ab / area
        e = self.einc
        cols = [torch.as_tensor(self.C0 / self.freq), sca, ab, ab + sca, *q[6:], *q[:6],
                torch.as_tensor(np.abs(e)), torch.as_tensor(e.real.copy()), torch.as_tensor(e.imag.copy())]
        return torch.stack(cols, 1)

    def reflectance(self):
        q = self._fluxes()
        amp = torch.as_tensor(np.abs(self.einc))
        inc = self.n[0] * self.n[1] * (amp / 4) ** 2
        R, T = -q[0] / inc, q[1] / inc
        e = self.einc
        return torch.stack([torch.as_tensor(self.C0 / self.freq), R, T, 1 - R - T, amp, torch.as_tensor(e.real.copy()),
                            torch.as_tensor(e.imag.copy())], 1)

    def probe_record(self):
        return torch.stack(self.probe).cpu()
