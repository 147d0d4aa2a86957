"""Workloads for timing the framework through its public entry points.

A case is what a user's program does with one job of a moving-window study:
create a run (`native.Run`), give it the inlet reference and the bunch, step
it, sample the lab detector plane as it goes, read the final state back and
close it; or submit a batch of such jobs to the scan server (`native.Scan`);
or solve the initial self-field of a bunch.  The sizes are those of the
configurations in `aprl_b200.workloads`, of the tests and of the parameter
scan's ranges, odd extents among them.

`exact` restates the same physics in plain torch binary64, without the
framework's kernels: the Cowan-z field update with its CPML, the
conservative-source fixed point with either particle shape, held injection,
exits at the fixed lab plane, and the spectral solution of the Cowan Poisson
problem.
"""
import math

import numpy as np
import torch

from aprl_b200 import abi, native, workloads

C = workloads.C_LIGHT
QE = workloads.ELEMENTARY_CHARGE
ME = workloads.ELECTRON_MASS
EPS0 = 8.8541878128e-12
MU0 = 1.25663706212e-6
F64 = torch.float64


# ---------------------------------------------------------------------------
# the cases
def _run(name, nx, ny, nz, particles, steps, **options):
    case = dict(kind="run", nx=nx, ny=ny, nz=nz, particles=particles, steps=steps,
                shape="linear-binomial3", precision="fp64", magnet="dipole", field_t=1.0,
                cpml=8, table=True, held=False, deterministic=False, ledger=False,
                seams=False, detector_every=16, fields=False)
    case.update(options)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # The smallest job of a parameter scan: 35x33x37 cells, the mixed
        # precision of the scan, vacuum inlet.  Launches and latency.
        _run("scan-job-small", 35, 33, 37, 10_000, 10, precision="fp32-mixed", table=False,
             fields=True),
        # A host program that drives the operators one by one (the seams of
        # the C ABI), as a C++ driver in the shape of the reference loop does.
        _run("seams-small", 40, 36, 64, 20_000, 16, seams=True, fields=True),
        # A middling job of the scan, odd extents.
        _run("scan-job-medium", 91, 107, 263, 150_000, 64, precision="fp32-mixed", table=False,
             field_t=0.6),
        # The scan server with a small batch of unequal jobs in flight.
        dict(name="served-scan", kind="scan", jobs=6, slots=2, runs_per_slot=3, cells_max=128,
             nz_max=256, particles_max=200_000, steps=32),
        # The plain drift configuration (64x64x256 cells, 100k particles,
        # FP64): the parity run, its fields read back.
        _run("drift", 64, 64, 256, 100_000, 80, magnet="none", fields=True),
        # Held lab-plane injection in the bit-reproducible mode: a bunch
        # streams in through the inlet, pending, held and then active.
        _run("held-injection", 64, 56, 120, 60_000, 56, cpml=6, held=True, deterministic=True),
        # After the bunch has left: field-only steps of a mid-sized window.
        _run("field-only", 96, 88, 201, 0, 128, magnet="none", fields=True),
        # The headline configuration: dipole bending radiation, FP64.
        _run("dipole", 128, 128, 512, 1_000_000, 64, cpml=10),
        # The same window in the mixed precision with a thinner bunch.
        _run("dipole-mixed", 128, 128, 512, 300_000, 64, cpml=10, precision="fp32-mixed",
             table=False),
        # The quintic-compensated longitudinal shape on an ordinary window.
        _run("quintic", 112, 97, 300, 300_000, 24, shape="quintic-compensated"),
        # The planar-undulator configuration with the energy ledger: the
        # largest window.
        _run("undulator", 128, 128, 2048, 4_000_000, 12, cpml=10, precision="fp32-mixed",
             magnet="undulator", ledger=True, table=False),
        # The initial self-field of a bunch by conjugate gradients, E and B
        # read back.
        dict(name="self-field", kind="selffield", nx=96, ny=96, nz=256, particles=250_000,
             cpml=8, solver="cg"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    which = rng.random()
    if which < 0.12:
        return dict(kind="selffield", nx=rng.randint(40, 112), ny=rng.randint(40, 112),
                    nz=rng.randint(64, 300), particles=_log(rng, 2e4, 5e5),
                    cpml=rng.choice([4, 6, 8]), solver=rng.choice(["cg", "modal"]))
    if which < 0.2:
        return dict(kind="scan", jobs=rng.randint(3, 8), slots=rng.randint(1, 3),
                    runs_per_slot=rng.randint(1, 3), cells_max=rng.randint(48, 128),
                    nz_max=rng.randint(64, 256), particles_max=_log(rng, 2e4, 2e5),
                    steps=rng.randint(12, 32))
    shape = "quintic-compensated" if rng.random() < 0.25 else "linear-binomial3"
    held = rng.random() < 0.15
    nx, ny, nz = _log(rng, 32, 160), _log(rng, 32, 160), _log(rng, 36, 640)
    cells = nx * ny * nz
    most = 1.2e6 if shape == "linear-binomial3" else 4e5
    particles = 0 if rng.random() < 0.05 else _log(rng, 1e4, most)
    steps = rng.randint(16, 64) if cells < 4e6 and particles < 4e5 else rng.randint(12, 32)
    magnet = "dipole" if held else rng.choice(["dipole", "dipole", "none", "undulator"])
    if magnet == "undulator":
        steps = min(steps, 14)
        nz = max(nz, 2 * steps + 64)
    return _run(None, nx, ny, nz, max(particles, 10_000) if held else particles, steps,
                shape=shape, precision=rng.choice(["fp64", "fp64", "fp32-mixed"]), magnet=magnet,
                field_t=round(rng.uniform(0.1, 1.5), 3), cpml=rng.choice([6, 8, 10]),
                table=rng.random() < 0.5, held=held, deterministic=rng.random() < 0.2,
                seams=rng.random() < 0.15, fields=cells < 1e6)


# ---------------------------------------------------------------------------
# inputs
def _config(case):
    if case.get("magnet") == "undulator":
        boost = 3000.0 / math.sqrt(1.5)
        magnets = [workloads.planar_undulator(1.0, 0.03, -1.0, 1000)]
        d, dz = 4e-6, 1e-6
    else:
        boost = 10.0
        magnets = [workloads.dipole(case["field_t"])] if case.get("magnet") == "dipole" else []
        d, dz = 5e-6, 2e-6
    steps = case.get("steps", 4)
    cfg = workloads.make_config(case["nx"], case["ny"], case["nz"], d, d, dz, case["cpml"], boost,
                                case.get("shape", "linear-binomial3"), steps, magnets=magnets)
    cfg = workloads.with_precision(cfg, case.get("precision", "fp64"))
    return workloads.with_determinism(cfg, case.get("deterministic", False))


def _bunch(case, cfg, seed):
    """A Gaussian bunch of the lab frame truncated to the trusted region of
    the window and taken to the box frame (host arrays, as a user has them)."""
    n = case["particles"]
    names = ("x", "y", "z", "ux", "uy", "uz", "charge", "mass")
    if n == 0:
        out = {k: np.zeros(0) for k in names}
        out["id"] = np.zeros(0, dtype=np.uint64)
        return out
    undulator = case.get("magnet") == "undulator"
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 1000003 + 17)
    boost = cfg.boost_gamma
    if undulator:
        gamma_lab, sigma, sigma_z, charge = 3000.0, 30e-6, 50e-6, 355.0 * n * QE
    elif case["kind"] == "selffield":
        gamma_lab, sigma, sigma_z, charge = 8.84e6 / workloads.ELECTRON_REST_EV, 50e-6, 20e-6, 1e-10
    else:
        gamma_lab, sigma, sigma_z, charge = 1e9 / workloads.ELECTRON_REST_EV, 50e-6, 20e-6, 1e-10
    margin = 3
    half = [0.5 * (m - 2 * (cfg.cpml_cells_x + margin)) * h
            for m, h in ((cfg.nx, cfg.dx), (cfg.ny, cfg.dy))]
    sigma = min(sigma, 0.5 * min(half))
    exit_box = cfg.exit_lab_z / boost
    if case.get("held"):
        z_lo, z_hi = -48 * cfg.dz, 0.8 * exit_box
    else:
        z_lo = 2 * cfg.dz + 0.05 * (exit_box - 2 * cfg.dz)
        z_hi = 2 * cfg.dz + 0.95 * (exit_box - 2 * cfg.dz)
    u0 = math.sqrt(gamma_lab * gamma_lab - 1.0)

    def normal(count):
        return torch.randn(count, generator=gen, device=dev, dtype=F64)

    def truncated(count, scale, lo, hi, centre):
        got = []
        have = 0
        while have < count:
            v = centre + scale * normal(2 * count)
            v = v[(v > lo) & (v < hi)]
            got.append(v)
            have += v.numel()
        return torch.cat(got)[:count]

    # A quiet start: z at the quantiles of its distribution, so the number of
    # particles that pass a plane does not depend on the seed.
    quantile = (torch.randperm(n, generator=gen, device=dev).to(F64) + 0.5) / n

    x = truncated(n, sigma, -half[0], half[0], 0.0)
    y = truncated(n, sigma, -half[1], half[1], 0.0)
    if undulator:
        # none leaves during the pass: the drift in the resonant frame differs
        # from particle to particle, and so would their number
        z_hi = min(z_hi, exit_box - 2 * (case["steps"] + 2) * cfg.dz)
    sigma_zb = sigma_z * boost * (1.0 + cfg.boost_beta)
    if undulator:
        z = z_lo + (z_hi - z_lo) * quantile
    else:
        cut = math.erf(0.5 * (z_hi - z_lo) / sigma_zb / math.sqrt(2.0))
        z = 0.5 * (z_lo + z_hi) + sigma_zb * math.sqrt(2.0) * torch.erfinv(
            cut * (2.0 * quantile - 1.0))
    spread = 1e-6 / (max(sigma, 30e-6) if undulator else sigma)
    ux, uy = spread * normal(n), spread * normal(n)
    uz = u0 * (1.0 + 1e-4 * normal(n))
    rapidity = boost + cfg.boost_gamma_beta
    mt2 = 1.0 + ux * ux + uy * uy
    positive = (torch.sqrt(mt2 + uz * uz) + uz) / rapidity
    out = {"x": x, "y": y, "z": z, "ux": ux, "uy": uy, "uz": 0.5 * (positive - mt2 / positive)}
    held = (torch.sqrt(1.0 + uz * uz) + uz) / rapidity
    u_held = 0.5 * (held - 1.0 / held)
    out["beta_held"] = u_held / torch.sqrt(1.0 + u_held * u_held)
    out = {k: v.cpu().numpy() for k, v in out.items()}
    per = charge / QE / n
    out["charge"] = np.full(n, -QE * per)
    out["mass"] = np.full(n, ME * per)
    out["id"] = np.arange(1, n + 1, dtype=np.uint64)
    return out


def _table(cfg, seed):
    """A smooth inlet reference, native layout (k, j, i)."""
    gen = torch.Generator()
    gen.manual_seed(int(seed) * 7919 + 5)
    out = []
    for a in range(6):
        nx_c, ny_c, nz_c = abi.reference_shape(cfg, a)
        phase = 2 * math.pi * torch.rand(3, generator=gen, dtype=F64)
        i, j, k = (torch.arange(m, dtype=F64, device="cuda") for m in (nx_c, ny_c, nz_c))
        value = (torch.sin(2 * math.pi * (i + 0.5) / nx_c + phase[0].item())[None, None, :] *
                 torch.cos(2 * math.pi * (j + 0.25) / ny_c + phase[1].item())[None, :, None] *
                 torch.cos(2 * math.pi * k / 37.0 + phase[2].item())[:, None, None])
        out.append(((1e3 if a < 3 else 1e3 / C) * value).cpu().numpy())
    return out


def _inputs(case, seed):
    cfg = _config(case)
    particles = _bunch(case, cfg, seed)
    frozen = None
    if case.get("held"):
        release = (cfg.activation_plane_lab_z - cfg.lab_z_origin) / cfg.boost_gamma
        frozen = (particles["z"] < release).astype(np.uint8)
    return cfg, particles, frozen, _table(cfg, seed) if case.get("table") else None


def _jobs(case, seed):
    """The unequal jobs of a scan batch; their sizes belong to the case."""
    rng = np.random.default_rng([case["jobs"], case["cells_max"], case["nz_max"],
                                 case["particles_max"]])
    out = []
    for n in range(case["jobs"]):
        job = _run(None, int(rng.integers(32, case["cells_max"] + 1)),
                   int(rng.integers(32, case["cells_max"] + 1)),
                   int(rng.integers(40, case["nz_max"] + 1)),
                   int(10 ** rng.uniform(4.0, math.log10(case["particles_max"]))), case["steps"],
                   precision="fp32-mixed", table=False,
                   field_t=round(float(rng.uniform(0.1, 1.5)), 3))
        out.append((job, _inputs(job, 100 * seed + n)))
    return out


def prepare(case, seed):
    if case["kind"] == "scan":
        return {"case": case, "jobs": _jobs(case, seed),
                "server": native.Scan(native.load(), slots=case["slots"],
                                      runs_per_slot=case["runs_per_slot"])}
    cfg, particles, frozen, table = _inputs(case, seed)
    state = {"case": case, "cfg": cfg, "particles": particles, "frozen": frozen, "table": table}
    if case["kind"] == "selffield":
        run_ = native.Run(native.load(), cfg)
        run_.set_particles(particles)
        state["run"] = run_
        state["solve"] = abi.self_field_config(cfg, solver=case["solver"])
    return state


# ---------------------------------------------------------------------------
# one pass
def _step(r, case, steps):
    if not case["seams"]:
        r.step(steps)
        return
    cfg = r.config
    for _ in range(steps):
        r.advance_magnetic()
        r.preview_electric()
        for trial in range(cfg.max_trials):
            force, defect, scale, calls = r.coupling_trial()
            work = 0.0 if calls == 0 else (defect / scale if scale > 0 else defect)
            if (trial + 1 >= (2 if calls > 0 else 1) and force < cfg.force_tolerance and
                    work < cfg.work_tolerance):
                break
        r.commit_electric()
        r.shift()


def run(state):
    case = state["case"]
    if case["kind"] == "scan":
        server = state["server"]
        tickets = [server.submit(cfg, particles, case["steps"],
                                 detector_lab_z=workloads.detector_plane_lab_z(cfg))
                   for _, (cfg, particles, _, _) in state["jobs"]]
        done = [server.wait(t) for t in tickets]
        for d in done:
            if d["state"] != abi.SCAN_DONE or d["status"] != abi.APRL_OK:
                raise RuntimeError("scan job failed: %s" % d["message"])
        return {"planes": [d["detector"] for d in done],
                "particles": [d["stats"]["particles"] for d in done]}
    if case["kind"] == "selffield":
        r = state["run"]
        r.initialize_self_field(state["solve"])
        return {"fields": [r.get_field(a) for a in range(6)]}
    cfg = state["cfg"]
    r = native.Run(native.load(), cfg)
    if state["table"] is None:
        r.allocate_reference()
    else:
        r.set_reference(state["table"])
    r.set_particles(state["particles"])
    if state["frozen"] is not None:
        r.set_held(state["frozen"], state["particles"]["beta_held"])
    if case["ledger"]:
        r.enable_energy_ledger()
    lab_z = workloads.detector_plane_lab_z(cfg)
    planes = []
    left = case["steps"]
    while left > 0:
        steps = min(left, case["detector_every"])
        _step(r, case, steps)
        planes.append(r.sample_field_plane(lab_z))
        left -= steps
    out = {"planes": planes, "particles": r.get_particles(), "carriers": r.carrier_count()}
    out["particles"]["id"] = out["particles"]["id"].view(np.int64)
    if case["fields"]:
        out["fields"] = [r.get_field(a) for a in range(6)]
    if case["ledger"]:
        out["ledger"] = r.energy_ledger()["field_energy_interior"]
    r.close()
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
def work(case):
    if case["kind"] == "scan":
        parts = [work(job) for job, _ in _sizes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    cells = case["nx"] * case["ny"] * case["nz"]
    n = case["particles"]
    if case["kind"] == "selffield":
        # rho and the six fields once, the particles once; a spectral solve
        # of the operator (three sine transforms each way by FFT)
        return {"bytes": 8.0 * (7 * cells + 8 * n),
                "flops": 15.0 * cells * math.log2(cells) + 60.0 * cells + 60.0 * n}
    steps = case["steps"]
    # per step: E and B read and written (96 B a cell); a particle's position
    # and momentum read and written, its charge and mass read (112 B)
    moved = steps * (96.0 * cells + 112.0 * n)
    # the bunch in; the particles, planes and (where asked) fields out
    planes = -(-steps // case["detector_every"])
    ends = 72.0 * n * 2 + planes * 48.0 * case["nx"] * case["ny"]
    if case["fields"]:
        ends += 48.0 * cells
    # per cell the smoothed curl of the magnetic update (about 220) and the
    # plain curl of the electric one (20); per particle and trial (two at
    # least) a gather and a deposit of the shape's nodes, and a push
    nodes = 44 if case["shape"] == "linear-binomial3" else 132
    flops = steps * (240.0 * cells + 2 * n * (4.0 * nodes + 300.0))
    return {"bytes": moved + ends, "flops": flops}


def _sizes(case):
    rng = np.random.default_rng([case["jobs"], case["cells_max"], case["nz_max"],
                                 case["particles_max"]])
    out = []
    for _ in range(case["jobs"]):
        job = _run(None, int(rng.integers(32, case["cells_max"] + 1)),
                   int(rng.integers(32, case["cells_max"] + 1)),
                   int(rng.integers(40, case["nz_max"] + 1)),
                   int(10 ** rng.uniform(4.0, math.log10(case["particles_max"]))), case["steps"])
        rng.uniform(0.1, 1.5)
        out.append((job, None))
    return out


def tolerance(case):
    # About four times what the worst output is off exact() by: 1.4e-11 in
    # FP64 (Bz, a cancellation residue that any other order of the current's
    # sum moves), 3.1e-9 with the gathers in binary32 (the transverse
    # momenta), 3.4e-11 for the conjugate gradients, which stop at a relative
    # residual of 1e-10.
    if case["kind"] == "selffield":
        return {"rel": 1.5e-10, "max": 1e-8}
    if case["kind"] == "scan" or case["precision"] == "fp32-mixed":
        return {"rel": 1.2e-8, "max": 1e-7}
    return {"rel": 6e-11, "max": 1e-9}


# ---------------------------------------------------------------------------
# the same in plain torch binary64
class _Profile:
    """CFS-CPML coefficients along one axis (zero outside the layers)."""

    def __init__(self, n, cells, spacing, cfg, electric):
        count = n + (1 if electric else 0)
        pos = np.arange(count) + (0.0 if electric else 0.5)
        depth = np.clip(np.maximum((cells - pos) / cells, (pos - (n - cells)) / cells), 0.0, 1.0)
        order = cfg.cpml_polynomial_order
        smax = -(order + 1.0) * C * math.log(cfg.cpml_target_reflection) / (2.0 * cells * spacing)
        graded = depth ** order
        sigma, kappa = smax * graded, 1.0 + (cfg.cpml_kappa_max - 1.0) * graded
        alpha = cfg.cpml_alpha_fraction * smax * (1.0 - depth)
        on = depth > 0.0
        decay = np.where(on, np.exp(-(sigma / kappa + alpha) * cfg.dt), 0.0)
        den = sigma * kappa + alpha * kappa * kappa
        drive = np.where(on & (den > 0), sigma * (decay - 1.0) / np.where(den > 0, den, 1.0), 0.0)
        self.ikm1 = torch.tensor(np.where(on, 1.0 / kappa - 1.0, 0.0), device="cuda")
        self.decay = torch.tensor(decay, device="cuda")
        self.drive = torch.tensor(drive, device="cuda")

    def correction(self, axis, difference, psi):
        """psi is advanced in place; axis 2 = x, 1 = y of a (k, j, i) array."""
        view = (lambda v: v[None, None, :]) if axis == 2 else (lambda v: v[None, :, None])
        psi.mul_(view(self.decay)).add_(view(self.drive) * difference)
        return view(self.ikm1) * difference + psi


def _cowan(dx, dy, dz):
    rx, ry, rz = (dz / dx) ** 2, (dz / dy) ** 2, 1.0
    den = rx * ry + ry * rz + rz * rx
    pf = rx * ry * rz / den
    beta = [r * (1 - pf) / 8 for r in (rx, ry, rz)]
    dxy = rx * ry * (1 / 16 - rx * ry / (8 * den))
    dyz = ry * rz * (1 / 16 - ry * rz / (8 * den))
    dzx = rz * rx * (1 / 16 - rz * rx / (8 * den))
    delta = [dyz, dzx, dxy]
    alpha = [1 - 2 * beta[1] - 2 * beta[2] - 4 * dyz, 1 - 2 * beta[2] - 2 * beta[0] - 4 * dzx,
             1 - 2 * beta[0] - 2 * beta[1] - 4 * dxy]
    return alpha, beta, delta


def _smooth(p, d, coeff):
    """The 9-point smoothing across axis d (0 x, 1 y, 2 z) of an array padded
    by one in every direction; the result drops the padding across d only."""
    alpha, beta, delta = coeff
    dims = [2, 1, 0]
    ta, tb = (d + 1) % 3, (d + 2) % 3

    def at(a, b):
        v = p
        for axis, o in ((ta, a), (tb, b)):
            v = v.narrow(dims[axis], 1 + o, p.shape[dims[axis]] - 2)
        return v

    out = alpha[d] * at(0, 0)
    out += beta[ta] * (at(-1, 0) + at(1, 0)) + beta[tb] * (at(0, -1) + at(0, 1))
    out += delta[d] * (at(-1, -1) + at(-1, 1) + at(1, -1) + at(1, 1))
    return out


def _pad_electric(e, c, lower):
    """E component c with its PEC parity in x and y, the inlet plane below
    and zero above, one node on every side."""
    p = torch.zeros([s + 2 for s in e.shape], dtype=F64, device="cuda")
    p[1:-1, 1:-1, 1:-1] = e
    p[0, 1:-1, 1:-1] = lower
    if c == 0:
        p[:, :, 0], p[:, :, -1] = p[:, :, 1], p[:, :, -2]
    else:
        p[:, :, 0], p[:, :, -1] = -p[:, :, 2], -p[:, :, -3]
    if c == 1:
        p[:, 0], p[:, -1] = p[:, 1], p[:, -2]
    else:
        p[:, 0], p[:, -1] = -p[:, 2], -p[:, -3]
    return p


class _Box:
    """One moving-window run."""

    def __init__(self, cfg, particles, frozen, table):
        self.cfg = cfg
        self.n3 = (cfg.nx, cfg.ny, cfg.nz)
        zeros = lambda a: torch.zeros(abi.field_shape(cfg, a)[::-1], dtype=F64, device="cuda")  # noqa: E731
        self.e = [zeros(a) for a in range(3)]
        self.b = [zeros(3 + a) for a in range(3)]
        self.psi_b = {"xy": zeros(3), "yx": zeros(4), "zx": zeros(5), "zy": zeros(5)}
        self.psi_e = {"xy": zeros(0), "yx": zeros(1), "zx": zeros(2), "zy": zeros(2)}
        self.mx = _Profile(cfg.nx, cfg.cpml_cells_x, cfg.dx, cfg, False)
        self.my = _Profile(cfg.ny, cfg.cpml_cells_y, cfg.dy, cfg, False)
        self.ex = _Profile(cfg.nx, cfg.cpml_cells_x, cfg.dx, cfg, True)
        self.ey = _Profile(cfg.ny, cfg.cpml_cells_y, cfg.dy, cfg, True)
        self.coeff = _cowan(cfg.dx, cfg.dy, cfg.dz)
        self.table = None if table is None else [torch.tensor(t, device="cuda") for t in table]
        self.step_index, self.offset, self.time = 0, cfg.initial_offset, 0.0
        self.h = torch.tensor([cfg.dx, cfg.dy, cfg.dz], dtype=F64, device="cuda")
        self.origin = torch.tensor([cfg.reference_origin[0], cfg.reference_origin[1],
                                    cfg.reference_origin[2] + cfg.initial_offset * cfg.dz],
                                   dtype=F64, device="cuda")
        t = {k: torch.tensor(np.ascontiguousarray(v.astype(np.float64)), device="cuda")
             for k, v in particles.items()}
        n = t["x"].numel()
        p = {"pos": torch.stack([t["x"], t["y"], t["z"]], 1),
             "u": torch.stack([t["ux"], t["uy"], t["uz"]], 1), "q": t["charge"], "m": t["mass"],
             "id": t["id"],
             "frozen": torch.zeros(n, dtype=torch.bool, device="cuda") if frozen is None
             else torch.tensor(frozen.astype(bool), device="cuda"),
             "beta": t.get("beta_held", torch.zeros(n, dtype=F64, device="cuda"))}
        self.queue, self.due = None, None
        if frozen is not None:
            inc = C * cfg.dt * p["beta"]
            start = self.origin[2]
            # due at the first step whose held chord ends at or above its inlet
            s = torch.clamp(torch.ceil((start - p["pos"][:, 2] - inc) / (cfg.dz + inc)), min=0.0)
            upstream = p["frozen"] & (p["pos"][:, 2] < start) & (s > 0)
            self.queue = {k: v[upstream] for k, v in p.items()}
            due = s[upstream]
            order = torch.argsort(due, stable=True)
            self.queue = {k: v[order] for k, v in self.queue.items()}
            self.due = due[order]
            p = {k: v[~upstream] for k, v in p.items()}
        self.p = p
        none = torch.zeros((0, 3), dtype=F64, device="cuda")
        self.carriers = {"pos": none, "vel": none.clone(), "q": none[:, 0].clone()}
        self.prescribed = [cfg.magnets[m] for m in range(cfg.n_magnets)]

    # -- fields
    def inlet(self, a, k, step):
        if self.table is None:
            return 0.0
        z = float(k) - self.cfg.translation_beta * float(step)
        lo = int(math.floor(z))
        f = z - lo
        t = self.table[a]
        return t[lo] if f == 0.0 else (1.0 - f) * t[lo] + f * t[min(lo + 1, t.shape[0] - 1)]

    def magnetic(self):
        cfg = self.cfg
        dtx, dty, dtz = cfg.dt / cfg.dx, cfg.dt / cfg.dy, cfg.dt / cfg.dz
        pads = [_pad_electric(self.e[a], a, self.inlet(a, self.offset - 1, self.step_index))
                for a in range(3)]
        y_z = _smooth(pads[1], 2, self.coeff)[1:-1]
        z_y = _smooth(pads[2], 1, self.coeff)[:, 1:-1]
        ez_y, ey_z = z_y[:, 1:] - z_y[:, :-1], y_z[1:] - y_z[:-1]
        self.b[0] -= dty * ez_y - dtz * ey_z
        self.b[0] -= dty * self.my.correction(1, ez_y, self.psi_b["xy"])
        del y_z, z_y, ez_y, ey_z
        x_z = _smooth(pads[0], 2, self.coeff)[1:-1]
        z_x = _smooth(pads[2], 0, self.coeff)[:, :, 1:-1]
        ex_z, ez_x = x_z[1:] - x_z[:-1], z_x[:, :, 1:] - z_x[:, :, :-1]
        self.b[1] -= dtz * ex_z - dtx * ez_x
        self.b[1] += dtx * self.mx.correction(2, ez_x, self.psi_b["yx"])
        del x_z, z_x, ex_z, ez_x
        y_x = _smooth(pads[1], 0, self.coeff)[:, :, 1:-1]
        x_y = _smooth(pads[0], 1, self.coeff)[:, 1:-1]
        ey_x, ex_y = y_x[:, :, 1:] - y_x[:, :, :-1], x_y[:, 1:] - x_y[:, :-1]
        self.b[2] -= dtx * ey_x - dty * ex_y
        self.b[2] -= dtx * self.mx.correction(2, ey_x, self.psi_b["zx"])
        self.b[2] += dty * self.my.correction(1, ex_y, self.psi_b["zy"])

    def preview(self):
        cfg, (bx, by, bz) = self.cfg, self.b
        curl = cfg.dt / (MU0 * EPS0)
        cx, cy, cz = curl / cfg.dx, curl / cfg.dy, curl / cfg.dz
        ex, ey, ez = (v.clone() for v in self.e)
        d = torch.zeros_like(ex)
        d[:, 1:-1] = bz[:, 1:] - bz[:, :-1]
        ex[1:-1, 1:-1] += cy * d[1:-1, 1:-1] - cz * (by[1:, 1:-1] - by[:-1, 1:-1])
        ex += cy * self.ey.correction(1, d, self.psi_e["xy"])
        ex[:, 0] = ex[:, -1] = 0.0
        ex[0] = self.inlet(0, self.offset, self.step_index + 1)
        d = torch.zeros_like(ey)
        d[:, :, 1:-1] = bz[:, :, 1:] - bz[:, :, :-1]
        ey[1:-1, :, 1:-1] += (cz * (bx[1:, :, 1:-1] - bx[:-1, :, 1:-1]) - cx * d[1:-1, :, 1:-1])
        ey -= cx * self.ex.correction(2, d, self.psi_e["yx"])
        ey[:, :, 0] = ey[:, :, -1] = 0.0
        ey[0] = self.inlet(1, self.offset, self.step_index + 1)
        d = torch.zeros_like(ez)
        d[:, 1:-1, 1:-1] = by[:, 1:-1, 1:] - by[:, 1:-1, :-1]
        g = torch.zeros_like(ez)
        g[:, 1:-1, 1:-1] = bx[:, 1:, 1:-1] - bx[:, :-1, 1:-1]
        ez += cx * d - cy * g
        ez += cx * self.ex.correction(2, d, self.psi_e["zx"])
        ez -= cy * self.ey.correction(1, g, self.psi_e["zy"])
        ez[:, :, 0] = ez[:, :, -1] = 0.0
        ez[:, 0] = ez[:, -1] = 0.0
        return [ex, ey, ez]

    # -- shapes: the weighted nodes of a chord
    def _visits(self, begin, end, visit):
        """visit(component, selected, (i, j, k), extents, weights) over the cut
        pieces: the weights (n, z, y, x) of the nodes from (i, j, k) on."""
        x = (begin - self.origin) / self.h
        v = (end - begin) / self.h
        lo, hi = torch.minimum(x, x + v), torch.maximum(x, x + v)
        first, last = torch.floor(lo) + 1, torch.ceil(hi) - 1
        count = torch.clamp(last - first + 1, min=0)
        most = [int(c) for c in count.amax(0)] if x.shape[0] else [0, 0, 0]
        cuts = [torch.zeros(x.shape[0], dtype=F64, device="cuda"),
                torch.ones(x.shape[0], dtype=F64, device="cuda")]
        for a in range(3):
            for c in range(most[a]):
                plane = first[:, a] + c
                t = torch.where(c < count[:, a], (plane - x[:, a]) / torch.where(
                    v[:, a] == 0, torch.ones_like(x[:, a]), v[:, a]), torch.ones_like(x[:, a]))
                cuts.append(t)
        cuts = torch.sort(torch.stack(cuts, 1), 1).values
        for s in range(cuts.shape[1] - 1):
            every = torch.nonzero(cuts[:, s + 1] > cuts[:, s])[:, 0]
            for sel in torch.split(every, 1 << 19):
                if sel.numel():
                    self._piece(x[sel], v[sel], cuts[sel, s], cuts[sel, s + 1], sel, visit)

    def _cell(self, p):
        i, j, k = (torch.floor(p[:, a]) for a in range(3))
        i = torch.where(i == self.n3[0], i - 1, i)
        j = torch.where(j == self.n3[1], j - 1, j)
        return i, j, k

    def _piece(self, x, v, first, last, sel, visit):
        width = last - first
        n = width.numel()
        if self.cfg.shape == abi.SHAPES["linear-binomial3"]:
            p = x + (0.5 * (first + last))[:, None] * v
            i, j, k = self._cell(p)
            fx, fy, fz = p[:, 0] - i, p[:, 1] - j, p[:, 2] - k
            node = lambda f: torch.stack([.25 * (1 - f), .5 - .25 * f, .25 + .25 * f,  # noqa: E731
                                          .25 * f], 1)
            wx, wy, wz = node(fx), torch.stack([1 - fy, fy], 1), node(fz)
            edge = torch.tensor([.25, .5, .25], dtype=F64, device="cuda")
            slope = torch.tensor([-.25, -.25, .25, .25], dtype=F64, device="cuda")
            sy = torch.tensor([-1., 1.], dtype=F64, device="cuda")
            c = width * width / 12.
            xy, xz, yz = c * v[:, 0] * v[:, 1], c * v[:, 0] * v[:, 2], c * v[:, 1] * v[:, 2]

            def pair(a, b, cross, sa, sb):  # (n, |a|, |b|): the two directions' weights
                return width[:, None, None] * (a[:, :, None] * b[:, None, :] +
                                               cross[:, None, None] * sa[:, None] * sb[None, :])

            i, j, k = i.long() - 1, j.long(), k.long() - 1
            w = pair(wz, wy, yz, slope, sy)
            visit(0, sel, (i, j, k), (3, 2, 4), w[:, :, :, None] * edge)
            w = pair(wz, wx, xz, slope, slope)
            visit(1, sel, (i, j, k), (4, 1, 4), w[:, :, None, :])
            w = pair(wy, wx, xy, sy, slope)
            visit(2, sel, (i, j, k), (4, 2, 3), edge[:, None, None] * w[:, None, :, :])
            return
        s3, s7 = math.sqrt(6.0 / 5.0), math.sqrt(30.0)
        nodes = [-math.sqrt(3 / 7 + 2 / 7 * s3), -math.sqrt(3 / 7 - 2 / 7 * s3),
                 math.sqrt(3 / 7 - 2 / 7 * s3), math.sqrt(3 / 7 + 2 / 7 * s3)]
        gauss = [(18 - s7) / 36, (18 + s7) / 36, (18 + s7) / 36, (18 - s7) / 36]
        for q, gw in zip(nodes, gauss):
            p = x + (.5 * (last + first + width * q))[:, None] * v
            i, j, k = self._cell(p)
            fx, fy, f = p[:, 0] - i, p[:, 1] - j, p[:, 2] - k
            factor = .5 * width * gw
            i, j, k = i.long(), j.long(), k.long() - 5
            spline = torch.ones((n, 1), dtype=F64, device="cuda")
            basis = {}
            for d in range(1, 6):
                t = torch.arange(d, dtype=F64, device="cuda")
                share = spline / d
                new = torch.zeros((n, d + 1), dtype=F64, device="cuda")
                new[:, :d] += (t + 1 - f[:, None]) * share
                new[:, 1:] += (f[:, None] + d - t - 1) * share
                spline = new
                full = torch.zeros((n, d + 7), dtype=F64, device="cuda")
                for m in range(7):
                    full[:, m:m + d + 1] += spline * _QUINTIC[m]
                basis[d] = full * factor[:, None]
            wx, wy = torch.stack([1 - fx, fx], 1), torch.stack([1 - fy, fy], 1)
            visit(0, sel, (i, j, k), (1, 2, 12), (basis[5][:, :, None] * wy[:, None, :])[..., None])
            visit(1, sel, (i, j, k), (2, 1, 12), basis[5][:, :, None, None] * wx[:, None, None, :])
            visit(2, sel, (i, j, k), (2, 2, 11),
                  basis[4][:, :, None, None] * wy[:, None, :, None] * wx[:, None, None, :])

    @staticmethod
    def _nodes(shape, low, count):
        """Flat node indices (n, cz, cy, cx) and whether they lie inside."""
        at, ok = 0, True
        for d in (2, 1, 0):  # z, y, x
            size = shape[2 - d]
            view = [-1, 1, 1, 1]
            q = low[d].view(view) + torch.arange(count[d], device="cuda").view(
                [count[d] if 2 - d == m else 1 for m in range(3)])
            ok = ok & (q >= 0) & (q < size)
            at = at * size + q.clamp(0, size - 1)
        return at, ok

    def gather(self, begin, end, s):
        n = begin.shape[0]
        out = torch.zeros((n, 3), dtype=F64, device="cuda")
        mag = torch.zeros((n, 3), dtype=F64, device="cuda")
        if n == 0:
            return out, mag
        if n > 1 << 19:
            parts = [self.gather(b, e, s) for b, e in zip(torch.split(begin, 1 << 19),
                                                          torch.split(end, 1 << 19))]
            return tuple(torch.cat(t) for t in zip(*parts))
        # the chord's part inside the domain (a chord may leave it above)
        x = (begin - self.origin) / self.h
        v = (end - begin) / self.h
        size = torch.tensor([float(m) for m in self.n3], dtype=F64, device="cuda")
        safe = torch.where(v == 0, torch.ones_like(v), v)
        t0, t1 = -x / safe, (size - x) / safe
        lo = torch.where(v == 0, torch.zeros_like(v), torch.minimum(t0, t1)).amax(1).clamp(min=0.)
        hi = torch.where(v == 0, torch.ones_like(v), torch.maximum(t0, t1)).amin(1).clamp(max=1.)
        b, e = begin + lo[:, None] * (end - begin), begin + hi[:, None] * (end - begin)
        b, e = torch.where((lo == 0)[:, None], begin, b), torch.where((hi == 1)[:, None], end, e)

        def visit(d, sel, low, count, w):
            at, ok = self._nodes(s[d].shape, low, count)
            out[:, d].index_add_(0, sel, (.5 * w * ok * s[d].view(-1)[at]).sum((1, 2, 3)))

        self._visits(b, e, visit)
        out *= (hi - lo)[:, None]
        p = (0.5 * (b + e) - self.origin) / self.h
        wide = self.cfg.shape == abi.SHAPES["linear-binomial3"]
        for a in range(3):
            shift = torch.tensor([0. if a == d else .5 for d in range(3)], dtype=F64, device="cuda")
            c = torch.floor(p - shift)
            f = p - shift - c
            c = c.long()
            lin = lambda g: [1 - g, g]  # noqa: E731
            node = lambda g: [.25 * (1 - g), .5 - .25 * g, .25 + .25 * g, .25 * g]  # noqa: E731
            wx, wz = (node(f[:, 0]), node(f[:, 2])) if wide else (lin(f[:, 0]), lin(f[:, 2]))
            wy, o = lin(f[:, 1]), 1 if wide else 0
            low = (c[:, 0] - o, c[:, 1], c[:, 2] - o)
            at = 0
            for d, m in ((2, len(wz)), (1, 2), (0, len(wx))):
                size = self.b[a].shape[2 - d]
                q = low[d].view(-1, 1, 1, 1) + torch.arange(m, device="cuda").view(
                    [m if 2 - d == t else 1 for t in range(3)])
                at = at * size + q.clamp(0, size - 1)
            wx, wy, wz = (torch.stack(t, 1) for t in (wx, wy, wz))
            mag[:, a] = (wz[:, :, None, None] * wy[:, None, :, None] * wx[:, None, None, :] *
                         self.b[a].view(-1)[at]).sum((1, 2, 3))
        return out, mag

    def deposit(self, j, begin, end, q):
        cfg = self.cfg
        scale = q[:, None] * (end - begin) / (cfg.dx * cfg.dy * cfg.dz * cfg.dt)

        def visit(d, sel, low, count, w):
            at, ok = self._nodes(j[d].shape, low, count)
            j[d].view(-1).index_add_(0, at.reshape(-1),
                                     (scale[sel, d].view(-1, 1, 1, 1) * w * ok).reshape(-1))

        if begin.shape[0]:
            self._visits(begin, end, visit)

    # -- push
    def prescribed_fields(self, point, time):
        cfg = self.cfg
        lab = cfg.lab_z_origin + cfg.boost_gamma_beta * C * time + cfg.boost_gamma * (
            point[:, 2] - cfg.box_z_origin)
        bl = torch.zeros_like(point)
        for m in self.prescribed:
            z = lab - m.center[2]
            on = ((z >= 0) & (z <= m.length)).to(F64)
            if m.type == abi.MAGNET_UNIFORM_DIPOLE:
                bl[:, 0] += on * m.peak_field * m.cos_angle
                bl[:, 1] += on * m.peak_field * m.sin_angle
            else:
                k = m.wave_number
                tc = point[:, 0] * m.cos_angle + point[:, 1] * m.sin_angle
                tf = on * m.peak_field * torch.cosh(k * tc) * torch.sin(k * z)
                bl[:, 0] += tf * m.cos_angle
                bl[:, 1] += tf * m.sin_angle
                bl[:, 2] += on * m.peak_field * torch.sinh(k * tc) * torch.cos(k * z)
        gb = cfg.boost_gamma_beta
        e = torch.stack([-gb * C * bl[:, 1], gb * C * bl[:, 0], torch.zeros_like(lab)], 1)
        b = torch.stack([cfg.boost_gamma * bl[:, 0], cfg.boost_gamma * bl[:, 1], bl[:, 2]], 1)
        return e, b

    def push(self, pos, u, q, m, time, dt, e, b):
        """Lapenta-Markidis: the mean gamma of the step from its scalar root."""
        g0 = torch.sqrt(1 + (u * u).sum(1))
        ee, bb = self.prescribed_fields(pos + (.5 * dt * C / g0)[:, None] * u, time + .5 * dt)
        kick = (q * dt / (2 * m * C))[:, None] * (e + ee)
        bv = (q * dt / (2 * m))[:, None] * (b + bb)
        a = u + kick
        axb = torch.cross(a, bv, dim=1)
        dot = lambda s, t: (s * t).sum(1)  # noqa: E731
        b2, ka, ab, kc, kb = dot(bv, bv), dot(kick, a), dot(a, bv), dot(kick, axb), dot(kick, bv)
        first = dot(kick, u) / g0
        g = g0 + first + (dot(kick, kick) + kc / g0 - first * first) / g0
        g = torch.maximum(g, .5 * (g0 + 1))
        for _ in range(8):
            den, num = g * g + b2, g * g * ka + g * kc + ab * kb
            f = g * (g - g0) - num / den
            df = 2 * g - g0 - ((2 * g * ka + kc) * den - 2 * g * num) / (den * den)
            g = torch.maximum(g - f / df, .5 * (g0 + 1))
        den = (g * g + b2)[:, None]
        new = 2 * ((g * g)[:, None] * a + ab[:, None] * bv + g[:, None] * axb) / den - u
        g1 = torch.sqrt(1 + (new * new).sum(1))
        return pos + (dt * C / (g0 + g1))[:, None] * (u + new), new

    def lab_z(self, z, t):
        cfg = self.cfg
        return cfg.lab_z_origin + cfg.boost_gamma_beta * C * t + cfg.boost_gamma * (
            z - cfg.box_z_origin)

    def trial(self, j, e_used, b_used):
        """One trial: J, the new state and the carriers it leaves; without J
        only where each push starts and which particles are pushed."""
        cfg, p = self.cfg, self.p
        t, dt = self.time, cfg.dt
        upper = self.origin[2] + cfg.nz * cfg.dz
        kept = {"pos": [], "vel": [], "q": []}

        def carry(start, end, vel, q):
            f = torch.where(end[:, 2] > upper, (upper - start[:, 2]) / (end[:, 2] - start[:, 2]),
                            torch.ones_like(q))
            stop = start + f[:, None] * (end - start)
            self.deposit(j, start, stop, q)
            stays = end[:, 2] <= upper
            kept["pos"].append(end[stays])
            kept["vel"].append(vel[stays])
            kept["q"].append(q[stays])

        if j is not None:
            c = self.carriers
            carry(c["pos"], c["pos"] + dt * c["vel"], c["vel"], c["q"])
        if self.queue is not None and j is not None:
            inc = C * dt * self.queue["beta"]
            near = (self.due > self.step_index) & (self.due <= self.step_index + 8)
            at = self.queue["pos"][near].clone()
            at[:, 2] += self.step_index * inc[near]
            to = at.clone()
            to[:, 2] += inc[near]
            self.deposit(j, at, to, self.queue["q"][near])
        start, u, frozen = p["pos"], p["u"], p["frozen"]
        held_z = start[:, 2] + C * dt * p["beta"]
        a0, a1 = self.lab_z(start[:, 2], t), self.lab_z(held_z, t + dt)
        plane = cfg.activation_plane_lab_z
        released = frozen & (a1 >= plane)
        crossing = torch.where(released, torch.clamp((plane - a0) / torch.where(
            released, a1 - a0, torch.ones_like(a0)), 0., 1.), torch.zeros_like(a0))
        kink = start.clone()
        kink[:, 2] = torch.where(released, start[:, 2] + C * crossing * dt * p["beta"], start[:, 2])
        time = t + crossing * dt
        span = (1. - crossing) * dt
        pushed = (~frozen | released) & (span > 0)
        if j is None:
            return kink, pushed
        pos, new = kink.clone(), u.clone()
        moved, unew = self.push(kink[pushed], u[pushed], p["q"][pushed], p["m"][pushed],
                                time[pushed], span[pushed], e_used[pushed], b_used[pushed])
        pos[pushed], new[pushed] = moved, unew
        stays_held = frozen & ~released
        pos[:, 2] = torch.where(stays_held, held_z, pos[:, 2])
        if bool(released.any()):
            self.deposit(j, start[released], kink[released], p["q"][released])
        za = self.lab_z(kink[:, 2], time) - cfg.exit_lab_z
        zb = self.lab_z(pos[:, 2], t + dt) - cfg.exit_lab_z
        exits = (zb >= 0) & (zb > za)
        f = torch.where(exits, -za / torch.where(exits, zb - za, torch.ones_like(za)),
                        torch.ones_like(za))
        hit = torch.where(exits[:, None], kink + f[:, None] * (pos - kink), pos)
        self.deposit(j, kink, hit, p["q"])
        if bool(exits.any()):
            g = torch.sqrt(1 + (new[exits] ** 2).sum(1))
            carry(hit[exits], pos[exits], new[exits] * (C / g)[:, None], p["q"][exits])
        carriers = {k: torch.cat(v) for k, v in kept.items()}
        return kink, pos, new, stays_held, pushed, ~exits, carriers

    def step(self):
        cfg = self.cfg
        if self.queue is not None:
            now = self.due == self.step_index
            if bool(now.any()):
                new = {k: v[now].clone() for k, v in self.queue.items()}
                new["pos"][:, 2] += self.step_index * C * cfg.dt * new["beta"]
                self.p = {k: torch.cat([self.p[k], new[k]]) for k in self.p}
        self.magnetic()
        star = self.preview()
        p = self.p
        n = p["q"].numel()
        zeros = torch.zeros((n, 3), dtype=F64, device="cuda")
        j = [torch.zeros_like(v) for v in self.e]
        jcoef = -cfg.dt / EPS0
        if n:
            g = torch.sqrt(1 + (p["u"] ** 2).sum(1))
            kink, pushed = self.trial(None, zeros, zeros)
            span = cfg.dt * torch.ones_like(g)
            part = p["frozen"] & pushed
            if bool(part.any()):
                a0 = self.lab_z(p["pos"][:, 2], self.time)
                a1 = self.lab_z(p["pos"][:, 2] + C * cfg.dt * p["beta"], self.time + cfg.dt)
                cross = torch.clamp((cfg.activation_plane_lab_z - a0) / (a1 - a0), 0., 1.)
                span = torch.where(part, (1 - cross) * cfg.dt, span)
            guess = kink + (span * C / g)[:, None] * p["u"]
            e, b = zeros.clone(), zeros.clone()
            s = [x + y for x, y in zip(star, self.e)]
            e[pushed], b[pushed] = self.gather(kink[pushed], guess[pushed], s)
        else:
            e = b = zeros
        for trial in range(cfg.max_trials):
            for v in j:
                v.zero_()
            kink, pos, new, held, pushed, kept, carriers = self.trial(j, e, b)
            cand = [v.clone() for v in star]
            cand[0][1:-1, 1:-1] += jcoef * j[0][1:-1, 1:-1]
            cand[1][1:-1, :, 1:-1] += jcoef * j[1][1:-1, :, 1:-1]
            cand[2][:, 1:-1, 1:-1] += jcoef * j[2][:, 1:-1, 1:-1]
            if not n:
                break
            s = [x + y for x, y in zip(cand, self.e)]
            e2, b2 = zeros.clone(), zeros.clone()
            e2[pushed], b2[pushed] = self.gather(kink[pushed], pos[pushed], s)
            force = ((p["q"] / p["m"]).abs() * cfg.dt / C * ((e2 - e).norm(dim=1) +
                                                           C * (b2 - b).norm(dim=1))).max()
            chord = pos - kink
            defect = (p["q"] * ((e2 - e) * chord).sum(1)).abs().sum()
            scale = ((p["q"] * (e * chord).sum(1)).abs() + (p["q"] * (e2 * chord).sum(1)).abs()).sum()
            e, b = e2, b2
            if trial >= 1 and float(force) < 1e-13 and float(defect) < 1e-8 * float(scale):
                break
        self.e = cand
        if n:
            p = dict(p, pos=pos, u=new, frozen=held)
            self.p = {k: v[kept] for k, v in p.items()}
        self.carriers = carriers
        # the window moves one cell
        self.time += cfg.dt
        self.step_index += 1
        self.offset = cfg.initial_offset - self.step_index
        for group, first in ((self.e, 0), (self.b, 3)):
            for a in range(3):
                group[a][1:] = group[a][:-1].clone()
                group[a][0] = self.inlet(first + a, self.offset, self.step_index)
        for psi in list(self.psi_b.values()) + list(self.psi_e.values()):
            psi[1:] = psi[:-1].clone()
            psi[0] = 0.0
        self.origin[2] = cfg.reference_origin[2] + self.offset * cfg.dz
        stays = self.carriers["pos"][:, 2] < self.origin[2] + cfg.nz * cfg.dz
        self.carriers = {k: v[stays] for k, v in self.carriers.items()}

    def plane(self, lab_z):
        cfg = self.cfg
        z = cfg.box_z_origin + (lab_z - cfg.lab_z_origin) / cfg.boost_gamma - (
            cfg.boost_beta * C * self.time)
        z = (z - float(self.origin[2])) / cfg.dz

        def sample(v, pos):
            out = v
            for dim, (at, n) in enumerate(zip(pos, v.shape)):
                at = torch.as_tensor(at, dtype=F64, device="cuda").reshape(-1).clamp(0, n - 1)
                lo = torch.floor(at).long().clamp(max=n - 2)
                f = (at - lo).reshape([-1 if q == dim else 1 for q in range(3)])
                out = out.index_select(dim, lo) * (1 - f) + out.index_select(dim, lo + 1) * f
            return out[0]

        x = torch.arange(cfg.nx, dtype=F64, device="cuda") + .5
        y = torch.arange(cfg.ny, dtype=F64, device="cuda") + .5
        (ex, ey, ez), (bx, by, bz) = self.e, self.b
        near = max(0, int(math.floor(z)) - 2)
        cut = [v[near:near + 6] for v in (ex, ey, ez, bx, by, bz)]
        z -= near
        ex, ey, ez = sample(cut[0], (z, y, x - .5)), sample(cut[1], (z, y - .5, x)), sample(
            cut[2], (z - .5, y, x))
        bx, by, bz = sample(cut[3], (z - .5, y - .5, x)), sample(cut[4], (z - .5, y, x - .5)), sample(
            cut[5], (z, y - .5, x - .5))
        g, gb = cfg.boost_gamma, cfg.boost_gamma_beta
        return torch.stack([g * ex + gb * C * by, g * ey - gb * C * bx, ez,
                            g * bx - gb / C * ey, g * by + gb / C * ex, bz], -1).cpu().numpy()


def _quintic_coefficients():
    p = 5.0
    a = p / 6
    b = 3 * p / 40 + p * (p - 1) / 72
    d = 5 * p / 112 + p * (p - 1) / 80 + p * (p - 1) * (p - 2) / 1296
    half = [-d / 64, b / 16 + 3 * d / 32, -a / 4 - b / 4 - 15 * d / 64]
    return half + [1 + a / 2 + 3 * b / 8 + 5 * d / 16] + half[::-1]


_QUINTIC = _quintic_coefficients()


def _exact_self_field(cfg, particles):
    """CIC charge, the Cowan Poisson problem by sine transforms, E and B."""
    n3 = (cfg.nx, cfg.ny, cfg.nz)
    h = (cfg.dx, cfg.dy, cfg.dz)
    alpha, beta, delta = _cowan(*h)
    t = {k: torch.tensor(particles[k], device="cuda") for k in
         ("x", "y", "z", "ux", "uy", "uz", "charge", "mass")}
    gamma = torch.sqrt(1 + t["ux"] ** 2 + t["uy"] ** 2 + t["uz"] ** 2)
    bz = float((t["mass"] * t["uz"] / gamma).sum() / t["mass"].sum())
    rho = torch.zeros([m + 1 for m in n3[::-1]], dtype=F64, device="cuda")
    cells, frac = [], []
    for a, k in enumerate("xyz"):
        start = cfg.reference_origin[a] + (cfg.initial_offset * cfg.dz if a == 2 else 0.0)
        p = (t[k] - start) / h[a]
        c = torch.floor(p).clamp(0, n3[a] - 1)
        cells.append(c.long())
        frac.append(p - c)
    for c in range(2):
        for b in range(2):
            for a in range(2):
                w = t["charge"] / (h[0] * h[1] * h[2])
                for f, o in zip(frac, (a, b, c)):
                    w = w * (f if o else 1 - f)
                at = ((cells[2] + c) * (n3[1] + 1) + cells[1] + b) * (n3[0] + 1) + cells[0] + a
                rho.view(-1).index_add_(0, at, w)
    lo = (cfg.cpml_cells_x, cfg.cpml_cells_y, 0)
    inner = tuple(slice(lo[a] + 1, n3[a] - lo[a]) for a in (2, 1, 0))
    f = rho[inner] / EPS0
    tables, theta = [], []
    for a in (2, 1, 0):
        m = n3[a] - 2 * lo[a]
        k = torch.arange(1, m, dtype=F64, device="cuda")
        tables.append(torch.sin(math.pi * ((k[:, None] * k[None, :]) % (2 * m)) / m))
        theta.append(math.pi * k / m)
    cz, cy, cx = (torch.cos(v) for v in theta)
    cos = [cx[None, None, :], cy[None, :, None], cz[:, None, None]]
    translation = (bz * C) ** 2 * EPS0 * MU0
    symbol = 0.0
    for a in range(3):
        u, v = (a + 1) % 3, (a + 2) % 3
        s = alpha[a] + 2 * beta[u] * cos[u] + 2 * beta[v] * cos[v] + 4 * delta[a] * cos[u] * cos[v]
        symbol = symbol + (s - (translation if a == 2 else 0.0)) * (2 - 2 * cos[a]) / h[a] ** 2

    def transform(v):
        v = torch.einsum("pk,kji->pji", tables[0], v)
        v = torch.einsum("qj,pji->pqi", tables[1], v)
        return torch.einsum("ri,pqi->pqr", tables[2], v)

    phi_in = transform(transform(f) / symbol)
    for table in tables:
        phi_in *= 2.0 / (table.shape[0] + 1)
    phi = torch.zeros([m + 3 for m in n3[::-1]], dtype=F64, device="cuda")
    phi[1:-1, 1:-1, 1:-1][inner] = phi_in
    e = []
    for a in range(3):
        s = _smooth(phi, a, (alpha, beta, delta))
        s = s.narrow(2 - a, 1, s.shape[2 - a] - 2).clone()
        if a == 2:
            s -= translation * phi[1:-1, 1:-1, 1:-1]
        mask = torch.zeros_like(s)
        mask[inner] = 1.0
        s = s * mask
        dim = 2 - a
        e.append(-(s.narrow(dim, 1, n3[a]) - s.narrow(dim, 0, n3[a])) / h[a])
    scale = bz * C * EPS0 * MU0
    up = .5 + .5 * bz * C * cfg.dt / cfg.dz
    b = [-scale * ((1 - up) * e[1][:-1] + up * e[1][1:]), scale * ((1 - up) * e[0][:-1] + up * e[0][1:]),
         torch.zeros((n3[2] + 1, n3[1], n3[0]), dtype=F64)]
    return {"fields": [v.cpu().numpy() for v in e + b]}


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "selffield":
            cfg, particles, _, _ = _inputs(case, seed)
            return _exact_self_field(cfg, particles)
        if case["kind"] == "scan":
            planes = []
            for job, (cfg, particles, frozen, table) in _jobs(case, seed):
                box = _Box(cfg, particles, frozen, table)
                for _ in range(job["steps"]):
                    box.step()
                planes.append(box.plane(workloads.detector_plane_lab_z(cfg)).ravel())
            return {"planes": planes, "particles": [None] * len(planes)}
        cfg, particles, frozen, table = _inputs(case, seed)
        box = _Box(cfg, particles, frozen, table)
        planes = []
        for n in range(1, case["steps"] + 1):
            box.step()
            if n % case["detector_every"] == 0 or n == case["steps"]:
                planes.append(box.plane(workloads.detector_plane_lab_z(cfg)))
        p = box.p
        got = {"x": p["pos"][:, 0], "y": p["pos"][:, 1], "z": p["pos"][:, 2], "ux": p["u"][:, 0],
               "uy": p["u"][:, 1], "uz": p["u"][:, 2], "charge": p["q"], "mass": p["m"]}
        out = {"planes": planes, "particles": {k: v.cpu().numpy() for k, v in got.items()},
               "carriers": None}
        out["particles"]["id"] = p["id"].to(torch.int64).cpu().numpy()
        if case["fields"]:
            out["fields"] = [v.cpu().numpy() for v in box.e + box.b]
        if case["ledger"]:
            out["ledger"] = None
        return out
