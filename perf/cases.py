"""Performance cases of the quasi-static slice loop.

Every case is a call that a program driving this framework makes through its Python interface (or,
for the Poisson solve, its C ABI): whole time steps on small, ordinary and large grids, both
precisions, both Bx/By solvers, the per-slice surface, the gradient of one step, and the
allocation-free Poisson solve. A pass of a step case hands the step its beam from pinned host
memory, runs the step from time 0 and reads the pushed beam, the last slice's fields and the y = 0
plane of the wake back, as a program that couples the slice loop to its own beam transport does; a
pass therefore starts from the same state every time.
"""
import ctypes
import math

import numpy as np
import torch

import hipace2_b200 as hp

BEAM = ("x", "y", "z", "w", "ux", "uy", "uz")
LAST_SLICE = ("Ez", "Psi", "Bx", "By", "EypBx", "ExmBy")
PLANES = ("Ez", "ExmBy", "By")


def _step(name, nx, ny, nz, **over):
    """A step case: the driver of the framework's blowout workload on an nx x ny x nz grid."""
    case = {"name": name, "kind": "step", "nx": nx, "ny": ny, "nz": nz, "precision": "fp64",
            "solver": "explicit", "half_width": 6.0, "zeta_lo": -8.0, "zeta_hi": 4.0, "dt": 20.0,
            "beam_particles": 1000000, "beam_density": 10.0, "beam_sigma": 0.3, "gamma": 2000.0,
            "channel": 0.0, "ppc": 1, "tolerance": 1e-4, "z_push": True}
    case.update(over)
    return case


def listed():
    return [
        # the smallest calls: one Poisson solve on a coarse grid inside a caller's own loop
        {"name": "poisson_63", "kind": "poisson", "nx": 63, "ny": 63},
        # the same solve on the largest grid that the entry point takes
        {"name": "poisson_1023", "kind": "poisson", "nx": 1023, "ny": 1023},
        # a coarse weak-wake run driven slice by slice (a coupled code between the slices), tight
        # multigrid tolerance
        _step("slices_63", 63, 63, 48, kind="slices", beam_particles=20000, beam_density=0.5,
              beam_sigma=0.5, tolerance=1e-10),
        # the same run in single precision: FP64-refined multigrid (tolerance below 1e-5)
        _step("slices_63_mixed", 63, 63, 48, kind="slices", precision="mixed", beam_particles=20000,
              beam_density=0.05, beam_sigma=0.5, tolerance=1e-10, z_push=False),
        # the linear-wake deck: predictor-corrector solver, even grid (no fast transform length)
        _step("linear_wake_64", 64, 64, 100, solver="pc", half_width=8.0, zeta_lo=-12.0, zeta_hi=6.0,
              dt=10.0, beam_particles=100000, beam_density=0.01, beam_sigma=0.5, gamma=1000.0),
        # a ragged production grid: non-square, even (cell-centred multigrid), sizes of the form 3 * 2^n
        # and 5 * 2^n, outside the fast transform lengths
        _step("ragged_384x320", 384, 320, 48, beam_particles=300000),
        # the headline run: nonlinear blowout, 255^2 x 256 slices, 1e6 beam particles, FP64 ...
        _step("blowout_255", 255, 255, 256),
        # ... and in mixed precision (a box that ends inside the bubble, where FP32 rounding is not yet
        # amplified, and no slippage of the driver)
        _step("blowout_255_mixed", 255, 255, 256, precision="mixed", zeta_lo=-4.0, z_push=False),
        # a plasma channel on a fine grid with 2 x 2 particles per cell
        _step("channel_1023", 1023, 1023, 128, half_width=8.0, zeta_lo=-3.0, zeta_hi=3.0, channel=0.05,
              ppc=2, beam_particles=500000),
        _step("channel_1023_mixed", 1023, 1023, 128, precision="mixed", half_width=8.0, zeta_lo=-3.0,
              zeta_hi=3.0, channel=0.05, ppc=2, beam_particles=500000, z_push=False),
        # the largest grid of the framework's own configurations, in the precision it is run in
        _step("large_2047_mixed", 2047, 2047, 64, precision="mixed", half_width=10.0, zeta_lo=-3.0,
              zeta_hi=3.0, beam_particles=500000, z_push=False),
        # the backward direction: gradient of the beam-loading objective on 64 + 8 knots
        _step("gradient_255", 255, 255, 128, kind="gradient", zeta_lo=-10.0, beam_density=2.0,
              beam_particles=300000),
    ]


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithm, odd ones among them."""
    kind = rng.choice(("poisson", "slices", "step", "step", "step", "step", "gradient"))
    if kind == "poisson":
        n = (31, 63, 127, 255, 511, 1023)
        return {"kind": kind, "nx": rng.choice(n), "ny": rng.choice(n)}
    mixed = kind != "gradient" and rng.random() < 0.5
    even = rng.random() < 0.25

    def size(lo, hi):
        # m 2^k, less one for a node-centred grid: the sizes that the multigrid coarsens well
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        k = max(0, round(math.log2(n / 6.0)))
        m = min(8, max(4, round(n / 2 ** k)))
        return m * 2 ** k - (0 if even else 1)

    top = {"slices": 127, "step": 1023, "gradient": 255}[kind]
    nx = size(31, top)
    ny = size(max(31, nx // 2), nx)
    cells = nx * ny
    most = {"slices": 64, "step": 256, "gradient": 128}[kind]
    most = min(most, max(24, int(128 * 1023 ** 2 / (2 * cells))))
    nz = int(math.exp(rng.uniform(math.log(24), math.log(most + 1))))
    solver = "pc" if kind == "step" and cells < 20000 and rng.random() < 0.25 else "explicit"
    dens = math.exp(rng.uniform(math.log(0.01), math.log(0.2 if solver == "pc" else 2.0 if kind == "gradient" else 10.0)))
    return dict(_step("", nx, ny, nz), kind=kind, precision="mixed" if mixed else "fp64", solver=solver,
                half_width=rng.choice((6.0, 8.0)), beam_density=dens, zeta_lo=-10.0 if kind == "gradient" else -4.0 if mixed else -8.0,
                beam_sigma=0.5, beam_particles=int(math.exp(rng.uniform(math.log(2e4), math.log(1e6)))),
                channel=rng.choice((0.0, 0.05)), ppc=rng.choice((1, 1, 2)), tolerance=rng.choice((1e-4, 1e-4, 1e-10)),
                z_push=not mixed)


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _deck(c):
    gradient = c["kind"] == "gradient"
    channel = " + %g*(x*x+y*y)" % c["channel"] if c["channel"] else ""
    pc = c["solver"] == "pc"
    lines = ["amr.n_cell = %d %d %d" % (c["nx"], c["ny"], c["nz"]),
             "hipace.normalized_units = 1", "max_step = 0", "hipace.dt = %g" % c["dt"],
             "hipace.MG_tolerance_rel = %g" % c["tolerance"],
             "boundary.field = Dirichlet", "boundary.particle = %s" % ("Periodic" if pc else "Reflecting"),
             "geometry.prob_lo = %g %g %g" % (-c["half_width"], -c["half_width"] * c["ny"] / c["nx"], c["zeta_lo"]),
             "geometry.prob_hi = %g %g %g" % (c["half_width"], c["half_width"] * c["ny"] / c["nx"], c["zeta_hi"]),
             "diagnostic.diag_type = xz", "random_seed = 1",
             "plasmas.names = plasma", "plasma.density(x,y,z) = 1.%s" % channel,
             "plasma.ppc = %d %d" % (c["ppc"], c["ppc"]), "plasma.element = electron",
             "beams.names = driver" + (" witness" if gradient else "")]
    if pc:
        lines += ["hipace.bxby_solver = predictor-corrector", "hipace.predcorr_max_iterations = 3",
                  "hipace.predcorr_B_error_tolerance = -1"]
    for b in ("driver", "witness")[:2 if gradient else 1]:
        # the particles themselves come from set_beam
        lines += [b + ".injection_type = fixed_weight", b + ".num_particles = 1",
                  b + ".position_mean = 0. 0. 0.", b + ".position_std = 0.3 0.3 1.",
                  b + ".density = 1.", b + ".u_mean = 0. 0. %g" % c["gamma"],
                  b + ".do_z_push = %d" % c["z_push"]]
    if gradient:
        lines += ["adjoint.witness = witness", "adjoint.profile_zeta = -7. -5.", "adjoint.n_profile_knots = 64",
                  "adjoint.density_z = -100. 100.", "adjoint.n_density_knots = 8",
                  "adjoint.objective_zeta = -7. -5.", "adjoint.checkpoint_interval = 32"]
    return "\n".join(lines) + "\n"


def _weight(c, density, n, sx, sy, length):
    """Weight of one of n particles of a Gaussian (transversely) beam, in units of one cell's charge."""
    cell = (2 * c["half_width"] / c["nx"]) ** 2 * (c["zeta_hi"] - c["zeta_lo"]) / c["nz"]
    return density * 2 * math.pi * sx * sy * length / (n * cell)


def _driver(c, rng):
    n, s = c["beam_particles"], c["beam_sigma"]
    u = 0.01 / s
    z = rng.normal(0, 1.0, n)
    # inside the box, ahead of its last slice (out of which particles slip and are lost)
    lo = c["zeta_lo"] + (c["zeta_hi"] - c["zeta_lo"]) / c["nz"]
    while (out := (z < lo) | (z >= c["zeta_hi"])).any():
        z[out] = rng.normal(0, 1.0, int(out.sum()))
    return {"x": rng.normal(0, s, n), "y": rng.normal(0, s, n), "z": z,
            "w": np.full(n, _weight(c, c["beam_density"], n, s, s, math.sqrt(2 * math.pi))),
            "ux": rng.normal(0, u, n), "uy": rng.normal(0, u, n), "uz": np.full(n, c["gamma"]),
            "id": np.arange(1, n + 1, dtype=np.int64)}


def _witness(c, rng):
    n = max(1, c["beam_particles"] // 2)
    return {"x": rng.normal(0, 0.1, n), "y": rng.normal(0, 0.1, n), "z": rng.uniform(-7.0, -5.0, n),
            "w": np.full(n, _weight(c, 5.0, n, 0.1, 0.1, 2.0)), "ux": np.zeros(n), "uy": np.zeros(n),
            "uz": np.full(n, c["gamma"]), "id": np.arange(1, n + 1, dtype=np.int64)}


def _beams(c, seed):
    rng = np.random.default_rng(seed)
    return [_driver(c, rng)] + ([_witness(c, rng)] if c["kind"] == "gradient" else [])


def _knots(c, seed):
    rng = np.random.default_rng([seed, 1])
    return np.concatenate([0.5 * (1 + 0.1 * rng.uniform(-1, 1, 64)), 1 + 0.02 * rng.uniform(-1, 1, 8)])


def _rhs(c, seed):
    """A charge-like right-hand side: a Gaussian blob on noise (unit square)."""
    rng = np.random.default_rng(seed)
    x = (np.arange(c["nx"]) + 1) / (c["nx"] + 1) - rng.uniform(0.4, 0.6)
    y = (np.arange(c["ny"]) + 1) / (c["ny"] + 1) - rng.uniform(0.4, 0.6)
    return np.exp(-(y[:, None] ** 2 + x[None, :] ** 2) / 0.02) + 0.1 * rng.standard_normal((c["ny"], c["nx"]))


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.int64 if a.dtype == np.int64 else torch.float64,
                    pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t.numpy()


def prepare(case, seed):
    c = case
    if c["kind"] == "poisson":
        f = torch.from_numpy(_rhs(c, seed)).cuda()
        return {"case": c, "f": f, "u": torch.empty_like(f), "lib": hp.load_library()}
    sim = hp.Hipace(_deck(c), precision=hp.MIXED if c["precision"] == "mixed" else hp.PLAIN_FP64)
    sim.init_data()
    state = {"case": c, "sim": sim}
    if c["kind"] == "gradient":
        for b, beam in enumerate(_beams(c, seed)):
            sim.set_beam(b, beam)
        state["knots"] = _knots(c, seed)
        return state
    sim.set_diag(PLANES)
    beam = _beams(c, seed)[0]
    state["beam"] = {k: _pinned(v) for k, v in beam.items()}
    state["out"] = {k: _pinned(np.zeros_like(v)) for k, v in beam.items()}
    return state


def run(state):
    c = state["case"]
    if c["kind"] == "poisson":
        f, u = state["f"], state["u"]
        rc = state["lib"].hpq_poisson_dirichlet_noalloc(
            f.data_ptr(), u.data_ptr(), c["nx"], c["ny"], 1.0 / (c["nx"] + 1), 1.0 / (c["ny"] + 1),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise hp.HpqError(rc, "Poisson solve")
        return u
    sim = state["sim"]
    if c["kind"] == "gradient":
        objective, gradient = sim.adjoint(state["knots"])
        return {"objective": objective, "gradient": gradient}
    sim.set_time(0.0)
    sim.set_beam(0, state["beam"])
    if c["kind"] == "slices":
        sim.begin_step(0)
        for islice in range(c["nz"] - 1, -1, -1):
            sim.solve_one_slice(islice)
        sim.end_step()
    else:
        sim.step(0)
    beam = sim.get_beam(0, out=state["out"])
    return {"beam": beam, "slice": {k: sim.get_field(k) for k in LAST_SLICE},
            "plane": {k: sim.get_diag(k) for k in PLANES}}


# ------------------------------------------------------------------------------------------
# work and tolerance
# ------------------------------------------------------------------------------------------
def work(case):
    """Bytes and operations of one pass. Poisson solve: f read, u written, two sine transforms per
    axis. A slice: its plasma particles' state (6 reals) read and 5 of them written once, the ten
    field planes written and read once, the beam particles read and written once per step (host
    and device); about 1500 operations per plasma particle (deposits, gather, push), 420 per cell
    for three V-cycles of two components, the transforms of three (predictor-corrector: 9)
    Poisson solves, and 3000 per beam particle (10 sub-cycles). A gradient: the march forward
    twice (once recomputed) and its reverse, about as much again per kernel."""
    c = case
    nx, ny = c["nx"], c["ny"]
    dst = 10.0 * nx * ny * (math.log2(2 * (nx + 1)) + math.log2(2 * (ny + 1)))
    if c["kind"] == "poisson":
        return {"bytes": 16.0 * nx * ny, "flops": dst}
    real = 4 if c["precision"] == "mixed" else 8
    plasma, cells, nz, nb = nx * ny * c["ppc"] ** 2, nx * ny, c["nz"], c["beam_particles"]
    pc = c["solver"] == "pc"
    flops = nz * (plasma * (3000.0 if pc else 1500.0) + (9 if pc else 3) * dst + (0 if pc else 420.0) * cells)
    data = nz * real * (11.0 * plasma + 20.0 * cells)
    if c["kind"] == "gradient":
        return {"bytes": 4 * data, "flops": 4 * flops}
    return {"bytes": data + 2 * 64.0 * nb, "flops": flops + 3000.0 * nb}


def tolerance(case):
    """Relative 2-norm. The march amplifies rounding from slice to slice: two FP64 runs, whose atomics
    add in another order, differ by up to 1.4e-10 behind a strong driver; two single-precision runs by
    up to 9e-5, and by several times that where a transform or a solver rounds differently. The Poisson
    solve alone is 2e-15 from the dense transform."""
    c = case
    if c["kind"] == "poisson":
        return {"rel": 2e-14}
    if c["kind"] == "gradient":
        return {"rel": 1e-7}
    if c["precision"] == "fp64":
        return {"rel": 1e-9}
    return {"rel": 2e-3}


# ------------------------------------------------------------------------------------------
# the same results in 64 bits from plain torch
# ------------------------------------------------------------------------------------------
G = 3  # guard cells of the slice planes


def _sine(n, like):
    k = torch.arange(1, n + 1, dtype=torch.float64, device=like.device)
    return torch.sin(torch.outer(k, k) * (math.pi / (n + 1)))


class _Poisson:
    """Lap(u) = f with u = 0 one cell outside, by dense sine matrices; shift: Lap - shift."""

    def __init__(self, nx, ny, dx, dy, device):
        z = torch.empty(0, dtype=torch.float64, device=device)
        self.sx, self.sy = _sine(nx, z), _sine(ny, z)
        ex = torch.sin(torch.arange(1, nx + 1, device=device, dtype=torch.float64) * (math.pi / (2 * (nx + 1)))) ** 2
        ey = torch.sin(torch.arange(1, ny + 1, device=device, dtype=torch.float64) * (math.pi / (2 * (ny + 1)))) ** 2
        self.eig = -4 * (ey[:, None] / dy ** 2 + ex[None, :] / dx ** 2)
        self.norm = (2.0 / (nx + 1)) * (2.0 / (ny + 1))

    def __call__(self, f, shift=0.0):
        t = self.sy @ f @ self.sx
        return self.sy @ (t * (self.norm / (self.eig - shift))) @ self.sx


def _shape2(t):
    """Quadratic shape: first cell and three weights."""
    c = torch.floor(t + 0.5)
    d = t - c
    return c.long() - 1, torch.stack([0.5 * (0.5 - d) ** 2, 0.75 - d * d, 0.5 * (0.5 + d) ** 2])


def _shape2_nodal(t):
    """Quadratic shape on four points with the derivative between nodes: first cell, weights, derivatives."""
    c = torch.floor(t)
    d = t - c
    lo, d2 = d < 0.5, d * d
    zero = torch.zeros_like(d)
    s = torch.stack([torch.where(lo, 0.5 * (0.5 - d) ** 2, zero),
                     torch.where(lo, 0.75 - d2, 0.5 * (1.5 - d) ** 2),
                     torch.where(lo, 0.5 * (0.5 + d) ** 2, 0.75 - (1 - d) ** 2),
                     torch.where(lo, zero, 0.5 * (d - 0.5) ** 2)])
    ds = torch.stack([0.5 * d2 - d + 0.5, 2 * d - 1.5 * d2, 1.5 * d2 - d - 0.5, -0.5 * d2])
    return c.long() - 1, s, ds


def _shape2_centred(t):
    """Quadratic shape on five points with the centred difference of the shape as derivative."""
    c, s = _shape2(t)
    zero = torch.zeros_like(t)
    w = [zero, zero, s[0], s[1], s[2], zero, zero]
    return (c - 1, torch.stack(w[1:6]), torch.stack([0.5 * (w[i + 2] - w[i]) for i in range(5)]))


class _March:
    """One time step of the quasi-static slice march in normalized units (c = mu0 = ep0 = 1)."""

    def __init__(self, case, device):
        c = self.c = case
        self.dev = device
        self.nx, self.ny, self.nz = c["nx"], c["ny"], c["nz"]
        self.lo = (-c["half_width"], -c["half_width"] * c["ny"] / c["nx"])
        self.dx = 2 * c["half_width"] / c["nx"]
        self.dy = -2 * self.lo[1] / c["ny"]
        self.dz = (c["zeta_hi"] - c["zeta_lo"]) / c["nz"]
        self.poisson = _Poisson(self.nx, self.ny, self.dx, self.dy, device)
        self.shape = (self.ny + 2 * G, self.nx + 2 * G)

    def plane(self):
        return torch.zeros(self.shape, dtype=torch.float64, device=self.dev)

    def inner(self, f, i=0, j=0):
        return f[G + j:G + j + self.ny, G + i:G + i + self.nx]

    def mid(self, x, y):
        """Cell units (cell centres at integers)."""
        return (x - self.lo[0]) / self.dx - 0.5, (y - self.lo[1]) / self.dy - 0.5

    def index(self, cx, cy, ix, iy):
        return (cy + iy + G) * self.shape[1] + cx + ix + G

    def deposit(self, x, y, values, outs):
        """outs[k] += values[k] with the quadratic shape."""
        tx, ty = self.mid(x, y)
        (cx, sx), (cy, sy) = _shape2(tx), _shape2(ty)
        for iy in range(3):
            for ix in range(3):
                at, s = self.index(cx, cy, ix, iy), sx[ix] * sy[iy]
                for v, o in zip(values, outs):
                    o.view(-1).index_add_(0, at, s * v)

    def gather(self, x, y, fields):
        tx, ty = self.mid(x, y)
        (cx, sx, dsx), (cy, sy, dsy) = _shape2_nodal(tx), _shape2_nodal(ty)
        psi, rest = fields[0].view(-1), torch.stack([f.view(-1) for f in fields[1:]])
        ex, ey, out = 0.0, 0.0, 0.0
        for iy in range(4):
            for ix in range(4):
                at = self.index(cx, cy, ix, iy)
                p = psi[at]
                ex = ex + dsx[ix] * sy[iy] * p / self.dx
                ey = ey + sx[ix] * dsy[iy] * p / self.dy
                out = out + sx[ix] * sy[iy] * rest[:, at]
        return (ex, ey) + tuple(out)

    def boundary(self, x, y, ux, uy):
        """Positions and momenta after the transverse particle boundary (reflecting or periodic)."""
        out = []
        for q, u, lo in ((x, ux, self.lo[0]), (y, uy, self.lo[1])):
            length = -2 * lo
            outside = (q < lo) | (q > -lo)
            if self.c["solver"] == "pc":
                out += [torch.where(outside, torch.remainder(q - lo, length) + lo, q), u]
            else:
                r = torch.remainder(q - lo, 2 * length)
                back = r > length
                out += [torch.where(outside, torch.where(back, 2 * length - r, r) + lo, q),
                        torch.where(outside & back, -u, u)]
        return out[0], out[2], out[1], out[3]

    # ---- plasma
    def init_plasma(self):
        p, c = self.c["ppc"], self.c
        f = torch.float64
        xs = self.lo[0] + (torch.arange(self.nx * p, device=self.dev, dtype=f) + 0.5) * (self.dx / p)
        ys = self.lo[1] + (torch.arange(self.ny * p, device=self.dev, dtype=f) + 0.5) * (self.dy / p)
        y, x = (t.reshape(-1).clone() for t in torch.meshgrid(ys, xs, indexing="ij"))
        zero = torch.zeros_like(x)
        w = (1.0 + c["channel"] * (x * x + y * y)) / (p * p)
        return {"x": x, "y": y, "w": w, "ux": zero, "uy": zero, "psi": zero + 1, "xp": x, "yp": y, "uxh": zero,
                "uyh": zero, "psih": zero + 1}

    def deposit_plasma(self, p, jx, jy, chi=None, jz=None, rhomjz=None):
        """Currents of electrons (charge -1, mass 1); particles beyond the quasi-static limit drop out."""
        pi = 1 / p["psi"]
        vx, vy = p["ux"] * pi, p["uy"] * pi
        gp = 0.5 * (pi * pi + vx * vx + vy * vy + 1)
        lost = (gp < 0) | (gp > 35.0) | (pi < 0)
        if bool(lost.any()):
            # out for good: no weight, at rest
            p["w"] = torch.where(lost, torch.zeros_like(gp), p["w"])
            for k in ("ux", "uy", "uxh", "uyh", "psi", "psih"):
                p[k] = torch.where(lost, torch.full_like(gp, 1.0 if k[:3] == "psi" else 0.0), p[k])
            return self.deposit_plasma(p, jx, jy, chi, jz, rhomjz)
        q = -p["w"]
        todo = [(q * vx, jx), (q * vy, jy), (q * (gp - 1), jz), (-q * pi, chi), (q, rhomjz)]
        todo = [(v, o) for v, o in todo if o is not None]
        self.deposit(p["x"], p["y"], [v for v, _ in todo], [o for _, o in todo])

    def explicit_source(self, p, psi, ex, ey, ez, bz, sx_out, sy_out):
        """Plasma contribution to the source of the explicit Bx/By equation."""
        pi = 1 / p["psi"]
        vx, vy = p["ux"] * pi, p["uy"] * pi
        gp = 0.5 * (pi * pi + vx * vx + vy * vy + 1)
        cdm, qm = -p["w"], -1.0
        tx, ty = self.mid(p["x"], p["y"])
        (cx, sx, dsx), (cy, sy, dsy) = _shape2_centred(tx), _shape2_centred(ty)
        f = torch.stack([t.view(-1) for t in (bz, ez, ex, ey)])
        for iy in range(5):
            for ix in range(5):
                if ix in (0, 4) and iy in (0, 4):
                    continue
                at = self.index(cx, cy, ix, iy)
                b, e, fx, fy = f[:, at]
                s, dx, dy = sx[ix] * sy[iy], dsx[ix] * sy[iy] / self.dx, sx[ix] * dsy[iy] / self.dy
                vsy = cdm * (-s * (-b * vx + e * vy - fx * vx * vy + fy * (gp - vy * vy)) * qm * pi
                             + dx * vx * vy - dy * (gp - vy * vy - 1))
                vsx = cdm * (s * (b * vy + e * vx + fx * (gp - vx * vx) - fy * vx * vy) * qm * pi
                             + dx * (gp - vx * vx - 1) - dy * vx * vy)
                sy_out.view(-1).index_add_(0, at, vsy)
                sx_out.view(-1).index_add_(0, at, vsx)

    def push_plasma(self, p, fields, temporary=False):
        ex, ey, ez, bx, by, bz = self.gather(p["xp"], p["yp"], fields)
        ux, uy, psi = p["uxh"], p["uyh"], p["psih"]
        h = self.dz / 4

        def substep(ux, uy, psi):
            # second-order Taylor step with charge/mass = -1
            pi = 1 / psi
            a2 = 1 + ux * ux + uy * uy
            gp, ue = 0.5 * pi * pi * a2 + 0.5, ux * ex + uy * ey
            d0 = -(gp * ex + by + uy * bz * pi)
            d1 = -(gp * ey - bx - ux * bz * pi)
            d2 = -(ue * pi - ez)
            dpi = -pi * pi * d2
            dgp = pi * dpi * a2 + pi * pi * (ux * d0 + uy * d1)
            e0 = -(dgp * ex + bz * (d1 * pi + uy * dpi))
            e1 = -(dgp * ey - bz * (d0 * pi + ux * dpi))
            e2 = -((d0 * ex + d1 * ey) * pi + ue * dpi)
            return ux + h * d0 + 0.5 * h * h * e0, uy + h * d1 + 0.5 * h * h * e1, psi + h * d2 + 0.5 * h * h * e2

        for _ in range(4):
            ux, uy, psi = substep(ux, uy, psi)
        x, y = p["xp"] + self.dz * ux / psi, p["yp"] + self.dz * uy / psi
        x, y, ux, uy = self.boundary(x, y, ux, uy)
        p["x"], p["y"] = x, y
        if not temporary:
            p["uxh"], p["uyh"], p["psih"], p["xp"], p["yp"] = ux, uy, psi, x, y
        for _ in range(2):
            ux, uy, psi = substep(ux, uy, psi)
        p["ux"], p["uy"], p["psi"] = ux, uy, psi

    # ---- beam (charge -1, mass 1)
    def deposit_beam(self, b, at, jx, jy, jz):
        if at is None or not len(at):
            return
        ux, uy, uz = b["ux"][at], b["uy"][at], b["uz"][at]
        gi = 1 / torch.sqrt(1 + ux * ux + uy * uy + uz * uz)
        q = -b["w"][at]
        todo = [(v, o) for v, o in ((q * ux * gi, jx), (q * uy * gi, jy), (q * uz * gi, jz)) if o is not None]
        self.deposit(b["x"][at], b["y"][at], [v for v, _ in todo], [o for _, o in todo])

    def push_beam(self, b, at, sub, zmin, fields):
        """Sub-cycles of the particles `at` of a slice until they leave it backwards."""
        n, dt = 10, self.c["dt"] / 10
        v = {k: b[k][at] for k in ("x", "y", "z", "ux", "uy", "uz")}
        done = sub[at]
        for k in range(n):
            go = (done == k) & (v["z"] >= zmin)
            gi = 1 / torch.sqrt(1 + v["ux"] ** 2 + v["uy"] ** 2 + v["uz"] ** 2)
            x, y = v["x"] + 0.5 * dt * v["ux"] * gi, v["y"] + 0.5 * dt * v["uy"] * gi
            x, y, ux, uy = self.boundary(x, y, v["ux"], v["uy"])
            uz = v["uz"]
            ex, ey, ez, bx, by, bz = self.gather(x, y, fields)
            uxn = ux - dt * (ex + (1 - uz * gi) * by + uy * gi * bz)
            uyn = uy - dt * (ey + (uz * gi - 1) * bx - ux * gi * bz)
            uxi, uyi, uzi = 0.5 * (ux + uxn), 0.5 * (uy + uyn), uz - 0.5 * dt * ez
            gm = 1 / torch.sqrt(1 + uxi * uxi + uyi * uyi + uzi * uzi)
            uzn = uz - dt * (ez + (uxi * by - uyi * bx) * gm)
            gn = 1 / torch.sqrt(1 + uxn * uxn + uyn * uyn + uzn * uzn)
            new = {"x": x + 0.5 * dt * uxn * gn, "y": y + 0.5 * dt * uyn * gn, "ux": uxn, "uy": uyn, "uz": uzn,
                   "z": v["z"] + dt * (uzn * gn - 1) if self.c["z_push"] else v["z"]}
            v = {q: torch.where(go, new[q], v[q]) for q in v}
            done = torch.where(go, done + 1, done)
        v["x"], v["y"], v["ux"], v["uy"] = self.boundary(v["x"], v["y"], v["ux"], v["uy"])
        for q in v:
            b[q][at] = v[q]
        sub[at] = done

    # ---- fields
    def laplacian(self, u):
        """5-point Laplacian of [2, ny, nx]; even grids: Dirichlet on the cell face."""
        fx, fy = 1 / self.dx ** 2, 1 / self.dy ** 2
        p = torch.nn.functional.pad(u, (1, 1, 1, 1))
        lap = fx * (p[:, 1:-1, 2:] + p[:, 1:-1, :-2]) + fy * (p[:, 2:, 1:-1] + p[:, :-2, 1:-1]) - 2 * (fx + fy) * u
        if self.nx % 2 == 0:
            lap[:, :, 0] += fx * (u[:, :, 1] / 3 - 2 * u[:, :, 0])
            lap[:, :, -1] += fx * (u[:, :, -2] / 3 - 2 * u[:, :, -1])
            lap[:, 0] += fy * (u[:, 1] / 3 - 2 * u[:, 0])
            lap[:, -1] += fy * (u[:, -2] / 3 - 2 * u[:, -1])
        return lap

    def solve_b(self, rhs, chi, guess):
        """Lap(B) - chi B = S for both components by BiCGStab, preconditioned with a fast solve."""
        shift = chi.mean()
        prec = lambda r: self.poisson(r, shift)  # noqa: E731
        op = lambda v: self.laplacian(v) - chi * v  # noqa: E731
        dot = lambda a, b: (a * b).sum()  # noqa: E731
        x = guess.clone()
        r = rhs - op(x)
        target = 1e-13 * torch.linalg.vector_norm(rhs)
        r0, p = r.clone(), r.clone()
        rho = dot(r0, r)
        for it in range(200):
            if it % 4 == 0 and torch.linalg.vector_norm(r) <= target:
                break
            ph = prec(p)
            v = op(ph)
            alpha = rho / dot(r0, v)
            s = r - alpha * v
            sh = prec(s)
            t = op(sh)
            omega = dot(t, s) / dot(t, t).clamp_min(1e-300)
            x = x + alpha * ph + omega * sh
            r = s - omega * t
            rho1 = dot(r0, r)
            p = r + rho1 / rho * alpha / omega * (p - omega * v)
            rho = rho1
        return x

    def put(self, f, v):
        f[G:G + self.ny, G:G + self.nx] = v

    def solve_psi_ez_bz(self, rhomjz, ions, jx, jy, F):
        i = self.inner
        dx, dy = lambda f: (i(f, 1) - i(f, -1)) / (2 * self.dx), lambda f: (i(f, 0, 1) - i(f, 0, -1)) / (2 * self.dy)
        rhs = torch.stack([-i(rhomjz + ions), dx(jx) + dy(jy), dy(jx) - dx(jy)])
        u = self.poisson(rhs)
        for k, name in enumerate(("Psi", "Ez", "Bz")):
            self.put(F[name], u[k])
        F["ExmBy"], F["EypBx"] = self.plane(), self.plane()
        p = F["Psi"]
        F["ExmBy"][1:-1, 1:-1] = -(p[1:-1, 2:] - p[1:-1, :-2]) / (2 * self.dx)
        F["EypBx"][1:-1, 1:-1] = -(p[2:, 1:-1] - p[:-2, 1:-1]) / (2 * self.dy)

    def __call__(self, beam):
        pc = self.c["solver"] == "pc"
        b = {k: torch.from_numpy(np.ascontiguousarray(v)).to(self.dev) for k, v in beam.items()}
        zlo = self.c["zeta_lo"]
        key = ((b["z"] - zlo) / self.dz).to(torch.int64)  # towards zero, like the binning
        order = torch.sort(torch.where((key >= 0) & (key < self.nz), self.nz - 1 - key,
                                       torch.full_like(key, self.nz)), stable=True).indices
        count = torch.bincount(key.clamp(-1, self.nz) + 1, minlength=self.nz + 2)[1:self.nz + 1].flip(0)
        own = torch.split(order[:int(count.sum())], count.tolist())  # from the head down
        own = {self.nz - 1 - k: own[k] for k in range(self.nz)}
        sub = torch.zeros_like(key)
        p = self.init_plasma()
        ions = self.plane()
        self.deposit(p["x"], p["y"], [p["w"]], [ions])
        F = {k: self.plane() for k in ("Psi", "Ez", "Bx", "By", "Bz", "ExmBy", "EypBx")}
        planes = {k: torch.zeros((self.nz, self.nx), dtype=torch.float64, device=self.dev) for k in PLANES}
        kept, carry = [], order[:0]
        hist = {"b": [self.plane() for _ in range(4)], "j": [self.plane(), self.plane()]}
        jb, pjb = [self.plane(), self.plane()], [self.plane(), self.plane()]
        for s in range(self.nz - 1, -1, -1):
            if pc:
                self.slice_pc(p, b, own, s, ions, F, hist)
            else:
                njb = [self.plane(), self.plane()]
                self.slice_explicit(p, b, own, s, ions, F, jb, pjb, njb)
                pjb, jb = jb, njb
            for k in PLANES:
                f = self.inner(F[k])
                m = self.ny // 2
                row = f[m] if self.ny % 2 else 0.5 * (f[m - 1] + f[m])
                planes[k][s] = row
            fields = [F[k] for k in ("Psi", "Ez", "Bx", "By", "Bz")]
            at = torch.cat([own[s], carry])
            if len(at):
                zmin = zlo + s * self.dz
                self.push_beam(b, at, sub, zmin, fields)
                stay = b["z"][at] >= zmin
                kept.append(at[stay])
                carry = at[~stay]
            self.push_plasma(p, fields)
        at = torch.cat(kept) if kept else order[:0]
        out = {k: b[k][at] for k in BEAM + ("id",)}
        return {"beam": out, "slice": {k: self.inner(F[k]) for k in LAST_SLICE}, "plane": planes}

    def slice_explicit(self, p, b, own, s, ions, F, jb, pjb, njb):
        jx, jy, jzb = jb[0].clone(), jb[1].clone(), self.plane()
        chi, rhomjz, sx, sy = self.plane(), self.plane(), self.plane(), self.plane()
        self.deposit_beam(b, own[s], None, None, jzb)
        self.deposit_beam(b, own.get(s - 1), njb[0], njb[1], None)
        self.deposit_plasma(p, jx, jy, chi=chi, rhomjz=rhomjz)
        self.solve_psi_ez_bz(rhomjz, ions, jx, jy, F)
        i = self.inner
        self.put(sy, -(i(jzb, 0, 1) - i(jzb, 0, -1)) / (2 * self.dy) + (i(pjb[1]) - i(njb[1])) / (2 * self.dz))
        self.put(sx, (i(jzb, 1) - i(jzb, -1)) / (2 * self.dx) - (i(pjb[0]) - i(njb[0])) / (2 * self.dz))
        self.explicit_source(p, F["Psi"], F["ExmBy"], F["EypBx"], F["Ez"], F["Bz"], sx, sy)
        u = self.solve_b(torch.stack([i(sy), i(sx)]), i(chi), torch.stack([i(F["Bx"]), i(F["By"])]))
        self.put(F["Bx"], u[0])
        self.put(F["By"], u[1])

    def slice_pc(self, p, b, own, s, ions, F, hist):
        """Predictor-corrector Bx/By: three iterations, mixing 0.05 weighted by the errors."""
        i = self.inner
        jx, jy, jz, rhomjz = self.plane(), self.plane(), self.plane(), self.plane()
        self.deposit_plasma(p, jx, jy, jz=jz, rhomjz=rhomjz)
        self.deposit_beam(b, own[s], jx, jy, jz)
        self.solve_psi_ez_bz(rhomjz, ions, jx, jy, F)
        pbx, pby, ppbx, ppby = hist["b"]

        def relative(ax, ay, bx, by):
            norm = torch.sqrt(i(ax) ** 2 + i(ay) ** 2).sum()
            diff = torch.sqrt((i(ax) - i(bx)) ** 2 + (i(ay) - i(by)) ** 2).sum()
            return float(diff / norm) if float(norm) > 0 else 0.0

        err = relative(pbx, pby, ppbx, ppby)
        factor = math.exp(-0.5 * (err / (2.5 * -1.0)) ** 2)
        F["Bx"] = (1 + factor) * pbx - factor * ppbx
        F["By"] = (1 + factor) * pby - factor * ppby
        previous, last = (F["Bx"], F["By"]), None
        for _ in range(3):
            self.push_plasma(p, [F[k] for k in ("Psi", "Ez", "Bx", "By", "Bz")], temporary=True)
            njx, njy = self.plane(), self.plane()
            self.deposit_plasma(p, njx, njy)
            self.deposit_beam(b, own.get(s - 1), njx, njy, None)
            hz = 2 * self.dz
            u = self.poisson(torch.stack(
                [-(i(jz, 0, 1) - i(jz, 0, -1)) / (2 * self.dy) + (i(hist["j"][1]) - i(njy)) / hz,
                 (i(jz, 1) - i(jz, -1)) / (2 * self.dx) - (i(hist["j"][0]) - i(njx)) / hz]))
            new = self.plane(), self.plane()
            self.put(new[0], u[0])
            self.put(new[1], u[1])
            err = relative(F["Bx"], F["By"], *new)
            last = err if last is None else last
            wn, wp = (last / (err + last), err / (err + last)) if err + last else (0.5, 0.5)
            F["Bx"] = 0.95 * F["Bx"] + 0.05 * (wn * new[0] + wp * previous[0])
            F["By"] = 0.95 * F["By"] + 0.05 * (wn * new[1] + wp * previous[1])
            previous, last = new, err
        hist["j"] = [jx, jy]
        hist["b"] = [F["Bx"], F["By"]] + hist["b"][:2]


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "poisson":
        f = torch.from_numpy(_rhs(case, seed)).to(device)
        return _Poisson(case["nx"], case["ny"], 1.0 / (case["nx"] + 1), 1.0 / (case["ny"] + 1), device)(f)
    if case["kind"] == "gradient" or case["nx"] * case["ny"] * case["nz"] > 20000000:
        return None  # takes too long
    if case["solver"] == "explicit" and case["tolerance"] > 1e-8:
        return None  # the path stops its multigrid long before 64 bits, and the march amplifies that
    r = _March(case, device)(_beams(case, seed)[0])
    return {k: {q: v.cpu().numpy() for q, v in r[k].items()} for k in r}
