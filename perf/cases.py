"""The work a user of this library has it do, as timed cases.

Three kinds of program use it:
  * a simulation that keeps its state on the GPU, advances it with ``step``
    and reads the fields back at its output interval (kind ``step``; with
    ``salinity`` the phase-3 loop);
  * a host program that owns the state and calls the step routine by routine,
    uploading before and downloading after (kind ``routines``: how the Fortran
    main loop binds the C ABI);
  * calibration runs of the differentiable WCSPH step (``wcsph``) and programs
    that only want the sparse solver (``csr``, ``csr_noalloc``).

Sizes are those of the benchmark tanks (12000, 192000 and 833250 fluid
particles, the 97070-particle calibration tank) and of the unit tests' tanks
(3000), with spacings in between for the drawn ones.  Below 1.2 mm the
formulation itself is unstable, so that is the finest tank.

``exact`` restates each path in plain FP64 torch: pair lists by binning,
pair sums by ``index_add``, the pressure system by BiCGSTAB with refinement.
"""
import math

import numpy as np
import torch

from beach_slope_confined_gb300 import Solver, setup_tank, solve_csr, solve_csr_noalloc
from beach_slope_confined_gb300 import scenario as sc

STEPS = 4  # steps between two outputs
FIELDS = ("x", "y", "vx", "vy", "p", "rho")  # what a program writes out (with con, where salinity is transported)


def listed():
    return [
        # the smallest tank of the tests, the drop-in path: a few launches' worth of work each
        {"name": "step_fp64_3k", "kind": "step", "dx": 0.02, "precision": "fp64", "solver": "mg"},
        # the first benchmark tank on the mixed path: latency and launches still count
        {"name": "step_mixed_12k", "kind": "step", "dx": 0.01, "precision": "mixed", "solver": "mg"},
        # the second benchmark tank on the drop-in path
        {"name": "step_fp64_192k", "kind": "step", "dx": 0.0025, "precision": "fp64", "solver": "mg"},
        # the headline tank, on both paths: the largest
        {"name": "step_mixed_833k", "kind": "step", "dx": 0.0012, "precision": "mixed", "solver": "mg"},
        {"name": "step_fp64_833k", "kind": "step", "dx": 0.0012, "precision": "fp64", "solver": "mg"},
        # the reference's own solver, without preconditioner, as the parity runs use it
        {"name": "step_bicgstab_6k", "kind": "step", "dx": 0.0137, "precision": "fp64", "solver": "bicgstab"},
        # the phase-3 loop: salinity sub-steps around the step
        {"name": "step_salinity_192k", "kind": "step", "dx": 0.0025, "precision": "mixed", "solver": "mg",
         "salinity": True},
        # a host program calling routine by routine with the reference's hybrid kernel
        {"name": "routines_fp64_23k", "kind": "routines", "dx": 0.0071, "precision": "fp64", "solver": "mg",
         "kernel": 0},
        # the calibration tank, forward only (a line search evaluates the misfit)
        {"name": "wcsph_forward_97k", "kind": "wcsph", "dx": 0.0035, "steps": 20, "every": 10, "gradient": False},
        # a gradient on a coarser calibration tank, the last segment shorter than the others
        {"name": "wcsph_gradient_14k", "kind": "wcsph", "dx": 0.0091, "steps": 20, "every": 7, "gradient": True},
        # the standalone solver: from host arrays, and in place on a caller's device memory
        {"name": "csr_host_4k", "kind": "csr", "nx": 131, "ny": 33},
        {"name": "csr_noalloc_125k", "kind": "csr_noalloc", "nx": 1250, "ny": 100},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "routines", "wcsph", "csr", "csr_noalloc"])
    if kind == "step":
        solver = rng.choice(["mg", "mg", "mg", "mg", "bicgstab"])
        if solver == "bicgstab":
            return {"kind": kind, "dx": round(_log_uniform(rng, 0.005, 0.02), 6), "precision": "fp64",
                    "solver": solver}
        if rng.random() < 0.25:
            return {"kind": kind, "dx": round(_log_uniform(rng, 0.0025, 0.01), 6), "precision": "mixed",
                    "solver": solver, "salinity": True}
        return {"kind": kind, "dx": round(_log_uniform(rng, 0.0012, 0.02), 6),
                "precision": rng.choice(["fp64", "mixed"]), "solver": solver}
    if kind == "routines":
        return {"kind": kind, "dx": round(_log_uniform(rng, 0.0025, 0.02), 6),
                "precision": rng.choice(["fp64", "mixed"]), "solver": "mg", "kernel": rng.choice([0, 1])}
    if kind == "wcsph":
        grad = rng.random() < 0.5
        return {"kind": kind, "dx": round(_log_uniform(rng, 0.0045 if grad else 0.0035, 0.02), 6),
                "steps": rng.randint(8, 20), "every": rng.randint(3, 12), "gradient": grad}
    n = _log_uniform(rng, 1000, 60000 if kind == "csr" else 131072)
    ny = max(8, int(math.sqrt(n / rng.uniform(4, 12))))
    return {"kind": kind, "nx": max(8, int(n / ny)), "ny": ny}


# ---- set-up ------------------------------------------------------------------------
def _spec(case, seed):
    dx = case["dx"]
    if case["kind"] == "wcsph":
        return sc.TankSpec(dx=dx, dt=5e-5, por_cells=(16, 4), por_jitter=0.05, por_seed=seed + 1, seed=seed)
    # the impulsive piston start is stable down to the second benchmark tank's spacing
    return sc.TankSpec(dx=dx, kernel=case.get("kernel", 1), por_jitter=0.05, por_seed=seed + 1, seed=seed,
                       piston_ramp=0.0 if dx >= 0.0025 else sc.STARTUP_RAMP)


def _params(case, spec, scen):
    if case["kind"] == "wcsph":
        return sc.make_params(spec, scen.bounds)
    if case["solver"] == "bicgstab":
        return sc.make_params(spec, scen.bounds, solver="bicgstab", tol=1e-12, maxit=20000)
    return sc.make_params(spec, scen.bounds, precision=case["precision"], solver="fgmres", precond="mg", tol=1e-8,
                          maxit=40000, restart=40, inner_tol=1e-5, max_outer=60, salinity=case.get("salinity", False))


def _fields(case):
    return FIELDS + (("con",) if case.get("salinity") else ())


def _pinned(n, fields):
    """A download target in pinned memory: the fields wanted, and what every download brings."""
    t = {f: torch.zeros(n, dtype=torch.float64).pin_memory() for f in fields}
    t["L"] = torch.zeros(4 * n, dtype=torch.float64).pin_memory()
    t["tid"] = torch.zeros(n, dtype=torch.int8).pin_memory()
    t["flags"] = torch.zeros(n, dtype=torch.uint8).pin_memory()
    return t


def _csr_system(case, seed):
    """A pressure system of a jittered lattice, Jacobi-scaled: unit diagonal, negative off-diagonals decaying to the
    support's edge, a top layer of free-surface rows with a heavier diagonal."""
    nx, ny = case["nx"], case["ny"]
    n = nx * ny
    g = torch.Generator().manual_seed(seed)
    jit = (torch.rand((2, nx, ny), generator=g, dtype=torch.float64) - 0.5) * 0.1
    px = torch.arange(nx, dtype=torch.float64)[:, None] + jit[0]
    py = torch.arange(ny, dtype=torch.float64)[None, :] + jit[1]
    px, py = px.reshape(-1), py.reshape(-1)
    ix, iy = torch.arange(nx)[:, None].expand(nx, ny).reshape(-1), torch.arange(ny)[None, :].expand(nx, ny).reshape(-1)
    row, col, val = [], [], []
    for a in range(-3, 4):
        for b in range(-3, 4):
            ok = (ix + a >= 0) & (ix + a < nx) & (iy + b >= 0) & (iy + b < ny)
            i = ok.nonzero()[:, 0]
            j = i + a * ny + b
            r = torch.hypot(px[i] - px[j], py[i] - py[j])
            k = (r < 2.6) & (i != j)
            row.append(i[k]), col.append(j[k]), val.append(-((1 - r[k] / 2.6) ** 3))
    row, col, val = torch.cat(row), torch.cat(col), torch.cat(val)
    diag = torch.zeros(n, dtype=torch.float64).index_add_(0, row, -val)
    diag = torch.where(iy >= ny - 2, 2.0 * diag, diag)
    val = val / diag[row]
    eye = torch.arange(n)
    row, col = torch.cat([row, eye]), torch.cat([col, eye])
    val = torch.cat([val, torch.ones(n, dtype=torch.float64)])
    order = torch.argsort(row * n + col)
    row, col, val = row[order], col[order], val[order]
    rowptr = torch.zeros(n + 1, dtype=torch.int64)
    rowptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    # a smooth divergence plus cell-scale noise, as the predictor leaves it
    b = torch.sin(px * (6.0 / nx)) * (py / ny) + 0.1 * (torch.rand(n, generator=g, dtype=torch.float64) - 0.5)
    return rowptr.to(torch.int32), col.to(torch.int32), val, b * 1e-3


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("csr", "csr_noalloc"):
        rp, col, val, b = _csr_system(case, seed)
        P = sc.make_params(sc.TankSpec(), solver="bicgstab", tol=1e-12, maxit=20000)
        if kind == "csr":
            return {"case": case, "P": P, "args": [t.numpy() for t in (rp, col, val, b)], "x0": np.zeros(b.numel())}
        d = [t.cuda() for t in (rp, col, val, b)]
        return {"case": case, "P": P, "args": d, "x": torch.zeros_like(d[3])}
    spec = _spec(case, seed)
    scen = sc.build(spec)
    g = Solver(_params(case, spec, scen))
    s = {"case": case, "g": g, "scen": scen}
    if kind == "wcsph":
        setup_tank(g, scen, initial_effpor=False)
        wp, s["grid"] = sc.wcsph_params(spec, scen)
        g.wcsph_setup(wp)
        rng = np.random.default_rng(seed)
        s["observed"] = rng.normal(0.0, 1e-3, (case["steps"], len(spec.probes)))
        return s
    setup_tank(g, scen)
    s["out"] = _pinned(scen.n, _fields(case))
    s["out_np"] = {k: v.numpy() for k, v in s["out"].items()}
    if kind == "routines":
        up = sc.state_arrays(scen)
        s["up"] = {k: torch.from_numpy(v).pin_memory() for k, v in up.items()}
        s["up_np"] = {k: v.numpy() for k, v in s["up"].items()}
    return s


# ---- one pass ------------------------------------------------------------------------
def _read_back(s):
    out = dict(s["out_np"])
    s["g"].download_state(out)
    fields = {f: s["out"][f] for f in _fields(s["case"])}
    # the mixed path's pair sums are single precision: its fields are kept as such
    return fields if s["case"]["precision"] == "fp64" else {f: v.float() for f, v in fields.items()}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "csr":
        rc, x, info = solve_csr(s["P"], *s["args"], s["x0"])
        if rc:
            raise RuntimeError("csr_solve: %d" % rc)
        return x
    if kind == "csr_noalloc":
        s["x"].zero_()
        rc, info = solve_csr_noalloc(s["P"], s["x"].numel(), *(t.data_ptr() for t in s["args"]), s["x"].data_ptr(),
                                     stream=torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError("csr_solve_noalloc: %d" % rc)
        return s["x"]
    g = s["g"]
    if kind == "wcsph":
        eta = g.wcsph_forward(case["steps"], case["every"])
        if not case["gradient"]:
            return eta
        return {"eta": eta, "gradient": g.wcsph_adjoint(eta - s["observed"])}
    if kind == "step":
        g.step(STEPS)
        return _read_back(s)
    # the step by its routines, from the host's state (main.f90:44-65)
    g.upload_state(s["up_np"])
    g.set_time(s["scen"].spec.dt, s["scen"].spec.dt)
    g.effpor()
    for f in (g.piston, g.projection, g.cellshift, g.resetid, g.neighbour, g.effpor, g.eddyvis, g.int_vel, g.ppesolve,
              g.comp_vel, g.comp_pos, g.cellshift, g.neighbour, g.freesurf, g.effpor, g.opt2_shift):
        f()
    return _read_back(s)


# ---- what a pass cannot do without -----------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("csr", "csr_noalloc"):
        n = case["nx"] * case["ny"]
        nnz = 21.0 * n
        its = 4.0 * max(case["nx"] / 8.0, case["ny"])  # two products each, and the vectors
        return {"bytes": 12.0 * nnz + 28.0 * n, "flops": its * (4.0 * nnz + 20.0 * n)}
    n = (4.0 / case["dx"]) * (0.3 / case["dx"])
    pairs = 20.0 * n  # neighbours within 2.6 spacings
    if kind == "wcsph":
        k = case["steps"]
        fwd, rev = 60.0 * pairs + 20.0 * 0.2 * pairs, 170.0 * pairs
        # the state in and out, and for the reverse sweep the states of every step
        return {"bytes": k * n * 80.0 * (3.0 if case["gradient"] else 1.0),
                "flops": k * (fwd + (rev if case["gradient"] else 0.0))}
    steps = STEPS if kind == "step" else 1
    # the pair sums of one step (two searches with their corrections, porosity, eddy viscosity, predictor, assembly,
    # projection, shift), and the solve: some 15 cycles of five products, or unpreconditioned BiCGSTAB
    per_pair = 2 * 24.0 + 3 * 4.0 + 24.0 + 43.0 + 35.0 + 20.0 + 16.0 + (70.0 if case.get("salinity") else 0.0)
    solve = 15 * 5 * 2.0 * pairs if case["solver"] == "mg" else 6.0 * 0.3 / case["dx"] * 4.0 * pairs
    # fourteen state fields in and out; the system matrix written and read once
    return {"bytes": steps * (n * 2 * 14 * 8.0 + 2 * 12.0 * pairs), "flops": steps * (per_pair * pairs + solve)}


# ---- the same in plain 64-bit torch ------------------------------------------------------
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=DEV)


def _cell(x, x0, step):
    """The grid cell of a coordinate: a rounded quotient (by a tensor: a scalar divisor becomes a reciprocal), since
    lattice points lie on cell edges."""
    return torch.floor((x - x0) / torch.full_like(x, step)).long()


def _pairs(xa, ya, xb, yb, H):
    """Indices (i, j) of all a_i, b_j closer than H, by binning b on cells of side H."""
    x0, y0 = min(float(xa.min()), float(xb.min())) - H, min(float(ya.min()), float(yb.min())) - H
    ny = int((max(float(ya.max()), float(yb.max())) - y0) / H) + 3
    nx = int((max(float(xa.max()), float(xb.max())) - x0) / H) + 3
    key = lambda x, y: ((x - x0) / H).long() * ny + ((y - y0) / H).long()  # noqa: E731
    kb = key(xb, yb)
    order = torch.argsort(kb)
    count = torch.bincount(kb, minlength=nx * ny)
    start = torch.cumsum(count, 0) - count
    ka = key(xa, ya)
    I, J = [], []
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            kc = (ka + a * ny + b).clamp(0, nx * ny - 1)
            c = count[kc]
            i = torch.repeat_interleave(torch.arange(ka.numel(), device=ka.device), c)
            q = torch.arange(i.numel(), device=ka.device) - torch.repeat_interleave(torch.cumsum(c, 0) - c, c)
            j = order[start[kc][i] + q]
            dx, dy = xa[i] - xb[j], ya[i] - yb[j]
            keep = torch.sqrt(dx * dx + dy * dy) < H
            I.append(i[keep]), J.append(j[keep])
    return torch.cat(I), torch.cat(J)


def _solve(n, row, col, val, b, x):
    """BiCGSTAB to 1e-13 with restarts from the true residual; val holds every entry."""
    order = torch.argsort(row * n + col)
    rp = torch.zeros(n + 1, dtype=torch.int64, device=row.device)
    rp[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    A = torch.sparse_csr_tensor(rp, col[order], val[order], (n, n))
    mul = lambda v: (A @ v[:, None])[:, 0]  # noqa: E731
    bn = b.norm()
    for _ in range(12):
        r = b - mul(x)
        if float(r.norm()) <= 1e-14 * float(bn):
            break
        d, rh, p, r0 = torch.zeros_like(b), r.clone(), r.clone(), float(r.norm())
        rho, best, best_r = rh @ r, d.clone(), r0
        for it in range(1, 20001):
            v = mul(p)
            al = rho / (rh @ v)
            s = r - al * v
            t = mul(s)
            om = (t @ s) / (t @ t)
            d = d + al * p + om * s
            r = s - om * t
            new = rh @ r
            p = r + (new / rho) * (al / om) * (p - om * v)
            rho = new
            if it % 20 == 0:
                rn = float(r.norm())
                if not math.isfinite(rn) or rn > 1e6 * r0:
                    break
                if rn < best_r:
                    best, best_r = d.clone(), rn
                if rn <= 1e-9 * r0 or rn <= 1e-15 * float(bn):
                    break
        if best_r >= 0.5 * r0:
            break
        x = x + best
    return x


class _Tank:
    """The particles of a tank and the step's operators on them."""

    def __init__(self, case, seed):
        spec = _spec(case, seed)
        scen = sc.build(spec)
        self.spec, self.scen, self.n = spec, scen, scen.n
        self.P = _params(case, spec, scen)
        a = sc.state_arrays(scen)
        for f in ("x", "y", "vx", "vy", "vxs", "vys", "p", "rho", "oden", "mass", "xrest", "con", "nut", "tke", "vel",
                  "varts"):
            setattr(self, f, _t(a[f]))
        self.tid = torch.as_tensor(scen.tid.astype(np.int64), device=DEV)
        self.fluid = self.tid == sc.TID_FLUID
        self.pist = torch.as_tensor((scen.flags & sc.FLAG_PISTON) != 0, device=DEV)
        self.n_ = torch.ones(self.n, dtype=torch.float64, device=DEV)
        self.vol, self.ovol = self.mass / self.rho, self.mass / self.oden
        self.L = [torch.ones_like(self.x), torch.zeros_like(self.x), torch.zeros_like(self.x), torch.ones_like(self.x)]
        self.sx, self.sy = _t(scen.sx), _t(scen.sy)
        self.svol = _t(scen.smass) / _t(scen.srho)
        self.grid = _t(scen.por_grid)
        self.spor = self.porosity_at(self.sx, self.sy)
        self.resist = torch.zeros_like(self.x)
        self.t, self.dt, self.umax, self.numax = 0.0, spec.dt, 0.0, 0.0
        self.h = self.P.h

    def porosity_at(self, x, y):
        s = self.scen
        ny, nx = self.grid.shape
        ix, iy = _cell(x, s.por_origin[0], s.por_step[0]), _cell(y, s.por_origin[1], s.por_step[1])
        inside = (ix >= 0) & (ix < nx) & (iy >= 0) & (iy < ny)
        g = self.grid[iy.clamp(0, ny - 1), ix.clamp(0, nx - 1)]
        return torch.where(inside, g, torch.full_like(g, self.spec.por))

    # W and F (grad W = F (x_i - x_j)) of kernel.f90:34-162
    def W(self, r):
        h = self.h
        q = r / h
        if self.spec.kernel == 1:
            return 7.0 / (4 * 3.140 * h * h) * (1 + 2 * q) * (1 - q / 2) ** 4
        A, B = 0.1 * (10.0 / (float(np.float32(28) * np.float32(3.14)) * h * h)), 0.9 / (float(np.float32(3) * np.float32(3.14)) * h * h)
        near = A * (4 - 6 * q * q + 3 * q ** 3) + B * (q ** 3 - 6 * q + 6)
        return torch.where(q < 1, near, (A + B) * (2 - q) ** 3)

    def F(self, r):
        h = self.h
        if self.spec.kernel == 1:
            return -35.0 / (4 * 3.140 * h ** 4) * (1 - r / (2 * h)) ** 3
        q = r / h
        A, B = 0.1 * (10.0 / (float(np.float32(28) * np.float32(3.14)) * h * h)), 0.9 / (float(np.float32(3) * np.float32(3.14)) * h * h)
        near = A * (9 * r / h ** 3 - 12 / h ** 2) + B * (3 * r / h ** 3 - 6 / (r * h))
        return torch.where(q < 1, near, -(A + B) * 3 / (r * h) * (2 - q) ** 2)

    def sum(self, i, v):
        return torch.zeros(self.n, dtype=torch.float64, device=DEV).index_add_(0, i, v)

    def search(self):
        i, j = _pairs(self.x, self.y, self.x, self.y, 2 * self.h)
        k = i != j
        self.i, self.j = i, j = i[k], j[k]
        dx, dy = self.x[i] - self.x[j], self.y[i] - self.y[j]
        self.r = torch.sqrt(dx * dx + dy * dy)
        F = self.F(self.r)
        self.gx, self.gy = F * dx, F * dy
        V = self.vol[j]
        a, b = self.sum(i, -V * dx * self.gx), self.sum(i, -V * dx * self.gy)
        c, d = self.sum(i, -V * dy * self.gx), self.sum(i, -V * dy * self.gy)
        det = a * d - b * c
        ok = (det.abs() >= float(np.float32(1e-5))) & torch.isfinite(det)
        one, zero = torch.ones_like(a), torch.zeros_like(a)
        new = [torch.where(ok, d / det, one), torch.where(ok, -b / det, zero), torch.where(ok, -c / det, zero),
               torch.where(ok, a / det, one)]
        self.L = [torch.where(self.fluid, u, v) for u, v in zip(new, self.L)]
        self.free = self.fluid & (a + d <= self.P.free_threshold)
        self.count = torch.bincount(i, minlength=self.n)

    def corrected(self, at):
        L = [l[at] for l in self.L]
        return L[0] * self.gx + L[1] * self.gy, L[2] * self.gx + L[3] * self.gy

    def effpor(self):
        P, f = self.P, self.fluid
        i, s = _pairs(self.x, self.y, self.sx, self.sy, 2 * self.h)
        r = torch.sqrt((self.x[i] - self.sx[s]) ** 2 + (self.y[i] - self.sy[s]) ** 2)
        frac = self.sum(i, (1 - self.spor[s]) * self.W(r) * self.svol[s])
        nn = 1 - torch.minimum(frac, 1 - self.porosity_at(self.x, self.y))
        self.n_ = torch.where(f, nn, self.n_)
        self.rho = torch.where(f, nn * self.oden, self.rho)
        self.vol = torch.where(f, self.mass / self.rho, self.vol)
        nu = self.nu()
        v = torch.sqrt(self.vx ** 2 + self.vy ** 2)
        n3, d = self.n_ ** 3, P.d50
        R = -(nu * P.darcy_alpha * (1 - self.n_) ** 2 / (n3 * d * d)) - P.forch_beta * v * (1 - self.n_) / (n3 * d)
        self.resist = torch.where(f, R, torch.zeros_like(R))

    def nu(self):
        s = self.oden - 1000.0
        return (1.002 + 0.001652 * s + 0.0000083 * s * s) * 0.001 / self.oden

    def eddyvis(self):
        P, i, j = self.P, self.i, self.j
        ux, uy = self.vx / self.n_, self.vy / self.n_
        gx, gy = self.corrected(i)
        du, dv, V = ux[j] - ux[i], uy[j] - uy[i], self.vol[j]
        a, b, c = self.sum(i, V * du * gx), self.sum(i, V * dv * gy), self.sum(i, 0.5 * V * (du * gy + dv * gx))
        s = torch.sqrt(2 * (a * a + b * b) + 4 * c * c)
        self.nut = torch.where(self.fluid, (P.eddy_cs * P.dl) ** 2 * s, self.nut)
        self.tke = torch.where(self.fluid, P.eddy_cv / P.eddy_ce * (P.dl * s) ** 2, self.tke)

    def int_vel(self):
        P, i, j, dt = self.P, self.i, self.j, self.dt
        small = float(np.float32(1e-6))
        gx, gy = self.corrected(i)
        V = self.vol[j]
        ux, uy = self.vx / self.n_, self.vy / self.n_
        T1, T2 = self.sum(i, V * (ux[j] - ux[i]) * gx), self.sum(i, V * (uy[j] - uy[i]) * gy)
        va = P.varts_ps * P.dl ** 2 * torch.sqrt(T1 ** 2 + T2 ** 2) * torch.sqrt(self.vx ** 2 + self.vy ** 2)
        varts = va / ((self.umax + small) * self.n_)
        nu, fj = self.nu(), self.fluid[j]
        cmu = torch.where(fj, 2 * nu[i] * nu[j] / (nu[i] + nu[j]), nu[i])
        w0 = float(self.W(torch.zeros(1, dtype=torch.float64)))
        near = torch.where(self.free[j], self.W(self.r_now()) * varts[j] / w0, torch.zeros_like(cmu))
        visc = cmu + torch.where(self.free[i], varts[i], near)
        a, b = self.nut[i], self.nut[j]
        eddy = torch.where((a < small) & (b < small), (a + b) * 0.5, 2 * a * b / (a + b))
        visc = visc + torch.where(fj, eddy, torch.zeros_like(eddy))
        dx, dy = self.x[i] - self.x[j], self.y[i] - self.y[j]
        geo = 2 * V * (dx * gx + dy * gy) / (dx * dx + dy * dy + P.lam)
        dk = V * (self.tke[j] - self.tke[i])
        sps = self.n_ * 2 / 3
        ax = self.sum(i, geo * (self.vx[i] - self.vx[j]) * visc) - sps * self.sum(i, dk * gx)
        ay = self.sum(i, geo * (self.vy[i] - self.vy[j]) * visc) - sps * self.sum(i, dk * gy)
        D = 1 - dt * self.resist * self.n_
        self.vxs = torch.where(self.fluid, (self.vx + dt * ax) / D, self.vxs)
        self.vys = torch.where(self.fluid, (self.vy + dt * ay) / D + P.g * self.n_ * dt, self.vys)

    def r_now(self):
        return torch.sqrt((self.x[self.i] - self.x[self.j]) ** 2 + (self.y[self.i] - self.y[self.j]) ** 2)

    def pressure(self):
        P, i, j = self.P, self.i, self.j
        ti, tj = self.tid[i], self.tid[j]
        fi, fj = ti == 3, tj == 3
        q, usx, usy = self.rho / self.n_, self.vxs / self.n_, self.vys / self.n_
        Li, Lj = self.corrected(i), self.corrected(j)
        wall_fluid = (ti == 1) & fj
        gx = torch.where(fi, Li[0], torch.where(wall_fluid, Lj[0], self.gx))
        gy = torch.where(fi, Li[1], torch.where(wall_fluid, Lj[1], self.gy))
        V = torch.where(wall_fluid, self.vol[i], self.vol[j])
        dx, dy = self.x[i] - self.x[j], self.y[i] - self.y[j]
        t = 2 * V * (dx * gx + dy * gy) / (dx * dx + dy * dy + P.lam)
        t = torch.where((ti == 2) & fj, torch.zeros_like(t), t)
        lamp = torch.where(fi & fj & self.free[i], 1 + self.oden[j] / (P.rho0 * P.rel_den), torch.ones_like(t))
        dia = self.sum(i, t * lamp)
        harm = 2 * q[i] * q[j] / (q[i] + q[j])
        ddx = torch.where(fj, harm * (usx[j] - usx[i]), q[i] * (self.vxs[j] - self.vxs[i]) / self.n_[i])
        ddy = torch.where(fj, harm * (usy[j] - usy[i]), q[i] * (self.vys[j] - self.vys[i]) / self.n_[i])
        ddx = torch.where(wall_fluid, q[j] * (usx[j] - usx[i]), ddx)
        ddy = torch.where(wall_fluid, q[j] * (usy[j] - usy[i]), ddy)
        fv = self.sum(i, torch.where(fi | wall_fluid, V * (ddx * gx + ddy * gy), torch.zeros_like(t)))
        ok = (dia != 0) & torch.isfinite(dia)
        d = torch.where(ok, dia, torch.ones_like(dia))
        val = torch.where(ok[i], -t / d[i], torch.zeros_like(t))
        b = torch.where(ok, fv / self.dt / d, torch.zeros_like(fv))
        eye = torch.arange(self.n, device=DEV)
        self.p = _solve(self.n, torch.cat([i, eye]), torch.cat([j, eye]), torch.cat([val, torch.ones_like(b)]), b,
                        self.p)

    def comp_vel(self):
        i, j, f = self.i, self.j, self.fluid
        q, p = self.rho / self.n_, self.p
        gx, gy = self.corrected(i)
        w = torch.where(f[j], 2 * (p[j] * q[i] + p[i] * q[j]) / (q[i] + q[j]), p[j] + p[i]) * self.vol[j]
        c0 = self.n_ ** 2 / self.rho
        self.vx = torch.where(f, self.vxs - self.dt * c0 * self.sum(i, w * gx), self.vx)
        self.vy = torch.where(f, self.vys - self.dt * c0 * self.sum(i, w * gy), self.vy)
        self.vel = torch.where(f, torch.sqrt(self.vx ** 2 + self.vy ** 2) / self.n_, self.vel)

    def shift(self):
        P, i, j = self.P, self.i, self.j
        V = self.vol[j]
        gx, gy = self.corrected(i)
        coef = -P.csh * self.h ** 2 * torch.where(self.free, 0.01, 1.0)
        xs, ys = coef * self.sum(i, V * self.gx), coef * self.sum(i, V * self.gy)
        lim = P.maxshift * P.dl
        on = self.fluid & (self.count > 0)
        dvx, dvy = V * (self.vx[j] - self.vx[i]), V * (self.vy[j] - self.vy[i])
        cvx = self.sum(i, dvx * gx) * xs + self.sum(i, dvx * gy) * ys
        cvy = self.sum(i, dvy * gx) * xs + self.sum(i, dvy * gy) * ys
        self.x, self.y = torch.where(on, self.x + xs.clamp(-lim, lim), self.x), torch.where(on, self.y + ys.clamp(-lim, lim), self.y)
        self.vx, self.vy = torch.where(on, self.vx + cvx, self.vx), torch.where(on, self.vy + cvy, self.vy)
        self.vxs, self.vys = torch.where(on, cvx, self.vxs), torch.where(on, cvy, self.vys)

    def salinity(self, dtsol):
        """One sub-step of scalar.f90:114-275 on the lists of the last search."""
        P, i, j = self.P, self.i, self.j
        al, at, Dm = P.disp_long, P.disp_trans, P.diffusivity
        v, cap = torch.sqrt(self.vx ** 2 + self.vy ** 2), 0.12 * P.dl ** 2 / self.dt

        def disp(a, b):
            D = Dm + (a * self.vx ** 2 + b * self.vy ** 2 + (al - at) * self.vx * self.vy) / (v * self.n_)
            D = torch.where(D > 0, D, torch.full_like(D, Dm))
            return torch.where(D <= cap, D, torch.full_like(D, cap))

        Dx, Dy, E = disp(al, at), disp(at, al), Dm + self.nut / P.tschmidt
        small = float(np.float32(1e-6))
        harm = lambda u: 2 * u[i] * u[j] / (u[i] + u[j])  # noqa: E731
        low = (self.nut[i] < small) & (self.nut[j] < small)
        eddy = torch.where(low, Dm + (self.nut[i] + self.nut[j]) * 0.5 / P.tschmidt, harm(E))
        open_ = (self.n_[i] >= 0.8) | (self.n_[j] >= 0.8)
        tx, ty = torch.where(open_, eddy, harm(Dx)), torch.where(open_, eddy, harm(Dy))
        dx, dy = self.x[i] - self.x[j], self.y[i] - self.y[j]
        t3 = self.ovol[i] * (1 / self.n_[i] + 1 / self.n_[j])
        q = t3 * (self.con[i] - self.con[j]) * self.F(self.r) / (self.r ** 2 + P.lam)
        both = self.fluid[i] & self.fluid[j]
        c = self.sum(i, torch.where(both, q * (tx * dx * dx + ty * dy * dy), torch.zeros_like(q)))
        self.con = torch.where(self.fluid, self.con + c * dtsol, self.con)

    def substeps(self):
        P = self.P
        dtsol = P.sig1 * P.dl ** 2 / (P.diffusivity + self.numax / P.tschmidt)
        k = 1 if dtsol >= self.dt else math.ceil(self.dt / dtsol)
        return k, self.dt / k

    def piston(self):
        xp, vp = sc.piston_stroke(self.spec, self.t)
        w = self.pist
        self.x = torch.where(w, self.xrest + xp, self.x)
        self.vx, self.vy = torch.where(w, torch.full_like(self.vx, vp), self.vx), self.vy.masked_fill(w, 0.0)
        self.vxs, self.vys = torch.where(w, torch.full_like(self.vx, vp), self.vxs), self.vys.masked_fill(w, 0.0)

    def step(self, salinity=False, advance=True):
        f, dt = self.fluid, self.dt
        if advance:
            self.t += dt
        if salinity:
            if not hasattr(self, "i"):
                self.search()
            k, dtsol = self.substeps()
            for _ in range(k):
                self.salinity(dtsol)
        self.piston()
        x, y = self.x, self.y
        self.x, self.y = torch.where(f, x + dt * self.vx / self.n_, x), torch.where(f, y + dt * self.vy / self.n_, y)
        self.search()
        self.effpor()
        self.eddyvis()
        self.int_vel()
        self.pressure()
        self.comp_vel()
        self.x = torch.where(f, (self.x + x + dt * self.vx / self.n_) / 2, self.x)
        self.y = torch.where(f, (self.y + y + dt * self.vy / self.n_) / 2, self.y)
        self.search()
        self.effpor()
        self.shift()
        if salinity:
            lo, hi = self.P.rho0, self.P.rho0 * self.P.rel_den
            self.oden = torch.where(f, 0.5 * (hi + lo) + self.con * (hi - lo), self.oden)
            self.mass = torch.where(f, self.oden * self.ovol, self.mass)
            self.rho = torch.where(f, self.oden * self.n_, self.rho)
            self.vol = torch.where(f, self.mass / self.rho, self.vol)
        self.umax, self.numax = float(self.vel.abs().max()), float(self.nut.abs().max())
        if salinity:
            self.eddyvis()


def _exact_wcsph(case, seed):
    """The forward run of the WCSPH step, and its gradient by reverse-mode differentiation of the same steps."""
    T = _Tank(case, seed)
    spec, scen, P = T.spec, T.scen, T.P
    wp, grid = sc.wcsph_params(spec, scen)
    h, dt, gam, rho0 = T.h, spec.dt, wp.gamma, P.rho0
    B, grav = rho0 * wp.c0 ** 2 / gam, abs(P.g) * gam / wp.c0 ** 2
    c2, f = wp.delta * 2 * h * wp.c0, T.fluid
    theta = _t(grid).reshape(-1).requires_grad_(case["gradient"])
    alpha = torch.tensor(wp.alpha, dtype=torch.float64, device=DEV, requires_grad=case["gradient"])
    beta = torch.tensor(wp.beta, dtype=torch.float64, device=DEV, requires_grad=case["gradient"])
    gnx = wp.grid_nx
    ix, iy = _cell(T.sx, wp.grid_x0, wp.grid_dx), _cell(T.sy, wp.grid_y0, wp.grid_dy)
    inside = (ix >= 0) & (ix < gnx) & (iy >= 0) & (iy < wp.grid_ny)
    cell = torch.where(inside, iy * gnx + ix, torch.zeros_like(ix))
    head = lambda y: rho0 * (1 + grav * (wp.surface_y - y)) ** (1 / gam)  # noqa: E731
    x, y, vx, vy = T.x, T.y, T.vx, T.vy
    rho = torch.where(y < wp.surface_y, head(y), torch.full_like(y, rho0))
    mass = rho * P.dl ** 2
    R1, eta = 2 * h, []
    keep = lambda a, b: torch.where(f, a, b)  # noqa: E731
    for _ in range(case["steps"]):
        T.t += dt
        xp, vp = sc.piston_stroke(spec, T.t)
        x = torch.where(T.pist, T.xrest + xp, x)
        vx, vy = torch.where(T.pist, torch.full_like(vx, vp), vx), vy.masked_fill(T.pist, 0.0)
        i, j = _pairs(x.detach(), y.detach(), x.detach(), y.detach(), 2 * h)
        k = (i != j) & f[i]
        i, j = i[k], j[k]
        si, s = _pairs(x.detach(), y.detach(), T.sx, T.sy, 2 * h)
        sw = (1 - torch.where(inside, theta[cell], torch.full_like(T.sx, P.por))) * T.svol
        sr = torch.sqrt((x[si] - T.sx[s]) ** 2 + (y[si] - T.sy[s]) ** 2)
        n_ = keep(1 - T.sum(si, sw[s] * T.W(sr)), torch.ones_like(x))
        rt = keep(rho.clamp(min=rho0), rho)
        p = B * ((rt / rho0) ** gam - 1)
        p = p.clamp(min=0)
        rh, V, pr = head(y), mass / rt, p / rt ** 2
        dx, dy = x[i] - x[j], y[i] - y[j]
        r2 = dx * dx + dy * dy
        F = T.F(torch.sqrt(r2))
        G = F * r2 / (r2 + P.lam)
        dvx, dvy = vx[i] - vx[j], vy[i] - vy[j]
        Dr = T.sum(i, rt[i] * V[j] * F * (dvx * dx + dvy * dy) - c2 * (rt[j] - rt[i] - rh[j] + rh[i]) * G * V[j])
        pc, vc = mass[j] * (pr[i] + pr[j]) * F, 2 * wp.nu * V[j] * G
        ax = -n_ * T.sum(i, pc * dx) + T.sum(i, vc * dvx)
        ay = -n_ * T.sum(i, pc * dy) + T.sum(i, vc * dvy) + n_ * P.g
        vv = vx ** 2 + vy ** 2
        vm = torch.where(vv > 0, torch.sqrt(torch.where(vv > 0, vv, torch.ones_like(vv))), torch.zeros_like(vv))
        on, n3 = 1 - n_, n_ ** 3
        R = -wp.nu * alpha * on ** 2 / (n3 * P.d50 ** 2) - beta * vm * on / (n3 * P.d50)
        D = 1 - dt * R * n_
        nvx, nvy = (vx + dt * ax) / D, (vy + dt * ay) / D
        x, y, rho = keep(x + dt * nvx / n_, x), keep(y + dt * nvy / n_, y), keep(rt + dt * Dr, rho)
        vx, vy = keep(nvx, vx), keep(nvy, vy)
        Vn = mass / rho
        q = [(x - xk).abs() / R1 for xk in spec.probes]
        eta.append(torch.stack([torch.where(f & (u < 1), Vn * (1.25 / R1) * (1 - u) ** 3 * (1 + 3 * u),
                                            torch.zeros_like(u)).sum() - wp.probe_depth for u in q]))
    eta = torch.stack(eta)
    if not case["gradient"]:
        return eta.cpu()
    observed = _t(np.random.default_rng(seed).normal(0.0, 1e-3, tuple(eta.shape)))
    g = torch.autograd.grad(eta, (alpha, beta, theta), grad_outputs=eta.detach() - observed)
    return {"eta": eta.detach().cpu(), "gradient": torch.cat([u.reshape(-1) for u in g]).cpu()}


def exact(case, seed):
    if case["kind"] in ("csr", "csr_noalloc"):
        rp, col, val, b = (t.to(DEV) for t in _csr_system(case, seed))
        n = b.numel()
        row = torch.repeat_interleave(torch.arange(n, device=DEV), (rp[1:] - rp[:-1]).long())
        return _solve(n, row, col.long(), val, b, torch.zeros_like(b)).cpu()
    if case["kind"] == "wcsph":
        return _exact_wcsph(case, seed)
    T = _Tank(case, seed)
    T.effpor()
    if case["kind"] == "routines":
        T.t = T.dt
        T.step(advance=False)
    else:
        for _ in range(STEPS):
            T.step(salinity=case.get("salinity", False))
    return {f: getattr(T, f).cpu() for f in _fields(case)}
