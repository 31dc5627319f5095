"""Performance cases: the calls a user of this framework makes, at the sizes it is used at.

A case is one of four calls, each through the package's public classes:

  linear    one assembly and one linear solve of a stationary 1p problem (FVAssembler and
            ILUBiCGSTABIstlSolver: the reference's LinearPDESolver use)
  step      one implicit-Euler time step of a 2p problem (Context.newton_solve), from the
            host's previous solution to the new one on the host
  assemble  residual and Jacobian of a 2p problem at a new solution, the residual read back
            (the assembler alone, as a user's own Newton loop calls it)
  ensemble  several independent 2p problems advanced one time step together (Batch), from
            admission to their solutions on the host

The problem tables (grid, permeability field, boundary values) and the uploaded context are
what a program keeps between calls and belong to prepare(); the solution vectors go in and
come out in run().
"""
import math

import numpy as np
import torch

from dumux_gb300 import Batch, Context, FVAssembler, ILUBiCGSTABIstlSolver, newton_params, problems

DT = 250.0   # s, the initial time step of the 2p test problems


def listed():
    return [
        # the reference's 1p lens test: the smallest problem anyone runs, all launches and latency
        dict(name="lens1p_10x10", call="linear", problem="lens1p", nx=10, ny=10, nz=1, reduction=1e-13),
        # the 1p workload of the benchmark: 100 x 100, one solve to 1e-12
        dict(name="darcy_100x100", call="linear", problem="darcy", nx=100, ny=100, nz=1, reduction=1e-12),
        # the reference's 2p Van Genuchten lens test (2D, 2x2 blocks)
        dict(name="lens2p_48x32", call="step", problem="lens2p", nx=48, ny=32, nz=1, precision="fp64", solver="ilu"),
        # the benchmark's headline: plain FP64, natural-order ILU(0)-BiCGSTAB
        dict(name="dnapl_64x64x32", call="step", problem="dnapl", nx=64, ny=64, nz=32, precision="fp64", solver="ilu"),
        # an odd grid of the served and ensemble range in mixed precision
        dict(name="dnapl_45x37x23_mixed", call="step", problem="dnapl", nx=45, ny=37, nz=23, precision="mixed",
             solver="ilu"),
        # the two other preconditioners at the headline size, as the benchmark's forms run them
        dict(name="dnapl_64x64x32_redblack", call="step", problem="dnapl", nx=64, ny=64, nz=32, precision="mixed",
             solver="redblack"),
        dict(name="dnapl_64x64x32_amg", call="step", problem="dnapl", nx=64, ny=64, nz=32, precision="mixed",
             solver="amg"),
        # the largest configuration (1,048,576 cells) in its fastest form
        dict(name="dnapl_128x128x64_amg", call="step", problem="dnapl", nx=128, ny=128, nz=64, precision="mixed",
             solver="amg"),
        # MPFA-O: the reference's convergence test on a fine grid, and the 2p model with full tensors
        dict(name="mpfa1p_256x256", call="linear", problem="mpfa1p", nx=256, ny=256, nz=1, reduction=1e-12),
        dict(name="mpfa2p_32x32x16", call="step", problem="mpfa2p", nx=32, ny=32, nz=16, precision="fp64",
             solver="ilu"),
        # the assembler alone at the headline size
        dict(name="assemble_64x64x32", call="assemble", problem="dnapl", nx=64, ny=64, nz=32),
        # a small ensemble of uneven grids, mixed precision, natural-order ILU(0)
        dict(name="ensemble_12", call="ensemble", problem="dnapl", count=12, nmin=16, nmax=40, precision="mixed",
             solver="ilu"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lens1p", "darcy", "lens2p", "dnapl", "dnapl", "dnapl", "mpfa1p", "mpfa2p", "assemble",
                       "ensemble"])
    if kind in ("lens1p", "darcy"):
        n = [_log(rng, 10, 60 if kind == "lens1p" else 128) for _ in range(2)]
        return dict(call="linear", problem=kind, nx=n[0], ny=n[1], nz=1, reduction=rng.choice([1e-12, 1e-13]))
    if kind == "lens2p":
        return dict(call="step", problem=kind, nx=_log(rng, 16, 72), ny=_log(rng, 12, 64), nz=1,
                    precision=rng.choice(["fp64", "mixed"]), solver="ilu")
    if kind == "dnapl":
        precision, solver = rng.choice([("fp64", "ilu"), ("mixed", "ilu"), ("mixed", "redblack"), ("fp64", "redblack"),
                                        ("mixed", "amg"), ("fp64", "amg")])
        return dict(call="step", problem=kind, nx=_log(rng, 16, 72), ny=_log(rng, 16, 72), nz=_log(rng, 8, 32),
                    precision=precision, solver=solver)
    if kind == "mpfa1p":
        n = _log(rng, 32, 256)
        return dict(call="linear", problem=kind, nx=n, ny=n, nz=1, reduction=1e-12)
    if kind == "mpfa2p":
        return dict(call="step", problem=kind, nx=_log(rng, 10, 32), ny=_log(rng, 10, 32), nz=_log(rng, 6, 16),
                    precision="fp64", solver="ilu")
    if kind == "assemble":
        return dict(call="assemble", problem="dnapl", nx=_log(rng, 16, 128), ny=_log(rng, 16, 128), nz=_log(rng, 8, 64))
    return dict(call="ensemble", problem="dnapl", count=rng.randint(4, 12), nmin=16, nmax=rng.randint(20, 40),
                precision=rng.choice(["fp64", "mixed"]), solver=rng.choice(["ilu", "ilu", "amg"]))


# ---------------------------------------------------------------- inputs
def _cells(case):
    n = (case["nx"], case["ny"], case["nz"])
    return n[:2] if case["problem"] in ("lens1p", "darcy", "lens2p", "mpfa1p") else n


def _problem(case, seed):
    """(desc, u0) of one case; every input follows from the seed."""
    rng = np.random.default_rng(seed)
    cells, kind = _cells(case), case["problem"]
    if kind == "mpfa1p":
        desc, u0, _ = problems.mpfa_convergence_problem(cells[0], c=float(rng.uniform(0.5, 0.95)))
        return desc, u0
    if kind == "darcy":
        return problems.darcy_1p(cells=cells, seed=seed)
    if kind in ("lens1p", "lens2p"):
        # the reference's fixed permeabilities with a seeded 20% perturbation per cell
        desc, u0 = (problems.onep_lens_problem if kind == "lens1p" else problems.twop_lens_problem)(cells)
        desc.permeability *= np.exp(0.2 * rng.standard_normal(desc.num_cells))
        return desc, u0
    build = problems.dnapl_2p_mpfa if kind == "mpfa2p" else problems.dnapl_2p
    return build(cells=cells, seed=seed, inflow=float(rng.uniform(0.03, 0.05)))


def _ensemble(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["count"]):
        # the grids belong to the case, the fields to the seed
        grid = np.random.default_rng(1000 + i)
        cells = tuple(int(v) for v in grid.integers(case["nmin"], case["nmax"] + 1, size=3))
        out.append(problems.dnapl_2p(cells=cells, seed=seed * 100 + i, sigma=float(rng.uniform(0.5, 2.0)),
                                     corr_len=float(rng.uniform(3.0, 10.0)), inflow=float(rng.uniform(0.01, 0.08))))
    return out


def _dt(case):
    # the finest grid's first step does not converge at 250 s; its time loop starts lower
    return DT if case.get("nx", 0) * case.get("ny", 0) * case.get("nz", 0) <= 400000 else DT / 4


def _params(case):
    # the weaker or single-precision ILU(0) forms run with a higher iteration cap
    return newton_params(linear_max_iter=1000)


def prepare(case, seed):
    call = case["call"]
    if call == "ensemble":
        batch = Batch(precision=case["precision"], solver=case["solver"])
        return dict(call=call, batch=batch, members=_ensemble(case, seed), params=_params(case))
    desc, u0 = _problem(case, seed)
    if call == "linear":
        return dict(call=call, assembler=FVAssembler(desc), u=u0,
                    solver=ILUBiCGSTABIstlSolver(residual_reduction=case["reduction"], max_iter=1000))
    if call == "assemble":
        return dict(call=call, assembler=FVAssembler(desc, prev_sol=u0, dt=DT), u=_developed(desc, u0, seed))
    ctx = Context(desc, precision=case["precision"])
    if case["solver"] == "amg":
        ctx.set_linear_solver("amg")
    elif case["solver"] == "redblack":
        ctx.set_ilu_kernel("redblack")
    return dict(call=call, ctx=ctx, u=u0, dt=_dt(case), params=_params(case))


def _developed(desc, u0, seed):
    """A developed state: DNAPL saturations up to 0.6 over a third of the cells, the pressure disturbed."""
    rng = np.random.default_rng(seed + 7)
    u = u0.reshape(-1, 2).copy()
    u[:, 0] *= 1.0 + 1e-3 * rng.standard_normal(len(u))
    u[:, 1] = 0.6 * np.clip(rng.uniform(-2.0, 1.0, len(u)), 0.0, None)
    return u.reshape(-1)


def run(state):
    call = state["call"]
    if call == "linear":
        asm = state["assembler"]
        asm.assemble_jacobian_and_residual(state["u"])
        _, x = state["solver"].solve(asm)
        return {"x": x, "residual": asm.residual()}
    if call == "assemble":
        asm = state["assembler"]
        asm.assemble_jacobian_and_residual(state["u"])
        return {"residual": asm.residual()}
    if call == "step":
        ctx = state["ctx"]
        ctx.set_prev_solution(state["u"])
        ctx.set_solution(state["u"])
        report = ctx.newton_solve(state["dt"], state["params"])
        return {"u": ctx.solution(), "dt": report["dt_used"]}
    batch = state["batch"]
    ids = [batch.add(desc, u0, dt=DT, t_end=DT, params=state["params"]) for desc, u0 in state["members"]]
    batch.run()
    out = [batch.solution(i) for i in ids]
    for i in ids:
        batch.remove(i)
    return out


# ---------------------------------------------------------------- work
def work(case):
    """One pass's unavoidable work: the problem tables and the solution read once, the result
    written once; the arithmetic of one assembly and one operator product per Newton iteration
    (at least two for a nonlinear step).  Krylov iterations depend on the data and are not counted."""
    if case["call"] == "ensemble":
        cells = 0
        for i in range(case["count"]):
            n = np.random.default_rng(1000 + i).integers(case["nmin"], case["nmax"] + 1, size=3)
            cells += int(n[0] * n[1] * n[2])
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    b = 1 if case["call"] == "linear" else 2
    dim = 2 if case.get("nz", 3) == 1 else 3
    newton = 2 if case["call"] in ("step", "ensemble") else 1
    faces = 2 * dim
    vectors = 8 * b * (3 if case["call"] == "step" else 2)
    tables = 8 * (dim * dim + 1 if case["problem"] in ("mpfa1p", "mpfa2p") else 2)
    per_cell = faces * (1 + b) * 6 * b + 2 * (faces + 1) * b * b
    return {"bytes": float(cells * (vectors + tables)), "flops": float(cells * newton * per_cell)}


# ---------------------------------------------------------------- exact results in 64 bits
# A plain torch restatement of the discrete equations: cells as (nz, ny, nx) arrays, faces as
# shifted slices, the Jacobian by forward-mode differentiation of the residual along the
# colours of the stencil, BiCGSTAB with block-Jacobi preconditioning.
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Tpfa:
    def __init__(self, desc, dt=None):
        d = self.dev = _device()
        self.dim, self.b = desc.dim, desc.num_eq
        self.shape = tuple(reversed(desc.cells[:3]))
        self.N = desc.num_cells
        t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=d)  # noqa: E731
        grid = lambda a: t(a).reshape(self.shape)  # noqa: E731
        self.K, self.phi = grid(desc.permeability), grid(desc.porosity)
        self.h = []
        for a in range(3):
            w = np.diff(desc.coords[a]) if a < self.dim else np.ones(1)
            s = [1, 1, 1]
            s[2 - a] = len(w)
            self.h.append(t(w).reshape(s).expand(self.shape))
        self.vol = self.h[0] * self.h[1] * self.h[2]
        self.rho, self.mu = desc.density, desc.viscosity
        self.g = desc.gravity if desc.enable_gravity else [0.0] * 3
        self.dt = dt
        self.laws = None
        if self.b == 2:
            mat = np.zeros(self.N, np.int64) if desc.material is None else desc.material.astype(np.int64)
            self.kind = desc.material_law
            self.laws = [_law_constants(self.kind, p) for p in desc.material_params]
            self.mat = torch.as_tensor(mat, device=d).reshape(self.shape)
        self.bc, at = [], 0
        for f in range(2 * self.dim):
            a = f // 2
            s = [n for k, n in enumerate(self.shape) if k != 2 - a]
            n = int(np.prod(s))
            kinds = torch.as_tensor(desc.bc_type[at:at + n].astype(np.int64), device=d).reshape(s).unsqueeze(2 - a)
            vals = t(desc.bc_values.reshape(-1, self.b)[at:at + n]).reshape(s + [self.b]).unsqueeze(2 - a)
            self.bc.append((kinds, vals))
            at += n

    def states(self, u, where=None):
        """Phase pressures and rho*mobility of states u (..., b)."""
        if self.b == 1:
            return [u[..., 0]], [torch.full_like(u[..., 0], self.rho[0] / self.mu[0])]
        mat = self.mat if where is None else self.mat[where]
        sw = 1 - u[..., 1]
        pc, kw, kn = torch.zeros_like(sw), torch.zeros_like(sw), torch.zeros_like(sw)
        for m, law in enumerate(self.laws):
            v = _law(self.kind, law, sw)
            pc, kw, kn = (torch.where(mat == m, x, y) for x, y in zip(v, (pc, kw, kn)))
        return [u[..., 0], u[..., 0] + pc], [self.rho[0] * kw / self.mu[0], self.rho[1] * kn / self.mu[1]]

    def storage(self, u):
        return [self.phi * self.rho[0] * (1 - u[..., 1]), self.phi * self.rho[1] * u[..., 1]]

    def residual(self, u, prev=None):
        """u: (nz, ny, nx, b)."""
        p, mob = self.states(u)
        r = [torch.zeros_like(p[0]) for _ in range(self.b)]
        if prev is not None and self.b == 2:
            r = [(s - q) * self.vol / self.dt for s, q in zip(self.storage(u), self.storage(prev))]
        for a in range(self.dim):
            ax, n = 2 - a, self.shape[2 - a]
            cut = lambda x, lo, hi: x.narrow(ax, lo, hi - lo)  # noqa: E731
            half = self.h[a] / (2 * self.K)
            area = self.vol / self.h[a]
            if n > 1:
                T = cut(area, 0, n - 1) / (cut(half, 0, n - 1) + cut(half, 1, n))
                dx = (cut(self.h[a], 0, n - 1) + cut(self.h[a], 1, n)) / 2
                for k in range(self.b):
                    F = T * (cut(p[k], 0, n - 1) - cut(p[k], 1, n) + self.rho[k] * self.g[a] * dx)
                    F = F * torch.where(F < 0, cut(mob[k], 1, n), cut(mob[k], 0, n - 1))
                    zero = torch.zeros_like(cut(F, 0, 1))
                    r[k] = r[k] + torch.cat([F, zero], ax) - torch.cat([zero, F], ax)
            for side in range(2):
                kinds, vals = self.bc[2 * a + side]
                at = n - 1 if side else 0
                where = tuple(slice(at, at + 1) if k == ax else slice(None) for k in range(3))
                pb, mb = self.states(vals, where)
                T = (area / half)[where]
                sign = 1.0 if side else -1.0
                for k in range(self.b):
                    F = T * (p[k][where] - pb[k] + self.rho[k] * self.g[a] * sign * self.h[a][where] / 2)
                    F = F * torch.where(F < 0, mb[k], mob[k][where])
                    F = torch.where(kinds == 1, F, vals[..., k] * area[where])
                    pad = [torch.zeros_like(r[k].narrow(ax, 0, at)), F, torch.zeros_like(r[k].narrow(ax, 0, n - 1 - at))]
                    r[k] = r[k] + torch.cat([x for x in pad if x.shape[ax] > 0], ax)
        return torch.stack(r, -1)

    def newton(self, u, prev=None, steps=18, linear=False):
        """The solution of residual = 0 (or the first update's x of a linear problem), or None."""
        for _ in range(steps):
            r = self.residual(u, prev)
            x = self.solve(lambda v: torch.func.jvp(lambda w: self.residual(w, prev), (u,), (v,))[1], r)
            if x is None:
                return None
            if linear:
                return x
            u = u - x
            if float((x.abs() / torch.clamp(u.abs(), min=1.0)).max()) < 1e-11:
                return u
        return None

    def solve(self, derivative, r):
        dim, b, d = self.dim, self.b, self.dev
        S = 2 * dim + 1
        idx = torch.meshgrid(*[torch.arange(n, device=d) for n in self.shape], indexing="ij")
        colour = (idx[2] + 2 * idx[1] + 3 * idx[0]) % S
        J = torch.empty(S, *self.shape, b, b, dtype=torch.float64, device=d)
        for c in range(S):
            for e in range(b):
                v = torch.zeros(*self.shape, b, dtype=torch.float64, device=d)
                v[..., e] = (colour == c).double()
                J[c, ..., e] = derivative(v)
        blocks = []
        for o in range(-dim, dim + 1):
            c = ((colour + o) % S).reshape(1, *self.shape, 1, 1).expand(1, *self.shape, b, b)
            a = {1: 0, 2: 1, 3: 2}.get(abs(o))
            blocks.append((J.gather(0, c)[0], None if a is None else (2 - a, -int(math.copysign(1, o)))))
        inv = torch.linalg.inv(blocks[dim][0])

        def times(M, x):
            return (M * x.unsqueeze(-2)).sum(-1)

        def op(x):
            y = 0
            for M, s in blocks:
                y = y + times(M, x if s is None else torch.roll(x, s[1], s[0]))
            return y
        return _bicgstab(op, lambda x: times(inv, x), r)


def _bicgstab(op, precond, b, reduction=1e-13, most=6000):
    """x with op(x) = b to the reduction (of the block-scaled defect), restarted once; None if it is not reached."""
    x, scale = torch.zeros_like(b), float(torch.linalg.norm(precond(b)))
    if scale == 0.0:
        return x
    best = math.inf
    for _ in range(3):
        r = precond(b - op(x))
        if float(torch.linalg.norm(r)) <= reduction * scale:
            return x
        s0, p = r.clone(), r.clone()
        rho = (s0 * r).sum()
        for k in range(most):
            v = precond(op(p))
            alpha = rho / (s0 * v).sum()
            x = x + alpha * p
            s = r - alpha * v
            t = precond(op(s))
            omega = (t * s).sum() / (t * t).sum()
            x = x + omega * s
            r = s - omega * t
            new = (s0 * r).sum()
            p = r + (new / rho) * (alpha / omega) * (p - omega * v)
            rho = new
            if k % 25 == 24:
                now = float(torch.linalg.norm(r))
                if not math.isfinite(now):
                    return None
                if now <= reduction * scale / 10:
                    break
        best = float(torch.linalg.norm(precond(b - op(x))))
    return x if best <= 1e-10 * scale else None


def _law_constants(kind, p):
    """Regularised Brooks-Corey (0) or Van Genuchten (1): constants of the extensions."""
    c = dict(zip(("pe", "lam", "swr", "snr", "low"), p)) if kind == 0 else \
        dict(zip(("alpha", "n", "l", "swr", "snr", "low", "high", "krn_low", "krw_high"), p))
    if kind == 0:
        c["pc_low"] = c["pe"] * c["low"] ** (-1 / c["lam"])
        c["slope_low"] = -c["pe"] / c["lam"] * c["low"] ** (-1 / c["lam"] - 1)
        c["slope_end"] = -c["pe"] / c["lam"]
        return c
    c["m"] = 1 - 1 / c["n"]
    at = lambda f, s: [float(v) for v in _value_slope(f, c, s)]  # noqa: E731
    c["pc_low"], c["slope_low"] = at(_vg_pc, c["low"])
    hi, slope = at(_vg_pc, c["high"])
    end = 2 * (0 - hi) / (1 - c["high"])
    c["pc_spline"] = (c["high"], 1.0, hi, 0.0, slope, end)
    c["slope_end"] = end
    v, s = at(_vg_krw, c["krw_high"])
    c["krw_spline"] = (c["krw_high"], 1.0, v, 1.0, s, 0.0)
    v, s = at(_vg_krn, c["krn_low"])
    c["krn_spline"] = (0.0, c["krn_low"], 1.0, v, 0.0, s)
    return c


def _value_slope(f, c, s):
    x = torch.tensor(float(s), dtype=torch.float64)
    return torch.func.jvp(lambda y: f(c, y), (x,), (torch.ones_like(x),))


def _vg_pc(c, s):
    return (s ** (-1 / c["m"]) - 1) ** (1 / c["n"]) / c["alpha"]


def _vg_krw(c, s):
    return s ** c["l"] * (1 - (1 - s ** (1 / c["m"])) ** c["m"]) ** 2


def _vg_krn(c, s):
    return (1 - s) ** c["l"] * (1 - s ** (1 / c["m"])) ** (2 * c["m"])


def _hermite(k, x):
    x0, x1, y0, y1, m0, m1 = k
    h = x1 - x0
    t = (x - x0) / h
    return ((1 + 2 * t) * (1 - t) ** 2 * y0 + t * (1 - t) ** 2 * h * m0 + t * t * (3 - 2 * t) * y1
            + t * t * (t - 1) * h * m1)


def _law(kind, c, sw):
    s = (sw - c["swr"]) / (1 - c["swr"] - c["snr"])
    low = c["pc_low"] + c["slope_low"] * (s - c["low"])
    mid = s.clamp(1e-6, 1 - 1e-12)
    one, zero = torch.ones_like(s), torch.zeros_like(s)
    if kind == 0:
        pc = torch.where(s >= 1, c["slope_end"] * (s - 1) + c["pe"], c["pe"] * mid ** (-1 / c["lam"]))
        krw = mid ** (2 / c["lam"] + 3)
        krn = (1 - mid) ** 2 * (1 - mid ** (2 / c["lam"] + 1))
    else:
        pc = torch.where(s > c["high"], _hermite(c["pc_spline"], s), _vg_pc(c, mid.clamp(max=c["high"])))
        pc = torch.where(s >= 1, c["slope_end"] * (s - 1), pc)
        krw = torch.where(s >= c["krw_high"], _hermite(c["krw_spline"], s), _vg_krw(c, mid.clamp(max=c["krw_high"])))
        krn = torch.where(s <= c["krn_low"], _hermite(c["krn_spline"], s), _vg_krn(c, mid.clamp(min=c["krn_low"])))
    pc = torch.where(s <= c["low"], low, pc)
    krw = torch.where(s <= 0, zero, torch.where(s >= 1, one, krw))
    krn = torch.where(s <= 0, one, torch.where(s >= 1, zero, krn))
    return pc, krw, krn


class _Mpfa2d:
    """The O-method of a 1p problem on a 2D grid with Dirichlet values on the whole boundary:
    per grid vertex up to four cells (SW, SE, NW, NE) and four half faces (S, N between the
    cells side by side, W, E between those above each other) with one pressure each."""

    def __init__(self, desc):
        d = self.dev = _device()
        nx, ny = self.nx, self.ny = desc.cells[:2]
        t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=d)  # noqa: E731
        K = t(desc.permeability_tensor).reshape(ny, nx, 2, 2)
        hx, hy = t(np.diff(desc.coords[0])), t(np.diff(desc.coords[1]))
        sides, at = [], 0
        for n in (ny, ny, nx, nx):
            sides.append(t(desc.bc_values[at:at + n]))
            at += n
        self.scale = desc.density[0] / desc.viscosity[0]
        self.source = t(np.zeros(nx * ny) if desc.source is None else desc.source).reshape(ny, nx) * hy[:, None] * hx
        z = dict(dtype=torch.float64, device=d)
        V = (ny + 1, nx + 1)
        # C[v, cell]: outward fluxes through the cell's vertical (x) and horizontal (y) half
        # face as rows over (p_cell, p_xface, p_yface)
        self.rows = torch.zeros(*V, 4, 2, 3, **z)
        self.valid = torch.zeros(*V, 4, dtype=torch.bool, device=d)
        self.cut = []
        for q in range(4):
            east, north = q & 1, q >> 1
            ys = slice(1, ny + 1) if not north else slice(0, ny)
            xs = slice(1, nx + 1) if not east else slice(0, nx)
            self.cut.append((ys, xs))
            gx = (-1.0 if east else 1.0)     # direction from the cell centre to its x face
            gy = (-1.0 if north else 1.0)
            ax, ay = gx * 2 / hx[None, :], gy * 2 / hy[:, None]
            r = torch.zeros(ny, nx, 2, 3, **z)
            for f, (nrm, area) in enumerate(((0, hy[:, None] / 2), (1, hx[None, :] / 2))):
                s = gx if nrm == 0 else gy
                kx, ky = K[..., nrm, 0] * ax, K[..., nrm, 1] * ay
                r[..., f, 0] = s * area * (kx + ky)
                r[..., f, 1] = -s * area * kx
                r[..., f, 2] = -s * area * ky
            self.rows[ys, xs, q] = r
            self.valid[ys, xs, q] = True
        # half faces: S (SW|SE), N (NW|NE), W (SW|NW), E (SE|NE); the x and y face of a cell
        self.face = [(0, 2), (0, 3), (1, 2), (1, 3)]
        self.pair = [(0, 1), (2, 3), (0, 2), (1, 3)]
        A = torch.zeros(*V, 4, 4, **z)
        known = torch.zeros(*V, 4, **z)
        for f, (c0, c1) in enumerate(self.pair):
            both = self.valid[..., c0] & self.valid[..., c1]
            for c in (c0, c1):
                row = self.rows[..., c, 0 if f < 2 else 1, :]
                A[..., f, self.face[c][0]] += torch.where(both, row[..., 1], 0.0)
                A[..., f, self.face[c][1]] += torch.where(both, row[..., 2], 0.0)
            A[..., f, f] = torch.where(both, A[..., f, f], torch.ones_like(A[..., f, f]))
        known[1:, 0, 0], known[:-1, 0, 1] = sides[0], sides[0]
        known[1:, nx, 0], known[:-1, nx, 1] = sides[1], sides[1]
        known[0, 1:, 2], known[0, :-1, 3] = sides[2], sides[2]
        known[ny, 1:, 2], known[ny, :-1, 3] = sides[3], sides[3]
        self.inv, self.known = torch.linalg.inv(A), known

    def fluxes(self, p, known):
        """Sum of the outward fluxes of every cell."""
        V = (self.ny + 1, self.nx + 1)
        pc = torch.zeros(*V, 4, dtype=torch.float64, device=self.dev)
        for q, (ys, xs) in enumerate(self.cut):
            pc[ys, xs, q] = p
        rhs = known.clone()
        for f, (c0, c1) in enumerate(self.pair):
            both = self.valid[..., c0] & self.valid[..., c1]
            w = 0 if f < 2 else 1
            s = self.rows[..., c0, w, 0] * pc[..., c0] + self.rows[..., c1, w, 0] * pc[..., c1]
            rhs[..., f] = torch.where(both, -s, rhs[..., f])
        pf = (self.inv * rhs.unsqueeze(-2)).sum(-1)
        out = torch.zeros_like(p)
        for q, (ys, xs) in enumerate(self.cut):
            fx, fy = self.face[q]
            v = torch.stack([pc[..., q], pf[..., fx], pf[..., fy]], -1)[ys, xs]
            out = out + (self.rows[ys, xs, q] * v.unsqueeze(-2)).sum((-1, -2))
        return out * self.scale

    def residual_and_x(self, u):
        p = torch.as_tensor(u, device=self.dev).reshape(self.ny, self.nx)
        r = self.fluxes(p, self.known) - self.source
        zero = torch.zeros_like(self.known)
        diag = torch.zeros_like(p)
        for q, (ys, xs) in enumerate(self.cut):
            diag = diag + self.rows[ys, xs, q, :, 0].sum(-1) * self.scale
        return r, _bicgstab(lambda x: self.fluxes(x, zero), lambda x: x / diag, r)


def exact(case, seed):
    if case["call"] == "ensemble" or case["problem"] == "mpfa2p":
        return None   # a dozen nonlinear solves, or a 3D O-method: beyond the time such a check may take
    if case["call"] != "linear" and case["call"] != "assemble" and case["nx"] * case["ny"] * case["nz"] > 45000:
        return None   # unpreconditioned Newton-Krylov at this size takes longer than that too
    desc, u0 = _problem(case, seed)
    flat = lambda x: None if x is None else x.reshape(-1).cpu().numpy()  # noqa: E731
    if case["problem"] == "mpfa1p":
        r, x = _Mpfa2d(desc).residual_and_x(u0)
        return {"x": flat(x), "residual": flat(r)}
    if case["call"] == "linear":
        m = _Tpfa(desc)
        u = torch.as_tensor(u0, device=m.dev).reshape(*m.shape, m.b)
        return {"x": flat(m.newton(u, linear=True)), "residual": flat(m.residual(u))}
    dt = DT if case["call"] == "assemble" else _dt(case)
    m = _Tpfa(desc, dt)
    prev = torch.as_tensor(u0, device=m.dev).reshape(*m.shape, 2)
    if case["call"] == "assemble":
        u = torch.as_tensor(_developed(desc, u0, seed), device=m.dev).reshape(*m.shape, 2)
        return {"residual": flat(m.residual(u, prev))}
    return {"u": flat(m.newton(prev, prev)), "dt": None}
