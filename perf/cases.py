"""Workloads by which the library's speed is measured, each through its public entry points.

A case is a dict of plain values. `prepare` builds what a user's program holds before the call (a
cavity, batch or adjoint handle, its input fields on the GPU, buffers for the results), `run` makes
one pass, `work` counts the bytes and operations a pass cannot do without, and `exact` computes
the same outputs with plain torch in FP64.
"""
from __future__ import annotations

import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluid-dynamics1_gb300"))
import cnv_torch  # noqa: E402
import cnvpy  # noqa: E402

DEV = "cuda"
F64 = torch.float64

# ------------------------------------------------------------------------------------- cases
# kind      entry point
# step      Cavity.set_fields_device, Cavity.step(steps), Cavity.get_fields_device
# poisson   cnv_poisson_device on one right-hand side
# batch     Batch.reset, Batch.step(steps), cnv_batch_get_fields of every cavity
# rollout   cnv_torch.CavityRollout forward and backward of the final enstrophy


def _case(name, kind, n, **kw):
    c = dict(name=name, kind=kind, n=n, steps=1, order=6, Lx=1, Re=1000.0, solver="sor", precision="fp64",
             tol=1e-6, omega=0.0, walls=False, field="flow", count=0)
    c.update(kw)
    return c


def listed():
    return [
        # the reference's own command-line configuration: 64^2, Re 100, SOR factor 1.5
        _case("sor_64", "step", 64, Re=100.0, omega=1.5),
        # an odd grid, fourth order, all eight wall velocities, unequal spacing, at the reference's
        # default tolerance: a configuration file that uses every boundary key
        _case("sor_97_walls", "step", 97, order=4, Lx=2, Re=400.0, tol=1e-3, walls=True, steps=2),
        # a mid-size run of the reference's solver
        _case("sor_256", "step", 256),
        # the benchmark's headline: one FP64 step of the 1024^2 cavity with the reference's rounding
        _case("sor_1024", "step", 1024),
        # a Poisson solve alone, as a caller that keeps its own time loop uses it: ragged grid, the
        # FMA arithmetic
        _case("poisson_fma_500", "poisson", 500, precision="fma"),
        # the mixed-precision step of the 1024^2 cavity
        _case("mixed_1024", "step", 1024, precision="mixed"),
        # the mixed-precision step from smoothed noise (decaying turbulence in a box), the largest grid
        _case("mixed_2048", "step", 2048, precision="mixed", field="noise"),
        # a small cavity marched with the exact solve: launches and latency count
        _case("direct_130", "step", 130, solver="direct", steps=20),
        # the exact solve on a ragged grid
        _case("direct_1000", "step", 1000, solver="direct", steps=5),
        # the exact solve from smoothed noise on the largest grid
        _case("direct_2048", "step", 2048, solver="direct", field="noise", steps=3),
        # a parameter sweep: many cavities of uneven size, Reynolds number and lid speed from rest
        _case("batch_128", "batch", 0, count=128, steps=4),
        # the gradient of the final enstrophy with respect to the initial vorticity and lid speed
        _case("rollout_256", "rollout", 256, solver="direct", steps=100),
    ]


def _size(rng, lo, hi):
    """Log-uniform over [lo, hi]; half the time odd, a quarter a multiple of 32."""
    n = round(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    r = rng.random()
    if r < 0.5:
        n |= 1
    elif r < 0.75:
        n = (n + 16) // 32 * 32
    return max(lo, min(hi, n))


def draw(rng):
    kind = rng.choice(["sor", "sor", "mixed", "mixed", "direct", "direct", "poisson", "batch", "rollout"])
    re = round(math.exp(rng.uniform(math.log(100), math.log(2000))), 1)
    order = rng.choice([2, 4, 6, 6, 6])
    lx = rng.choice([1, 1, 1, 2])
    field = rng.choice(["flow", "noise"])
    if kind == "sor":
        c = _case("", "step", _size(rng, 48, 1024), order=order, Lx=lx, Re=re, walls=rng.random() < 0.3, field=field,
                  tol=rng.choice([1e-3, 1e-6]))
        c["solver"] = rng.choice(["sor", "sor", "gs"]) if c["n"] <= 64 else "sor"
        if c["n"] > 700:
            c["Lx"] = 1  # unequal spacing takes about twice the sweeps
    elif kind == "mixed":
        c = _case("", "step", _size(rng, 64, 2048), order=order, Lx=lx, Re=re, precision="mixed", field=field)
    elif kind == "direct":
        c = _case("", "step", _size(rng, 64, 2048), order=order, Lx=lx, Re=re, solver="direct", field=field)
        c["steps"] = 20 if c["n"] < 300 else 4
    elif kind == "poisson":
        c = _case("", "poisson", _size(rng, 64, 1024), Lx=lx, solver=rng.choice(["sor", "direct"]), field=field)
        if c["solver"] == "sor":
            c["precision"] = rng.choice(["fp64", "fma", "mixed"])
    elif kind == "batch":
        c = _case("", "batch", 0, count=rng.randint(8, 128), steps=rng.randint(1, 4), order=order)
    else:
        c = _case("", "rollout", _size(rng, 64, 300), order=order, Re=re, solver="direct", steps=rng.randint(20, 100))
    del c["name"]
    return c


# ------------------------------------------------------------------------------------ inputs
def _dt(n, lx, re, u):
    h = 1.0 / n  # dy; dx = lx / n is not smaller
    return 0.2 * min(h * h * re / 4, h / u)


def _walls(c):
    """u1..u4, v1..v4: the lid alone, or all eight wall velocities."""
    if c["walls"]:
        return (0.1, -0.05, 0.2, 0.8), (0.3, -0.2, 0.05, 0.1)
    return (0.0, 0.0, 0.0, 1.0), (0.0, 0.0, 0.0, 0.0)


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * seed + 17)
    return g


def _flow(n, lx, g):
    """w, u, v of a developed cavity flow: a primary vortex and seeded smaller ones, psi = 0 on the walls."""
    k = torch.arange(1, 9, dtype=F64, device=DEV)
    amp = 0.03 * torch.randn(8, 8, generator=g, dtype=F64, device=DEV) / (k[:, None] ** 2 + k[None, :] ** 2)
    amp[0, 0] -= 0.09
    s = torch.arange(n, dtype=F64, device=DEV) / (n - 1) * math.pi
    sy, cy = torch.sin(torch.outer(s, k)), torch.cos(torch.outer(s, k))
    ky, kx = k * math.pi * n / (n - 1), k * math.pi * n / (n - 1) / lx
    u = (cy * ky) @ amp @ sy.T
    v = -sy @ (amp * kx) @ cy.T
    w = sy @ (amp * (ky[:, None] ** 2 + kx[None, :] ** 2)) @ sy.T
    return w.contiguous(), u.contiguous(), v.contiguous()


def _noise(n, g):
    """Seeded Gaussian vorticity smoothed by 8 Jacobi averaging passes, at rest."""
    w = torch.randn(n, n, generator=g, dtype=F64, device=DEV)
    for _ in range(8):
        t = w.clone()
        t[1:-1, 1:-1] = (w[2:, 1:-1] + w[:-2, 1:-1] + w[1:-1, 2:] + w[1:-1, :-2]) / 4
        w = t
    return w, torch.zeros_like(w), torch.zeros_like(w)


def _fields(c, seed):
    g = _gen(seed)
    return _noise(c["n"], g) if c["field"] == "noise" else _flow(c["n"], c["Lx"], g)


def _specs(c, seed):
    """Cavities of a sweep: n over six sizes (the case's, in a mixed order), and from the seed Re in
    [100, 2000] and the lid speed in [0.5, 1.5]."""
    sizes, rng = random.Random(c["count"]), random.Random(1000003 * seed + 29)
    out = []
    for _ in range(c["count"]):
        n, re, lid = sizes.choice([64, 96, 128, 192, 256, 384]), rng.uniform(100, 2000), rng.uniform(0.5, 1.5)
        out.append(dict(n=n, Re=re, lid=lid, dt=_dt(n, 1, re, lid)))
    return out


def _config(c):
    (u1, u2, u3, u4), (v1, v2, v3, v4) = _walls(c)
    return cnvpy.default_config(
        nx=c["n"], ny=c["n"], Lx=c["Lx"], Ly=1, Re=c["Re"], order=c["order"], dt=_dt(c["n"], c["Lx"], c["Re"], 1.0),
        poisson_type={"sor": cnvpy.POISSON_SOR, "gs": cnvpy.POISSON_GS, "direct": cnvpy.POISSON_DIRECT}[c["solver"]],
        precision={"fp64": cnvpy.PREC_FP64, "fma": cnvpy.PREC_FP64_FMA, "mixed": cnvpy.PREC_MIXED}[c["precision"]],
        poisson_tol=c["tol"], poisson_max_it=1000000, sor_omega=c["omega"], u1=u1, u2=u2, u3=u3, u4=u4, v1=v1, v2=v2,
        v3=v3, v4=v4)


def prepare(case, seed):
    c = case
    if c["kind"] == "batch":
        base = cnvpy.default_config(order=c["order"], mixed_rtol=1e-10)
        specs = _specs(c, seed)
        cells = sum(sp["n"] ** 2 for sp in specs)
        # the results of all cavities, one pinned host array per field, a cavity after the other
        out = [torch.empty(cells, dtype=F64).pin_memory() for _ in range(4)]
        return dict(case=c, batch=cnvpy.Batch(base, specs), out=out)
    w, u, v = _fields(c, seed)
    if c["kind"] == "rollout":
        lid = torch.tensor(1.0 + 0.01 * (seed % 7), dtype=F64, device=DEV)
        return dict(case=c, adjoint=cnvpy.Adjoint(_config(c), checkpoint_every=100), w=w, lid=lid)
    st = dict(case=c, cavity=cnvpy.Cavity(_config(c)), w=w, u=u, v=v)
    st["out"] = [torch.empty_like(w) for _ in range(1 if c["kind"] == "poisson" else 4)]
    return st


# -------------------------------------------------------------------------------------- run
def _infos(infos):
    return torch.tensor([r["iters"] for r in infos], dtype=torch.int64)


def run(state):
    c = state["case"]
    if c["kind"] == "batch":
        b = state["batch"]
        b.reset()
        _, last = b.step(c["steps"])
        out, at = state["out"], 0
        for k, sp in enumerate(b.specs):
            ptrs = (cnvpy.C.cast(x.data_ptr() + 8 * at, cnvpy._dp) for x in out)
            cnvpy.check(b._lib.cnv_batch_get_fields(b._h, k, *ptrs), "cnv_batch_get_fields")
            at += sp["n"] ** 2
        return [_infos(last)] + out
    if c["kind"] == "rollout":
        w0 = state["w"].detach().requires_grad_(True)
        lid = state["lid"].detach().requires_grad_(True)
        adj = state["adjoint"]
        wT = cnv_torch.CavityRollout.apply(w0, lid, adj, c["steps"])
        g_w0, g_lid = torch.autograd.grad(cnv_torch.enstrophy(wT, adj.h2), (w0, lid))
        return [wT.detach(), g_w0, g_lid]
    cav, out = state["cavity"], state["out"]
    torch.cuda.current_stream().synchronize()  # the library works on its own stream
    if c["kind"] == "poisson":
        it, err = cnvpy.C.c_int(0), cnvpy.C.c_double(0.0)
        cnvpy.check(cav._lib.cnv_poisson_device(cav._h, state["w"].data_ptr(), out[0].data_ptr(), cnvpy.C.byref(it),
                                                cnvpy.C.byref(err)), "cnv_poisson_device")
        return [torch.tensor([it.value], dtype=torch.int64), out[0]]
    cnvpy.check(cav.set_fields_device(state["w"].data_ptr(), state["u"].data_ptr(), state["v"].data_ptr()))
    _, infos = cav.step(c["steps"])
    cnvpy.check(cav.get_fields_device(*(x.data_ptr() for x in out)))
    return [_infos(infos)] + out


# ------------------------------------------------------------------------------------- work
def _solve_flops(n):
    """Operations of one exact solve by fast transforms (four real transforms of every row)."""
    return 4 * n * 2.5 * n * math.log2(max(n, 2)) + n * n


def work(case):
    c = case
    if c["kind"] == "batch":  # sizes 64 .. 384, uniform over six: 48256 cells on average
        cells = c["count"] * 48256
        return {"bytes": 32.0 * cells, "flops": c["steps"] * c["count"] * (_solve_flops(220) + 123 * 48256)}
    n = c["n"]
    nn = float(n * n)
    if c["kind"] == "rollout":
        return {"bytes": 3 * 8 * nn, "flops": c["steps"] * (2 * _solve_flops(n) + 123 * nn + 200 * nn)}
    if c["kind"] == "poisson":
        base = {"bytes": 16 * nn, "flops": _solve_flops(n)}
    else:
        base = {"bytes": 56 * nn, "flops": c["steps"] * (_solve_flops(n) + 123 * nn)}
    if c["solver"] in ("sor", "gs") and c["precision"] != "mixed":
        # the reference's sweeps are the result (its iteration count and its iterate): about 3.5 n
        # of them at 1e-6 with the optimal factor, a stage of 7 operations per cell
        sweeps = 3.5 * n * (0.5 if c["tol"] > 1e-4 else 1.0) * (1.0 if c["omega"] == 0 and c["solver"] == "sor" else 8.0)
        base["flops"] += c["steps"] * sweeps * 7 * nn
    return base


# ------------------------------------------------------------------------------------ exact
def _diff(n, order, deriv, h):
    """The reference's difference operators: first-order (deriv 1) or 4-point (deriv 2) one-sided
    edge rows, then central stencils of growing width."""
    d = torch.zeros(n, n, dtype=F64)
    central = {(2, 1): [-0.5, 0, 0.5], (4, 1): [1 / 12, -2 / 3, 0, 2 / 3, -1 / 12],
               (6, 1): [-1 / 60, 3 / 20, -3 / 4, 0, 3 / 4, -3 / 20, 1 / 60],
               (2, 2): [1, -2, 1], (4, 2): [-1 / 12, 4 / 3, -5 / 2, 4 / 3, -1 / 12],
               (6, 2): [1 / 90, -3 / 20, 3 / 2, -49 / 18, 3 / 2, -3 / 20, 1 / 90]}
    edge = [-1.0, 1.0] if deriv == 1 else [2.0, -5.0, 4.0, -1.0]
    for i in range(n):
        r = min(i, n - 1 - i, order // 2)
        if r == 0:
            row = edge if i == 0 else ([-1.0, 1.0] if deriv == 1 else edge[::-1])
            at = 0 if i == 0 else n - len(row)
        else:
            row, at = central[(2 * r, deriv)], i - r
        d[i, at:at + len(row)] = torch.tensor(row, dtype=F64)
    return (d / h ** deriv).to(DEV)


class _Plain:
    """One cavity's time step in plain torch FP64."""

    def __init__(self, n, order, lx, re, dt, u_walls, v_walls, solve):
        self.n, self.re, self.dt, self.solve = n, re, dt, solve
        dx, dy = lx / n, 1.0 / n
        self.d1x, self.d1y = _diff(n, order, 1, dx), _diff(n, order, 1, dy)
        self.d2x, self.d2y = _diff(n, order, 2, dx), _diff(n, order, 2, dy)
        self.edge = torch.ones(n, n, dtype=F64, device=DEV)
        self.edge[1:-1, 1:-1] = 0
        self.masks = []  # j = 0, j = n-1 win the corners over i = 0, i = n-1
        for sl in ((slice(None), 0), (slice(None), n - 1), (0, slice(1, n - 1)), (n - 1, slice(1, n - 1))):
            m = torch.zeros(n, n, dtype=F64, device=DEV)
            m[sl] = 1
            self.masks.append(m)
        self.u_walls, self.v_walls = u_walls, v_walls

    def _bc(self, f, walls):
        return f * (1 - self.edge) + sum(m * b for m, b in zip(self.masks, walls))

    def step(self, w, u, v):
        ub, vb = self._bc(u, self.u_walls), self._bc(v, self.v_walls)
        wb = w * (1 - self.edge) + self.edge * (vb @ self.d1x.T - self.d1y @ ub)
        lap = wb @ self.d2x.T + self.d2y @ wb
        wn = (-ub * (wb @ self.d1x.T) - vb * (self.d1y @ wb) + lap / self.re) * self.dt + wb
        psi, it = self.solve(-wn)
        return wn, self.d1y @ psi, -(psi @ self.d1x.T), psi, it


def _sine_solver(n, lx):
    """psi of den psi - dy^2 (up + dn) - dx^2 (lt + rt) = -dx^2 dy^2 f by dense sine transforms."""
    m, dx, dy = n - 2, lx / n, 1.0 / n
    k = torch.arange(1, m + 1, device=DEV)
    S = math.sqrt(2.0 / (m + 1)) * torch.sin((k[:, None] * k[None, :] % (2 * (m + 1))).to(F64) * (math.pi / (m + 1)))
    sk = torch.sin(k.to(F64) * (math.pi / (2 * (m + 1)))) ** 2
    lam = 4 * dy * dy * sk[:, None] + 4 * dx * dx * sk[None, :]

    def solve(f):
        x = S @ ((S @ (f[1:-1, 1:-1] * (-dx * dx * dy * dy)) @ S) / lam) @ S
        return torch.nn.functional.pad(x, (1, 1, 1, 1)), 0

    return solve


def _sor_solver(n, lx, beta, tol):
    """The reference's red-black sweeps from zero, to sum |change| < tol; the 0-based count of the last."""
    dx, dy = lx / n, 1.0 / n
    dx2, dy2 = dx * dx, dy * dy
    den = 2 * (dx2 + dy2)
    idx = torch.arange(1, n - 1, device=DEV)
    odd = (idx[:, None] + idx[None, :]) % 2 == 1

    def solve(f):
        psi = torch.zeros_like(f)
        g = dx2 * dy2 * f[1:-1, 1:-1]
        for it in range(1000000):
            old = psi[1:-1, 1:-1].clone()
            for mask in (~odd, odd):
                p = psi[1:-1, 1:-1]
                new = beta * (dy2 * (psi[2:, 1:-1] + psi[:-2, 1:-1]) + dx2 * (psi[1:-1, 2:] + psi[1:-1, :-2]) - g) / den
                new = new + (1 - beta) * p
                p.copy_(torch.where(mask, new, p))
            if float((psi[1:-1, 1:-1] - old).abs().sum()) < tol:
                return psi, it
        raise RuntimeError("not converged")

    return solve


def _solver(c):
    n = c["n"]
    if c["solver"] == "direct" or c["precision"] == "mixed":
        return _sine_solver(n, c["Lx"])
    beta = 1.0 if c["solver"] == "gs" else c["omega"] or 2 / (1 + math.sin(3.14159265359 / (n + 1)))
    return _sor_solver(n, c["Lx"], beta, c["tol"])


def exact(case, seed):
    c = case
    if c["kind"] == "batch":
        out, solvers = [[], [], [], []], {}
        for sp in _specs(c, seed):
            n = sp["n"]
            if n not in solvers:
                solvers[n] = _sine_solver(n, 1)
            p = _Plain(n, c["order"], 1, sp["Re"], sp["dt"], (0.0, 0.0, 0.0, sp["lid"]), (0.0,) * 4, solvers[n])
            w = u = v = torch.zeros(n, n, dtype=F64, device=DEV)
            for _ in range(c["steps"]):
                w, u, v, psi, _ = p.step(w, u, v)
            for all_of, x in zip(out, (w, u, v, psi)):
                all_of.append(x.reshape(-1))
        return [None] + [torch.cat(x) for x in out]
    w, u, v = _fields(c, seed)
    solve = _solver(c)
    # counts of the mixed solve's corrections have no plain counterpart
    counted = c["precision"] != "mixed" and c["precision"] != "fma"
    if c["kind"] == "poisson":
        psi, it = solve(w)
        return [torch.tensor([it], dtype=torch.int64) if counted else None, psi]
    uw, vw = _walls(c)
    if c["kind"] == "rollout":
        w0 = w.detach().requires_grad_(True)
        lid = torch.tensor(1.0 + 0.01 * (seed % 7), dtype=F64, device=DEV, requires_grad=True)
        p = _Plain(c["n"], c["order"], c["Lx"], c["Re"], _dt(c["n"], c["Lx"], c["Re"], 1.0), uw[:3] + (lid,), vw, solve)
        wt, u, v = w0, torch.zeros_like(w), torch.zeros_like(w)
        for _ in range(c["steps"]):
            wt, u, v, _, _ = p.step(wt, u, v)
        h2 = (c["Lx"] / c["n"]) * (1.0 / c["n"])
        g_w0, g_lid = torch.autograd.grad(0.5 * h2 * (wt * wt).sum(), (w0, lid))
        return [wt.detach(), g_w0, g_lid]
    p = _Plain(c["n"], c["order"], c["Lx"], c["Re"], _dt(c["n"], c["Lx"], c["Re"], 1.0), uw, vw, solve)
    its = []
    for _ in range(c["steps"]):
        w, u, v, psi, it = p.step(w, u, v)
        its.append(it)
    return [torch.tensor(its, dtype=torch.int64) if counted else None, w, u, v, psi]
