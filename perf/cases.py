"""The work that a user of the library has it do, as cases that can be timed and compared.

Three kinds of case, each through the public Python binding (dfdm.native):

  step     one simulation: upload a velocity field, take `steps` RK3 steps, download U, V, W and P (what a host program
           does between two snapshots);
  group    a serving group: several small simulations uploaded, stepped together, downloaded;
  poisson  one pressure solve from host array to host array (solve_poisson_equation), for the periodic and channel
           grids and for the grids that the library serves with the pressure solve alone.

Host arrays are pinned, FP64, Fortran-ordered, in the ghosted shapes of the C ABI.  exact() restates the same
computations in FP64 torch, without the library.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "dopamine-fdm_b200"))

from dfdm import cases as grids  # noqa: E402
from dfdm.native import Group, Solver  # noqa: E402

F64 = torch.float64
KAPPA = 0.41


def _step(name, wall, nx, ny, nz, lx, lz, alpha, re, dt, steps, precision, graphs=True, sgs=0, wall_model=0, scheme=0,
          order=3, adaptive=False, flux=True):
    c = {"kind": "step", "wall": wall, "nx": nx, "ny": ny, "nz": nz, "lx": lx, "lz": lz, "alpha": alpha, "re": re,
         "dt": dt, "steps": steps, "precision": precision, "graphs": graphs, "sgs": sgs, "wall_model": wall_model,
         "scheme": scheme, "order": order, "adaptive": adaptive, "flux": flux}
    if name:
        c["name"] = name
    return c


def _poisson(name, bc, nx, ny, nz, precision):
    c = {"kind": "poisson", "bc": bc, "nx": nx, "ny": ny, "nz": nz, "precision": precision}
    if name:
        c["name"] = name
    return c


def listed():
    pi = math.pi
    return [
        # the smallest call: the reference's 16^3 regression channel in FP64, with the binding's defaults (no step graph)
        _step("channel16_fp64", True, 16, 16, 16, 3.0, 1.5, 0.0, 200.0, 2e-3, 20, "fp64", graphs=False, flux=False),
        # the Taylor-Green box of the benchmark: a small grid, where launches count
        _step("tgv64_fp32", False, 64, 64, 64, 2 * pi, 2 * pi, 0.0, 1600.0, 1e-3, 100, "fp32", flux=False),
        # many small simulations served together
        {"name": "group16x32_fp32", "kind": "group", "members": 16, "n": 32, "dt": 1e-3, "steps": 60},
        # channel DNS at Re_tau = 180: the mid-size production run in both precisions
        _step("chan180_fp32", True, 128, 96, 128, 4 * pi, 4 * pi / 3, 2.0, 180.0, 2e-3, 100, "fp32"),
        _step("chan180_fp64", True, 128, 96, 128, 4 * pi, 4 * pi / 3, 2.0, 180.0, 2e-3, 40, "fp64"),
        # wall-modelled LES at Re_tau = 395 (AMD closure), driven by the pressure gradient
        _step("les395_fp32", True, 96, 64, 96, 2 * pi, pi, 1.5, 395.0, 1e-3, 100, "fp32", sgs=2, wall_model=1,
              flux=False),
        # LES with the Vreman closure in FP64 on ragged sizes, whose x and z lengths take the general transforms
        _step("les_vreman_ragged_fp64", True, 90, 53, 60, 2 * pi, pi, 1.5, 395.0, 1e-3, 30, "fp64", sgs=1, wall_model=1,
              flux=False),
        # the upwind-biased scheme with the adaptive time step on ragged sizes
        _step("hybrid_adaptive_ragged_fp32", True, 150, 73, 120, 2 * pi, pi, 2.0, 300.0, 5e-4, 40, "fp32", scheme=2,
              order=5, adaptive=True),
        # the throughput run, channel DNS at Re_tau = 550 on 12.6 million cells, in both precisions
        _step("chan550_fp32", True, 256, 192, 256, 2 * pi, pi, 2.0, 550.0, 4e-4, 60, "fp32"),
        _step("chan550_fp64", True, 256, 192, 256, 2 * pi, pi, 2.0, 550.0, 4e-4, 20, "fp64"),
        # pressure solves for host codes that step inflow/outflow and duct grids themselves
        _poisson("poisson_inflow_fp32", "inflow", 258, 129, 130, "fp32"),
        _poisson("poisson_duct_fp64", "duct", 258, 129, 130, "fp64"),
    ]


def _smooth(n, even):
    """The next length up from n whose factors are 2, 3 and 5 (twice such a length with even)."""
    m = (n + 1) // 2 if even else n
    while True:
        r = m
        for p in (2, 3, 5):
            while r % p == 0:
                r //= p
        if r == 1:
            return 2 * m if even else m
        m += 1


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["group"] + ["poisson"] * 2)
    if kind == "group":
        return {"kind": "group", "members": rng.randint(2, 24), "n": rng.choice([32, 48, 64]), "dt": 1e-3,
                "steps": rng.randint(20, 60)}
    if kind == "poisson":
        bc = rng.choice(["inflow", "duct", "inflow_duct", "spanwise", "channel", "periodic"])
        xwall, zwall = bc in ("inflow", "inflow_duct"), bc in ("duct", "inflow_duct", "spanwise")
        yper = bc in ("spanwise", "periodic")
        # inflow/outflow grids take any even face count up to 258 (257 x cells)
        nx = 2 * (_log_int(rng, 16, 256) // 2) + 2 if xwall else _smooth(_log_int(rng, 16, 240), True) + 2
        ny = (_smooth(_log_int(rng, 16, 180), True) + 2) if yper else _log_int(rng, 16, 180) + 1
        nz = 2 * (_log_int(rng, 16, 240) // 2) + 2 if zwall else _smooth(_log_int(rng, 16, 240), True) + 2
        return _poisson(None, bc, nx, ny, nz, rng.choice(["fp32", "fp64"]))
    wall = rng.random() < 0.75
    precision = rng.choice(["fp32", "fp32", "fp64"])
    nx, nz = _smooth(_log_int(rng, 16, 240), True), _smooth(_log_int(rng, 16, 240), True)
    ny = _log_int(rng, 12, 190) if wall else _smooth(_log_int(rng, 16, 180), True)
    sgs = rng.choice([0, 0, 0, 1, 2])
    wall_model = 1 if wall and sgs and rng.random() < 0.7 else 0
    scheme = rng.choice([0, 0, 0, 1, 2])
    steps = max(4, min(80, int(1.5e8 / (nx * ny * nz))))
    return _step(None, wall, nx, ny, nz, 2 * math.pi, math.pi if wall else 2 * math.pi, 2.0 if wall else 0.0,
                 round(rng.uniform(150.0, 600.0), 1), 0.0, steps, precision, graphs=rng.random() < 0.8, sgs=sgs,
                 wall_model=wall_model, scheme=scheme, order=rng.choice([3, 5]), adaptive=rng.random() < 0.25,
                 flux=wall and rng.random() < 0.6)


# ---- grids ----------------------------------------------------------------------------------------------------------
def _reichardt(yp):
    return (np.log(1.0 + KAPPA * yp) / KAPPA +
            (5.17 - math.log(KAPPA) / KAPPA) * (1.0 - np.exp(-yp / 11.0) - yp / 11.0 * np.exp(-yp / 3.0)))


def _grid(case):
    """The library's case description (dfdm.cases.Case) of a step or poisson case."""
    if case["kind"] == "poisson":
        bc = case["bc"]
        return grids.Case(name=bc, nx=case["nx"], ny=case["ny"], nz=case["nz"], Lx_i=3.0, Ly_i=2.0, Lz_i=1.5,
                          grid_type=1 if bc in ("spanwise", "periodic") else 2, alpha_grid=2.0,
                          y_bc_type=0 if bc in ("spanwise", "periodic") else 1,
                          x_bc_type=1 if bc in ("inflow", "inflow_duct") else 0,
                          z_bc_type=1 if bc in ("duct", "inflow_duct", "spanwise") else 0, nu=0.01, dt=0.002)
    wall, nx, ny, nz = case["wall"], case["nx"], case["ny"], case["nz"]
    les = case["sgs"] != 0
    c = grids.Case(name="case", nx=nx + 2, ny=ny + (1 if wall else 2), nz=nz + 2, Lx_i=case["lx"] * (nx + 1) / nx,
                   Ly_i=2.0 if wall else 2 * math.pi * (ny + 1) / ny, Lz_i=case["lz"] * (nz + 1) / nz,
                   grid_type=2 if wall and case["alpha"] > 0 else 1, alpha_grid=case["alpha"],
                   y_bc_type=1 if wall else 0, nu=1.0 / case["re"], dt=case["dt"],
                   dPdx=1.0 if wall and not case["flux"] else 0.0, sgs_model=case["sgs"],
                   flat_wall_model_flag=case["wall_model"], advection_scheme=case["scheme"], adv_order=case["order"],
                   flow_forcing_mode=1 if case["flux"] else 0, Ub_target=0.0 if les or not wall else _bulk(case))
    if case["flux"] and les:
        c = c.with_(Ub_target=_bulk(case))
    if not case["dt"]:      # a drawn case: a time step at a convective CFL number of about 0.3, within the viscous limit
        x, y, z = grids.faces(c)
        dx, dy, dz = x[1] - x[0], np.diff(y).min(), z[1] - z[0]
        big = 1.6 * _bulk(case) if wall else 1.0
        noise = 0.15 * big if wall else 1.0
        dt = min(0.3 / (big / dx + noise / dy + noise / dz), 0.1 / (4.0 * c.nu * (dx ** -2 + dy ** -2 + dz ** -2)))
        c = c.with_(dt=float("%.3g" % dt))
    return c


def _bulk(case):
    """The bulk velocity in friction units: 15.6 at Re_tau = 180, the Reichardt profile's mean for LES."""
    if case["sgs"]:
        yp = np.linspace(0.0, case["re"], 4001)
        u = _reichardt(np.maximum(yp, 1e-10))
        return float((0.5 * (u[1:] + u[:-1])).mean())
    return 15.6 * (case["re"] / 180.0) ** (1.0 / 7.0)


def _members(case):
    """The simulations of a group: half Taylor-Green boxes of different Re, half channels, on n^3 cells."""
    out = []
    for m in range(case["members"]):
        n = case["n"]
        if m % 2:
            out.append(_step(None, True, n, n, n, 4 * math.pi, 4 * math.pi / 3, 2.0, 180.0, case["dt"], case["steps"], "fp32"))
        else:
            out.append(_step(None, False, n, n, n, 2 * math.pi, 2 * math.pi, 0.0, 400.0 * 2.0 ** (m % 7 / 2), case["dt"],
                             case["steps"], "fp32", flux=False))
    return out


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _velocity(case, seed):
    """The start velocity on the independent cells, [z][y][x] in FP64: a Taylor-Green vortex of random amplitude and
    phase with 1 % noise, a laminar channel with 10 % uniform noise, or (LES) the Reichardt mean with 5 % Gaussian noise."""
    c = _grid(case)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(1000003 * int(seed) + 17)
    x, y, z = (torch.from_numpy(a).to(dev) for a in grids.faces(c))
    mid = lambda f: 0.5 * (f[1:] + f[:-1])
    shape = (nz, ny, nx)
    uni = lambda a: a * (2.0 * torch.rand(shape, generator=gen, device=dev, dtype=F64) - 1.0)
    if not case["wall"]:
        r = torch.rand(3, generator=gen, device=dev, dtype=F64).tolist()
        amp, px, pz = 0.75 + 0.5 * r[0], 2 * math.pi * r[1], 2 * math.pi * r[2]
        cos, sin = torch.cos, torch.sin
        xf, xc = x[1:nx + 1] + px, mid(x)[:nx] + px
        yf, yc = y[1:ny + 1], mid(y)[:ny]
        kx = 2 * math.pi / case["lx"]
        cz = cos(2 * math.pi / case["lz"] * mid(z)[:nz] + pz)[:, None, None]
        u = amp * sin(kx * xf)[None, None, :] * cos(yc)[None, :, None] * cz + uni(0.01)
        v = -amp * kx * cos(kx * xc)[None, None, :] * sin(yf)[None, :, None] * cz + uni(0.01)
        return u, v, uni(0.01)
    yc = mid(y)
    if case["sgs"]:
        wall_distance = torch.minimum(yc, 2.0 - yc).cpu().numpy() * case["re"]
        prof = torch.from_numpy(_reichardt(wall_distance)).to(dev)
        noise = lambda: 0.05 * _bulk(case) * torch.randn(shape, generator=gen, device=dev, dtype=F64)
    else:
        ub = _bulk(case)
        prof = 1.5 * ub * (1.0 - (yc - 1.0) ** 2)
        noise = lambda: uni(0.15 * ub)
    u = prof[None, :, None] + noise()
    v, w = noise(), noise()
    v[:, ny - 1] = 0.0      # the top wall face
    return u, v, w


def _ghosted(c, kind, f):
    """The independent cells f as the ghosted host array, [z][y][x]: periodic wraps, no-slip mirrors, wall faces zero."""
    n1, n2, n3 = c.shapes()[kind]
    nz, ny, nx = f.shape
    i = (torch.arange(n1) - 1) % nx
    k = (torch.arange(n3) - 1) % nz
    j = torch.arange(n2) - 1
    sign = torch.ones(n2, dtype=F64)
    if c.y_bc_type == 0:
        j = torch.where((j < 0) | (j >= ny), 0, j) if kind == "P" else j % ny
    elif kind == "V":
        sign[(j < 0) | (j >= ny - 1)] = 0.0
    elif kind != "P":
        sign[(j < 0) | (j >= ny)] = -1.0
    j = j.clamp(0, ny - 1)
    g = f[:, :, i.to(f.device)][:, j.to(f.device)][k.to(f.device)]
    return g * sign.to(f.device)[None, :, None]


def _rhs(case, seed):
    """A pressure right-hand side in the shape of rhs_p, [z][y][x]: noise without a mean, as the divergence is."""
    n1, n2, n3 = _grid(case).shapes()["rhs_p"]
    gen = torch.Generator(device=_device())
    gen.manual_seed(1000003 * int(seed) + 29)
    return torch.randn((n3, n2, n1), generator=gen, device=_device(), dtype=F64)


def _pinned(shape):
    return torch.empty(tuple(shape), dtype=F64, pin_memory=torch.cuda.is_available())


def _fortran(t):
    """A [z][y][x] tensor as the Fortran-ordered numpy array (x, y, z) over the same memory."""
    return t.numpy().transpose(2, 1, 0)


def _host_inputs(case, seed):
    c = _grid(case)
    out = []
    for kind, f in zip("UVW", _velocity(case, seed)):
        g = _ghosted(c, kind, f)
        out.append(_pinned(g.shape).copy_(g))
    return out


def prepare(case, seed):
    if case["kind"] == "poisson":
        g = _rhs(case, seed)
        rhs, out = _pinned(g.shape).copy_(g), _pinned(g.shape)
        return {"kind": "poisson", "solver": Solver(_grid(case), case["precision"]), "rhs": rhs, "out": out}
    if case["kind"] == "group":
        members, solvers = _members(case), []
        fields = []
        sizes = {k: 0 for k in "UVWP"}
        for m, mc in enumerate(members):
            c = _grid(mc)
            s = Solver(c, "fp32")
            ins = _host_inputs(mc, 97 * seed + m)
            s.set_state(*[_fortran(t) for t in ins])
            s.compute_time_step_RK3(1)      # a group steps members that have taken their first step
            solvers.append(s)
            fields.append(ins)
            for k in "UVWP":
                sizes[k] += math.prod(c.shapes()[k])
        flat = {k: _pinned((n,)) for k, n in sizes.items()}
        outs, at = [], {k: 0 for k in "UVWP"}
        for mc in members:
            one = []
            for k in "UVWP":
                shape = _grid(mc).shapes()[k][::-1]
                n = math.prod(shape)
                one.append(flat[k][at[k]:at[k] + n].view(shape))
                at[k] += n
            outs.append(one)
        return {"kind": "group", "group": Group(solvers), "solvers": solvers, "ins": fields, "outs": outs, "flat": flat,
                "steps": case["steps"]}
    c = _grid(case)
    s = Solver(c, case["precision"], graphs=case["graphs"])
    if case["adaptive"]:
        s.set_adaptive_dt(True, cfl_target=0.4, cfl_safety=0.9, dt_min=1e-8, dt_max=1.0)
    outs = {k: _pinned(c.shapes()[k][::-1]) for k in "UVWP"}
    return {"kind": "step", "solver": s, "ins": _host_inputs(case, seed), "outs": outs, "steps": case["steps"]}


def run(state):
    if state["kind"] == "poisson":
        state["solver"].solve_poisson_equation(_fortran(state["rhs"]), out=_fortran(state["out"]))
        return {"phi": state["out"]}
    if state["kind"] == "group":
        for s, ins in zip(state["solvers"], state["ins"]):
            s.set_state(*[_fortran(t) for t in ins])
            s.compute_time_step_RK3_async(1)
        state["group"].step(state["steps"] - 1)
        for s, outs in zip(state["solvers"], state["outs"]):
            s.get_state(out=[_fortran(t) for t in outs])
        return state["flat"]
    s = state["solver"]
    s.set_state(*[_fortran(t) for t in state["ins"]])
    s.compute_time_step_RK3(state["steps"])
    s.get_state(out=[_fortran(state["outs"][k]) for k in "UVWP"])
    return state["outs"]


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "group":
        one = [work(m) for m in _members(case)]
        return {"bytes": sum(w["bytes"] for w in one), "flops": sum(w["flops"] for w in one)}
    size = 8 if case["precision"] == "fp64" else 4
    if case["kind"] == "poisson":
        c = _grid(case)
        cells = float(math.prod(c.shapes()["rhs_p"]))
        # the host array in and out, and on the device the field and its spectrum once per direction of the transform
        flops = 60.0 * cells
        if case["bc"] in ("inflow", "inflow_duct"):
            flops += 4.0 * case["nx"] * cells
        if case["bc"] in ("duct", "inflow_duct"):
            flops += 4.0 * case["nz"] * cells
        return {"bytes": cells * (16.0 + 10.0 * size), "flops": flops}
    cells = float(case["nx"]) * case["ny"] * case["nz"]
    # words per cell and step: the stages read u, the base and F1 and write u* (9 + 2 * 13 with the projections of
    # stages 1 and 2), three Poisson solves (u* in, five passes over the spectrum, phi out: 12), the last correction
    # (8), the constant-flux shift (2); LES writes and reads nu_t (15); the adaptive step reads u, v, w (3)
    words = 9 + 26 + 36 + 8 + (2 if case["flux"] else 0) + (15 if case["sgs"] else 0) + (3 if case["adaptive"] else 0)
    flops = 3 * (350.0 + 20.0 * math.log2(cells)) + (3 * 150.0 if case["sgs"] else 0) + (3 * 200.0 if case["scheme"] == 2 else 0)
    return {"bytes": cells * (case["steps"] * words * size + 7 * 8.0), "flops": cells * case["steps"] * flops}


def tolerance(case):
    # about four times what two correct forms of the same computation differ by: the FP32 stage-kernel variants among
    # each other (up to 5.5e-6 in P at 12.6 million cells, 7e-7 in a pressure solve), the FP64 step and exact() (2.3e-13 in
    # P; a pressure solve on a stretched grid up to 1e-12)
    if case["kind"] == "poisson":
        return {"rel": 2e-6, "max": 5e-5} if case["precision"] == "fp32" else {"rel": 5e-12, "max": 1e-10}
    if case["kind"] == "group" or case["precision"] == "fp32":
        return {"rel": 3e-5, "max": 5e-4}
    return {"rel": 2e-12, "max": 5e-11}


# ---- the same computations in FP64 torch ----------------------------------------------------------------------------
class _Axis:
    """Metrics of one direction at the cells p = -1 .. n (index p + 1): centre widths dc, centre spacings df across the
    upper face, and the weights w0, w1 that interpolate to it.  Entries without a face keep 1 and are never used."""

    def __init__(self, f, n, view, dev):
        m = f.size
        g = np.zeros(m + 1)
        g[1:m] = 0.5 * (f[:-1] + f[1:])
        g[0], g[m] = 2 * f[0] - g[1], 2 * f[-1] - g[m - 1]
        dc, df, w0, w1 = (np.ones(n + 2) for _ in range(4))
        for p in range(-1, n + 1):
            if p >= 0 and p + 1 < m:
                dc[p + 1] = f[p + 1] - f[p]
            if p + 2 <= m:
                df[p + 1] = g[p + 2] - g[p + 1]
                if p + 1 < m:
                    w0[p + 1] = (g[p + 2] - f[p + 1]) / df[p + 1]
                    w1[p + 1] = 1.0 - w0[p + 1]
        self.n, self.f, self.g = n, f, g
        self.arr = {k: torch.from_numpy(a).to(dev) for k, a in (("dc", dc), ("df", df), ("w0", w0), ("w1", w1))}
        self.view = view

    def __call__(self, key, shift=0):
        return self.arr[key][1 + shift:1 + shift + self.n].view(self.view)

    def wall_operator(self):
        """Rows (lower, diagonal, upper) of the second difference with Neumann ends over the cells of a wall direction."""
        f, g, n = self.f, self.g, self.f.size - 1
        up, lo = np.zeros(n), np.zeros(n)
        for r in range(n):
            h = f[r + 1] - f[r]
            if r + 1 < n:
                up[r] = 1.0 / h / (g[r + 2] - g[r + 1])
            if r > 0:
                lo[r] = 1.0 / h / (g[r + 1] - g[r])
        return lo, -(lo + up), up


def _second_difference(n, h):
    return 2.0 * (np.cos(2.0 * math.pi * np.arange(n) / n) - 1.0) / h ** 2


def _thomas(spec, lam, op, pinned):
    """The tridiagonal systems (op + lam) x = spec along dimension 1 of [z][row][x]; the first diagonal entry of the
    system at `pinned` is scaled by 3/2."""
    lo, di, up = op
    n = spec.shape[1]
    d = di[0] + lam
    if pinned is not None:
        d = d.clone()
        d[pinned] *= 1.5
    inv, b, out = [1.0 / d], [spec[:, 0]], [None] * n
    for r in range(1, n):
        m = lo[r] * inv[-1]
        inv.append(1.0 / (di[r] + lam - m * up[r - 1]))
        b.append(torch.addcmul(spec[:, r], m.to(spec.dtype), b[-1], value=-1))
    out[n - 1] = b[n - 1] * inv[n - 1]
    for r in range(n - 2, -1, -1):
        out[r] = (b[r] - up[r] * out[r + 1]) * inv[r]
    return torch.stack(out, dim=1)


class _Exact:
    """One simulation's RK3 step on the independent cells, [z][y][x], FP64."""

    def __init__(self, case, u, v, w):
        self.case, self.c = case, _grid(case)
        c, dev = self.c, u.device
        self.nz, self.ny, self.nx = u.shape
        x, y, z = grids.faces(c)
        self.Y = _Axis(y, self.ny, (1, -1, 1), dev)
        self.Z = _Axis(z, self.nz, (-1, 1, 1), dev)
        gx, gz = grids.centres(x), grids.centres(z)
        self.dx, dz = float(np.diff(gx).min()), float(np.diff(gz).min())
        self.wall = case["wall"]
        self.u, self.v, self.w = u, v, w
        self.nut = None
        self.p = None
        self.dt = c.dt
        self.filter = None
        nwl = 8 if case["wall_model"] and case["scheme"] != 1 else 0
        j = torch.arange(self.ny, device=dev)
        band = (j < nwl) | (j >= self.ny - nwl) if case["wall_model"] else torch.zeros_like(j, dtype=torch.bool)
        w_adv = 0.0 if case["scheme"] == 1 else 0.5
        self.wa_band = torch.where(band, 0.0, w_adv).to(F64).view(1, -1, 1)
        self.wa = w_adv
        kx = torch.from_numpy(_second_difference(self.nx, self.dx)[:self.nx // 2 + 1]).to(dev)
        kz = torch.from_numpy(_second_difference(self.nz, dz)).to(dev)
        self.lam = kz[:, None] + kx[None, :]
        if not self.wall:
            self.ky = torch.from_numpy(_second_difference(self.ny, y[1] - y[0])).to(dev)

    def pad(self, f, kind):
        """Rows -1 .. ny of a field."""
        if not self.wall:
            return torch.cat([f[:, -1:], f, f[:, :1]], dim=1)
        if kind in "UW":
            return torch.cat([-f[:, :1], f, -f[:, -1:]], dim=1)
        zero = torch.zeros_like(f[:, :1])
        return torch.cat([zero, f, zero], dim=1)

    def accessor(self, f, kind):
        p, seen = self.pad(f, kind), {}

        def at(di=0, dj=0, dk=0):
            if (di, dj, dk) not in seen:
                t = p[:, 1 + dj:1 + dj + self.ny]
                if di:
                    t = torch.roll(t, -di, 2)
                if dk:
                    t = torch.roll(t, -dk, 0)
                seen[di, dj, dk] = t
            return seen[di, dj, dk]
        return at

    # Reichardt's law and the Newton iteration for the friction velocity
    def friction(self, u_ref, y_ref):
        nu = self.c.nu
        c_buf = 5.2 - math.log(KAPPA) / KAPPA
        ut = torch.maximum(1e-3 * u_ref, torch.sqrt(nu * u_ref / y_ref))
        done = torch.zeros_like(ut, dtype=torch.bool)
        for _ in range(20):
            yp = ut * y_ref / nu
            e1, e2 = torch.exp(-yp / 11.0), torch.exp(-0.33 * yp)
            up = torch.log(1.0 + KAPPA * yp) / KAPPA + c_buf * (1.0 - e1 - yp / 11.0 * e2)
            dup = 1.0 / (1.0 + KAPPA * yp) + c_buf * (e1 / 11.0 - e2 / 11.0 + yp * 0.33 / 11.0 * e2)
            f = u_ref / ut.clamp(min=1e-20) - up
            fp = -u_ref / (ut * ut).clamp(min=1e-20) - dup * y_ref / nu
            new = ut - f / (fp + torch.copysign(torch.full_like(fp, 1e-14), fp))
            new = torch.minimum(torch.maximum(new, 0.1 * ut), 10.0 * ut)
            stop = (new - ut).abs() < 1e-6 * new
            ut = torch.where(done, ut, new)
            done = done | stop
        return ut

    def wall_distance(self, row):
        return float(self.Y.g[1] if row == 0 else self.Y.f[-1] - self.Y.f[0] - self.Y.g[-2])

    def eddy_viscosity(self):
        if not self.case["sgs"]:
            return None
        U, V, W = (self.accessor(f, k) for f, k in zip((self.u, self.v, self.w), "UVW"))
        Y, Z, dx = self.Y, self.Z, self.dx
        half = lambda g, lo, hi: 0.5 * ((g[1] - g[0]) / lo + (g[2] - g[1]) / hi)
        ylo, yhi, zlo, zhi = Y("df", -1), Y("df"), Z("df", -1), Z("df")
        a11 = (U() - U(-1)) / dx
        a21 = half((U(0, -1), U(), U(0, 1)), ylo, yhi)
        a31 = half((U(0, 0, -1), U(), U(0, 0, 1)), zlo, zhi)
        a12 = 0.5 * (V(1) - V(-1)) / dx
        a22 = (V() - V(0, -1)) / Y("dc")
        a32 = half((V(0, 0, -1), V(), V(0, 0, 1)), zlo, zhi)
        a13 = 0.5 * (W(1) - W(-1)) / dx
        a23 = half((W(0, -1), W(), W(0, 1)), ylo, yhi)
        a33 = (W() - W(0, 0, -1)) / Z("dc")
        if self.case["wall_model"]:
            for row, sg in ((0, 1.0), (self.ny - 1, -1.0)):
                yw = self.wall_distance(row)
                uc, wc = 0.5 * (U() + U(-1))[:, row], 0.5 * (W() + W(0, 0, -1))[:, row]
                mag = torch.sqrt(uc * uc + wc * wc)
                fac = sg * self.friction(mag, max(yw, 1e-14)) / (KAPPA * yw * mag)
                on = mag > 1e-14
                a21[:, row] = torch.where(on, fac * uc, a21[:, row])
                a23[:, row] = torch.where(on, fac * wc, a23[:, row])
        sx, sy, sz = dx * dx, Y("dc") ** 2, Z("dc") ** 2
        row1, row2, row3 = (a11, a12, a13), (a21, a22, a23), (a31, a32, a33)
        b = lambda m, n: sx * (row1[m] * row1[n]) + sy * (row2[m] * row2[n]) + sz * (row3[m] * row3[n])
        b11, b22, b33, b12, b13, b23 = b(0, 0), b(1, 1), b(2, 2), b(0, 1), b(0, 2), b(1, 2)
        sq = sum(g * g for r in (row1, row2, row3) for g in r)
        zero = torch.zeros_like(sq)
        if self.case["sgs"] == 2:
            num = -(b11 * a11 + b22 * a22 + b33 * a33 + b12 * (a12 + a21) + b13 * (a13 + a31) + b23 * (a23 + a32))
            on = (sq > 1e-20) & (num > 1e-12 * (sx + sy + sz) * sq * torch.sqrt(sq))
            return torch.where(on, self.c.C_amd * num / sq, zero)
        beta = b11 * b22 - b12 * b12 + b11 * b33 - b13 * b13 + b22 * b33 - b23 * b23
        on = (sq > 1e-20) & (beta > 0)
        return torch.where(on, 2.5 * self.c.Cs_vreman ** 2 * torch.sqrt((beta / sq).clamp(min=0)), zero)

    def wall_stress(self):
        """The filtered wall model's stresses (tau_x at U faces, tau_z at W faces) of both walls, lower then upper."""
        if not self.case["wall_model"]:
            return None
        first = self.filter is None
        state, taus = self.filter or {}, []
        for row, sg in ((0, 1.0), (self.ny - 1, -1.0)):
            ym = max(self.wall_distance(row), 1e-14)
            u, w = self.u[:, row], self.w[:, row]
            at_u = (u, 0.5 * (torch.roll(w, 1, 0) + w))
            at_w = (0.5 * (torch.roll(u, 1, 1) + u), w)
            for which, now in (("x", at_u), ("z", at_w)):
                if first:
                    uf, wf = now
                else:
                    uf, wf, ut = state[row, which]
                    eps = torch.where(ut > 0, (self.dt * KAPPA * ut / ym).clamp(max=1.0), 1.0)
                    uf, wf = (1 - eps) * uf + eps * now[0], (1 - eps) * wf + eps * now[1]
                mag = torch.sqrt(uf * uf + wf * wf)
                ut = self.friction(mag, ym)
                state[row, which] = (uf, wf, ut)
                taus.append(sg * ut * ut * (uf if which == "x" else wf) / mag.clamp(min=1e-30))
        self.filter = state
        return {"x": (taus[0], taus[2]), "z": (taus[1], taus[3])}

    def rhs(self, tau):
        Y, Z, dx, nu = self.Y, self.Z, self.dx, self.c.nu
        U, V, W = (self.accessor(f, k) for f, k in zip((self.u, self.v, self.w), "UVW"))
        N = self.accessor(self.nut, "N") if self.nut is not None else None
        yi = lambda f, di=0, dk=0, s=0: Y("w0", s) * f(di, s, dk) + Y("w1", s) * f(di, s + 1, dk)   # to the y face j+s
        zi = lambda f, di=0, dj=0, s=0: Z("w0", s) * f(di, dj, s) + Z("w1", s) * f(di, dj, s + 1)   # to the z face k+s
        yi2 = lambda f, s, t: Y("w0", s) * f(0, s, t) + Y("w1", s) * f(0, s + 1, t)
        zs = lambda a, b, s=0: Z("w0", s) * a + Z("w1", s) * b

        def blend(wa, f1, f0, q, g1, g0):
            return (1.0 - wa) * (f1 - f0) + wa * q * (g1 - g0)
        first, last = (slice(None), 0), (slice(None), self.ny - 1)
        wm = tau is not None
        # u
        wa = self.wa_band
        t1, t0 = 0.5 * (U() + U(1)), 0.5 * (U(-1) + U())
        r = -blend(wa, t1 * t1, t0 * t0, U(), t1, t0) / dx
        u1, u0 = yi(U), yi(U, s=-1)
        v1, v0 = 0.5 * (V() + V(1)), 0.5 * (V(0, -1) + V(1, -1))
        r -= blend(wa, u1 * v1, u0 * v0, 0.5 * (v0 + v1), u1, u0) / Y("dc")
        u1, u0 = zi(U), zi(U, s=-1)
        w1, w0 = 0.5 * (W() + W(1)), 0.5 * (W(0, 0, -1) + W(1, 0, -1))
        r -= blend(wa, u1 * w1, u0 * w0, 0.5 * (w0 + w1), u1, u0) / Z("dc")
        nx1 = nx2 = ny1 = ny2 = nz1 = nz2 = nu
        if N:
            nx1, nx2 = nu + N(), nu + N(1)
            ny1, ny2 = nu + 0.5 * (yi(N, s=-1) + yi(N, 1, s=-1)), nu + 0.5 * (yi(N) + yi(N, 1))
            if self.wall:
                ny1[first], ny2[last] = nu, nu
            nz1, nz2 = nu + 0.5 * (zi(N, s=-1) + zi(N, 1, s=-1)), nu + 0.5 * (zi(N) + zi(N, 1))
        fy2 = ny2 * ((U(0, 1) - U()) / Y("df") + (V(1) - V()) / dx)
        fy1 = ny1 * ((U() - U(0, -1)) / Y("df", -1) + (V(1, -1) - V(0, -1)) / dx)
        if wm:
            fy1[first], fy2[last] = tau["x"][0], tau["x"][1]
        fz2 = nz2 * ((U(0, 0, 1) - U()) / Z("df") + (W(1) - W()) / dx)
        fz1 = nz1 * ((U() - U(0, 0, -1)) / Z("df", -1) + (W(1, 0, -1) - W(0, 0, -1)) / dx)
        r += 2.0 / dx ** 2 * (nx2 * (U(1) - U()) - nx1 * (U() - U(-1))) + (fy2 - fy1) / Y("dc") + (fz2 - fz1) / Z("dc")
        r += 0.0 if self.case["flux"] else self.c.dPdx
        ru = r
        # v
        wa = self.wa
        t1, t0 = 0.5 * (V() + V(0, 1)), 0.5 * (V(0, -1) + V())
        r = -blend(wa, t1 * t1, t0 * t0, V(), t1, t0) / Y("df")
        u1, u0 = yi(U), yi(U, -1)
        v1, v0 = 0.5 * (V() + V(1)), 0.5 * (V(-1) + V())
        r -= blend(wa, u1 * v1, u0 * v0, 0.5 * (u0 + u1), v1, v0) / dx
        v1, v0 = zi(V), zi(V, s=-1)
        w1, w0 = yi(W), yi2(W, 0, -1)
        r -= blend(wa, v1 * w1, v0 * w0, 0.5 * (w0 + w1), v1, v0) / Z("dc")
        if N:
            nx1, nx2 = nu + 0.5 * (yi(N, -1) + yi(N)), nu + 0.5 * (yi(N) + yi(N, 1))
            ny1, ny2 = nu + N(), nu + N(0, 1)
            nz1, nz2 = nu + zs(yi2(N, 0, -1), yi(N), -1), nu + zs(yi(N), yi2(N, 0, 1))
        fx2 = nx2 * ((V(1) - V()) / dx + (U(0, 1) - U()) / Y("df"))
        fx1 = nx1 * ((V() - V(-1)) / dx + (U(-1, 1) - U(-1)) / Y("df"))
        fz2 = nz2 * ((V(0, 0, 1) - V()) / Z("df") + (W(0, 1) - W()) / Y("df"))
        fz1 = nz1 * ((V() - V(0, 0, -1)) / Z("df", -1) + (W(0, 1, -1) - W(0, 0, -1)) / Y("df"))
        r += (fx2 - fx1) / dx + (fz2 - fz1) / Z("dc")
        r += 2.0 / Y("df") * (ny2 * (V(0, 1) - V()) / Y("dc", 1) - ny1 * (V() - V(0, -1)) / Y("dc"))
        if self.wall:
            r[last] = 0.0
        rv = r
        # w
        wa = self.wa_band
        t1, t0 = 0.5 * (W() + W(0, 0, 1)), 0.5 * (W(0, 0, -1) + W())
        r = -blend(wa, t1 * t1, t0 * t0, W(), t1, t0) / Z("df")
        u1, u0 = zi(U), zi(U, -1)
        w1, w0 = 0.5 * (W() + W(1)), 0.5 * (W(-1) + W())
        r -= blend(wa, u1 * w1, u0 * w0, 0.5 * (u0 + u1), w1, w0) / dx
        v1, v0 = zi(V), zi(V, 0, -1)
        w1, w0 = yi(W), yi(W, s=-1)
        r -= blend(wa, v1 * w1, v0 * w0, 0.5 * (v0 + v1), w1, w0) / Y("dc")
        if N:
            nx1, nx2 = nu + 0.5 * (zi(N) + zi(N, -1)), nu + 0.5 * (zi(N) + zi(N, 1))
            ny1, ny2 = nu + zs(yi(N, s=-1), yi2(N, -1, 1)), nu + zs(yi(N), yi2(N, 0, 1))
            if self.wall:
                ny1[first], ny2[last] = nu, nu
            nz1, nz2 = nu + N(), nu + N(0, 0, 1)
        fy2 = ny2 * ((W(0, 1) - W()) / Y("df") + (V(0, 0, 1) - V()) / Z("df"))
        fy1 = ny1 * ((W() - W(0, -1)) / Y("df", -1) + (V(0, -1, 1) - V(0, -1)) / Z("df"))
        if wm:
            fy1[first], fy2[last] = tau["z"][0], tau["z"][1]
        fx2 = nx2 * ((W(1) - W()) / dx + (U(0, 0, 1) - U()) / Z("df"))
        fx1 = nx1 * ((W() - W(-1)) / dx + (U(-1, 0, 1) - U(-1)) / Z("df"))
        r += (fx2 - fx1) / dx + (fy2 - fy1) / Y("dc")
        r += 2.0 / Z("df") * (nz2 * (W(0, 0, 1) - W()) / Z("dc", 1) - nz1 * (W() - W(0, 0, -1)) / Z("dc"))
        rw = r
        if self.case["scheme"] == 2:
            du, dv, dw = (self.dissipation(i) for i in range(3))
            ru, rw = ru + du, rw + dw
            rv = rv + dv
            if self.wall:
                rv[last] = 0.0
        return ru, rv, rw

    def dissipation(self, comp):
        """beta |u_c| D through every face of component comp, D the third or fifth difference of the component."""
        order, beta = self.case["order"], self.c.adv_beta0
        weights = {5: np.array([1.0, -5, 10, -10, 5, -1]) / 60, 3: np.array([0.0, -1, 3, -3, 1, 0]) / 12, 0: np.zeros(6)}
        F = (self.u, self.v, self.w)[comp]
        dim = (2, 1, 0)[comp]
        ny = self.ny
        # rows of the fields that the scheme reads, its index 1 being row -1
        extra = lambda f, kind: self.pad(f, kind)[:, :ny + 1] if kind == "V" and self.wall else \
            torch.cat([self.pad(f, kind)] + ([] if self.wall else [f[:, 1:2]]), dim=1)
        rows = extra(F, "UVW"[comp])
        if comp == 1 and not self.wall:
            rows = rows[:, :ny + 2]
        n = rows.shape[1]
        up = lambda f: torch.roll(f, -1, dim)                  # the neighbour on the component's own axis
        Y, Z = self.Y, self.Z
        r = 0.0
        for axis, vel, h in ((2, self.u, self.dx), (0, self.w, Z("df") if comp == 2 else Z("dc"))):
            if comp == 1:
                p = self.pad(vel, "U")
                uc = 0.5 * (p[:, 1:ny + 1] + p[:, 2:ny + 2])
            else:
                uc = 0.5 * (vel + up(vel))
            d = sum(float(weights[order][q]) * torch.roll(F, 2 - q, axis) for q in range(6) if weights[order][q])
            flux = beta * uc.abs() * d
            r = r - (flux - torch.roll(flux, 1, axis)) / h
        # y: faces between rows m and m+1 (1-based), m = 1 .. ny + 1 at most
        vrows = extra(self.v, "V")
        faces = []
        for m in range(1, ny + 2):
            if m + 1 > n:
                break
            o = 5 if order == 5 and m - 2 >= 1 and m + 3 <= n else (3 if m - 1 >= 1 and m + 2 <= n else 0)
            idx = [max(m - 2, 1), max(m - 1, 1), m, m + 1, min(m + 2, n), min(m + 3, n)]
            d = sum(float(weights[o][q]) * rows[:, idx[q] - 1] for q in range(6)) if o else torch.zeros_like(rows[:, 0])
            if comp == 1:
                uc = 0.5 * (vrows[:, m - 1] + vrows[:, m])
            elif comp == 0:
                uc = 0.5 * (vrows[:, m - 1] + torch.roll(vrows[:, m - 1], -1, 1))
            else:
                uc = 0.5 * (vrows[:, m - 1] + torch.roll(vrows[:, m - 1], -1, 0))
            faces.append(beta * uc.abs() * d)
        while len(faces) < ny + 1:
            faces.append(torch.zeros_like(faces[0]))
        f = torch.stack(faces, dim=1)
        return r - (f[:, 1:] - f[:, :-1]) / (Y("df") if comp == 1 else Y("dc"))

    def pressure(self, u, v, w):
        vm = self.pad(v, "V")[:, :self.ny]
        div = (u - torch.roll(u, 1, 2)) / self.dx + (v - vm) / self.Y("dc") + (w - torch.roll(w, 1, 0)) / self.Z("dc")
        if self.wall:
            spec = torch.fft.rfftn(div, dim=(0, 2))
            spec = _thomas(spec, self.lam, self.Y.wall_operator(), (0, 0))
            return torch.fft.irfftn(spec, s=(self.nz, self.nx), dim=(0, 2))
        spec = torch.fft.rfftn(div)
        k = self.lam[:, None, :] + self.ky[None, :, None]
        k[0, 0, 0] = 1.0
        spec = spec / k
        spec[0, 0, 0] = 0.0
        return torch.fft.irfftn(spec, s=(self.nz, self.ny, self.nx))

    def select_dt(self):
        U, V, W = (self.accessor(f, k) for f, k in zip((self.u, self.v, self.w), "UVW"))
        Y, Z, dx = self.Y, self.Z, self.dx
        conv = (0.5 * (U() + U(-1)).abs() / dx + 0.5 * (V() + V(0, -1)).abs() / Y("dc") +
                0.5 * (W() + W(0, 0, -1)).abs() / Z("dc")).max()
        nu = self.c.nu + (self.nut if self.nut is not None else 0.0 * self.u)
        visc = (nu * 2.0 * (dx ** -2 + Y("dc") ** -2 + Z("dc") ** -2)).max()
        self.dt = float(min(max(0.4 / float(torch.maximum(conv, visc)) * 0.9, 1e-8), 1.0))

    def step(self):
        base = (self.u, self.v, self.w)
        f1 = None
        for s in (1, 2, 3):
            self.nut = self.eddy_viscosity()
            if s == 1:
                if self.case["adaptive"]:
                    self.select_dt()
                tau = self.wall_stress()
            f = self.rhs(tau)
            dt = self.dt
            if s == 1:
                f1 = f
                star = [b + dt * (8.0 / 15.0) * r for b, r in zip(base, f)]
            else:
                c2 = 5.0 / 12.0 if s == 2 else 0.75
                star = [b + dt * (0.25 * a + c2 * r) for b, a, r in zip(base, f1, f)]
            phi = self.pressure(*star)
            self.u = star[0] - (torch.roll(phi, -1, 2) - phi) / self.dx
            self.w = star[2] - (torch.roll(phi, -1, 0) - phi) / self.Z("df")
            up = torch.cat([phi[:, 1:], phi[:, :1]], dim=1)
            self.v = star[1] - (up - phi) / self.Y("df")
            if self.wall:
                self.v[:, self.ny - 1] = 0.0
        self.p = phi / (dt * 0.75)
        if self.case["flux"]:
            wgt = self.Y("dc") * self.Z("dc")
            mean = (self.u * wgt).sum() / (wgt.sum() * self.nx)
            self.u = self.u + (self.c.Ub_target - mean)

    def outputs(self):
        return {k: _ghosted(self.c, k, f) for k, f in zip("UVWP", (self.u, self.v, self.w, self.p))}


def _exact_step(case, seed):
    e = _Exact(case, *_velocity(case, seed))
    for _ in range(case["steps"]):
        e.step()
    return e.outputs()


def _exact_poisson(case, seed):
    c, g = _grid(case), _rhs(case, seed)
    bc, dev = case["bc"], g.device
    out = g.clone()
    xwall, zwall = bc in ("inflow", "inflow_duct"), bc in ("duct", "inflow_duct", "spanwise")
    yper = bc in ("spanwise", "periodic")
    x, y, z = grids.faces(c)
    dx, dz = (float(np.diff(grids.centres(f)).min()) for f in (x, z))
    n = (c.nz - (1 if zwall else 2), c.ny - (2 if yper else 1), c.nx - (1 if xwall else 2))
    nz, ny, nx = n
    b = g[:nz, :ny, :nx]
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    if xwall:
        i = np.arange(nx)
        dct = to(2.0 * np.cos(math.pi * (((2 * i[:, None] + 1) * (2 * i[None, :] + 1)) % (8 * nx)) / (4.0 * nx)))
        kx = to(2.0 * (np.cos(math.pi * (2 * i + 1) / (2.0 * nx)) - 1.0) / dx ** 2)
        spec, inv_x = (b @ dct).to(torch.complex128), lambda s: (s.real @ dct) / (2.0 * nx)
    else:
        kx = to(_second_difference(nx, dx)[:nx // 2 + 1])
        spec, inv_x = torch.fft.rfft(b, dim=2), lambda s: torch.fft.irfft(s, n=nx, dim=2)
    ax = lambda f, m: _Axis(f, m, (-1,), dev)
    if bc in ("duct", "inflow_duct"):
        lo, di, up = ax(z, nz).wall_operator()
        w = z[1:] - z[:-1]
        off = up[:-1] * np.sqrt(w[:-1] / w[1:])
        lz, q = np.linalg.eigh(np.diag(di) + np.diag(off, 1) + np.diag(off, -1))
        fwd, inv = to((q * np.sqrt(w)[:, None]).T).to(torch.complex128), to(q / np.sqrt(w)[:, None]).to(torch.complex128)
        spec = torch.einsum("mk,kji->mji", fwd, spec)
        null = None if xwall else (int(np.abs(lz).argmin()), 0)
        spec = _thomas(spec, to(lz)[:, None] + kx[None, :], ax(y, ny).wall_operator(), null)
        phi = inv_x(torch.einsum("km,mji->kji", inv, spec))
    elif bc == "spanwise":
        ky = to(_second_difference(ny, y[1] - y[0]))
        spec = torch.fft.fft(spec, dim=1).transpose(0, 1)        # [ky][z][kx]
        spec = _thomas(spec, ky[:, None] + kx[None, :], ax(z, nz).wall_operator(), (0, 0))
        phi = inv_x(torch.fft.ifft(spec.transpose(0, 1), dim=1))
    else:
        kz = to(_second_difference(nz, dz))
        spec = torch.fft.fft(spec, dim=0)
        if bc == "periodic":
            ky = to(_second_difference(ny, y[1] - y[0]))
            k = kz[:, None, None] + ky[None, :, None] + kx[None, None, :]
            k[0, 0, 0] = 1.0
            spec = torch.fft.fft(spec, dim=1) / k
            spec[0, 0, 0] = 0.0
            spec = torch.fft.ifft(spec, dim=1)
        else:
            spec = _thomas(spec, kz[:, None] + kx[None, :], ax(y, ny).wall_operator(), None if xwall else (0, 0))
        phi = inv_x(torch.fft.ifft(spec, dim=0))
    # the planes beyond the cells: periodic copies, or the input where the library leaves it
    out[:nz, :ny, :nx] = phi
    if bc in ("channel", "periodic"):
        k, j, i = (torch.arange(m, device=dev) % p for m, p in zip(g.shape, n))
        return {"phi": phi[k][:, j][:, :, i]}
    if yper:
        out[:, ny] = out[:, 0]
    if not xwall:
        keep = nz if zwall else g.shape[0]
        out[:, :, nx] = out[:, :, 0]
        out[:keep, :, nx + 1] = out[:keep, :, 1]
        if bc == "spanwise":
            out[nz:, :, nx + 1] = g[nz:, :, nx + 1]
            out[nz:, ny] = out[nz:, 0]
    if not zwall:
        out[nz] = torch.cat([phi[0], g[nz, :, nx:]], dim=1)      # the inflow grid, the only one left here
    return {"phi": out}


def exact(case, seed):
    if case["kind"] == "poisson":
        return _exact_poisson(case, seed)
    if case["kind"] == "group":
        got = [_exact_step(m, 97 * seed + i) for i, m in enumerate(_members(case))]
        return {k: torch.cat([g[k].reshape(-1) for g in got]) for k in "UVWP"}
    return _exact_step(case, seed)
