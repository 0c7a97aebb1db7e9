"""Timed cases of the framework's main paths, through its public entry points.

A case is a dict of plain values; `kind` says which path it takes:

  rhs     one PETSc residual callback on a device vector: FRSolver.rhs_func, or
          fun_implicit with form = "ifunction";
  f32     FRSolver.residual_kernel_f32, the single-precision residual;
  step    one explicit time step in place, Integrator.step, with its stabilisation;
  run1d   a 1D shock-tube run, Integrator.run replaying CUDA graphs;
  jvp     one complex-step Jacobian-vector product, FRSolver.matmult;
  blocks  the Jacobian's element blocks, FRSolver.jac_blocks or jac_blocks5;
  newton  the linear solve of one Newton step: pre_jv_eval, pc_setup_gs and
          fr_sdg_b200.implicit.gmres over matmult and pc_apply;
  batch   a few steps of many independent uneven instances, DeviceBatch.run.

States are the workloads' own flows (fr_sdg_b200/workloads.py) with seeded smooth and
nodal perturbations, so that every branch of the fluxes and limiters is met the way a
run in progress meets it.  `exact` restates the paths in plain torch FP64.
"""
import math

import numpy as np
import torch

from fr_sdg_b200 import FRSolver
from fr_sdg_b200 import _abi as A
from fr_sdg_b200.batch import DeviceBatch
from fr_sdg_b200.implicit import gmres
from fr_sdg_b200.integrate import Integrator
from fr_sdg_b200.workloads import make_config

VDW = (0.05, 0.02)
GAMMA = 1.4
RESTART = 30         # Arnoldi steps of one GMRES cycle
BATCH_STEPS = 4      # steps of one batch call
P_TOTAL = 1.0        # inflow total pressure and temperature of the bump channel (R = 1)
MACH = 0.5


# ---------------------------------------------------------------- the cases
def listed():
    blast = dict(flow="blast", geom="cart", bc="outflow", gas="vdw", riemann="hllc")
    bump = dict(flow="bump", geom="bump", bc="bump", gas="ideal", riemann="hllc", p=3, nx=256, ny=64)
    return [
        # the smallest problem: the 1D Sod tube of 200 elements, bound by launches
        dict(name="sod_run", kind="run1d", nx=200, p=3, steps=256),
        # an accuracy run's right-hand side: 64 x 64 warped vortex, 3 MB, bound by latency
        dict(name="rhs_vortex_64_p4", kind="rhs", form="rhs", flow="vortex", geom="warp", bc="periodic", gas="ideal",
             riemann="hllc", p=4, nx=64, ny=64),
        # an ordinary mesh with ragged sizes, the reference's default order and flux
        dict(name="rhs_ragged_p3", kind="rhs", form="rhs", flow="blast", geom="cart", bc="walls", gas="ideal",
             riemann="rusanov", p=3, nx=211, ny=173),
        # the headline: the residual of the large 2D blast
        dict(name="rhs_blast_1024_p5", kind="rhs", form="rhs", p=5, nx=1024, ny=1024, **blast),
        # high order, odd sizes, periodic
        dict(name="rhs_high_p7", kind="rhs", form="rhs", flow="blast", geom="cart", bc="periodic", gas="ideal",
             riemann="hllc", p=7, nx=190, ny=131),
        # a time step of the blast as configured: SSP-RK3, spectral filter, positivity limiter
        dict(name="step_blast_512_p5", kind="step", scheme="ssprk3", stab="filter", p=5, nx=512, ny=512, **blast),
        # a shock run with the WENO limiter and its sensor, as the reference's tools set it
        dict(name="step_weno_p3", kind="step", scheme="ssprk3", stab="weno", flow="blast", geom="cart", bc="outflow",
             gas="ideal", riemann="hllc", p=3, nx=300, ny=200),
        # the single-precision residual of the mixed form
        dict(name="f32_blast_512_p5", kind="f32", p=5, nx=512, ny=512, **blast),
        # the implicit path on the bump channel: Jacobian product, Jacobian blocks, Newton's linear solve
        dict(name="jvp_bump", kind="jvp", **bump),
        dict(name="blocks_bump", kind="blocks", slots=5, **bump),
        dict(name="newton_bump", kind="newton", **bump),
        # many uneven small problems advanced together
        dict(name="batch_24", kind="batch", count=24, mesh_seed=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "rhs", "step", "step", "run1d", "f32", "jvp", "blocks", "newton", "batch"])
    if kind == "run1d":
        return dict(kind=kind, nx=_log(rng, 40, 3000), p=rng.randint(2, 6), steps=rng.choice([128, 192, 256]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 24), mesh_seed=rng.randint(2, 10 ** 6))
    if kind in ("jvp", "blocks", "newton"):
        p = rng.randint(1, 4)
        nd = 4 * (p + 1) ** 2
        # at most the listed case's block storage
        top = int(min(256 * 64, 256 * 64 * 64 * 64 / nd ** 2))
        nx = _log(rng, 12, 256)
        c = dict(kind=kind, flow="bump", geom="bump", bc="bump", gas="ideal", riemann=rng.choice(["hllc", "rusanov"]),
                 p=p, nx=nx, ny=max(4, min(_log(rng, 6, 130), top // nx)))
        if kind == "blocks":
            c["slots"] = rng.choice([1, 5])
        return c
    p = rng.randint(1, 8) if kind == "rhs" else rng.randint(2, 6)
    most = 1024 * 1024 * 36 if kind == "rhs" else 512 * 512 * 36   # nodes of the listed cases
    side = int(math.sqrt(most * (0.5 if p > 5 else 0.9))) // (p + 1)
    c = dict(kind=kind, p=p, nx=_log(rng, 16, side), ny=_log(rng, 16, side), riemann=rng.choice(["hllc", "rusanov"]))
    flow = rng.choice(["blast", "blast", "vortex"]) if kind != "f32" else "blast"
    if flow == "vortex":
        c.update(flow=flow, geom="warp", bc="periodic", gas="ideal")
        c["nx"], c["ny"] = min(c["nx"], 256), min(c["ny"], 256)
    else:
        c.update(flow=flow, geom="cart", bc=rng.choice(["outflow", "walls", "periodic"]), gas=rng.choice(["ideal", "vdw"]))
    if kind == "rhs":
        c["form"] = rng.choice(["rhs", "rhs", "ifunction"])
    if kind == "step":
        c["scheme"] = rng.choice(["ssprk3", "ssprk3", "rk4"])
        c["stab"] = rng.choice(["none", "none"] if flow == "vortex" else ["filter", "filter", "weno"])
    return c


# ---------------------------------------------------------------- configurations and states
def _config(c):
    box = dict(blast=(1.0, 1.0), vortex=(10.0, 10.0), bump=(3.0, 0.8))[c["flow"]]
    kw = dict(dim=2, p=c["p"], n_elems=(c["nx"], c["ny"]), box=box, riemann=c["riemann"], gas=c["gas"], gamma=GAMMA, vdw=VDW)
    faces = (A.LEFT, A.RIGHT, A.TOP, A.BOTTOM)
    if c["bc"] == "bump":
        kw["bcs"] = {A.LEFT: (A.BC_SUBSONIC_INFLOW, None, (P_TOTAL, 1.0, 1.0, 0.0)),
                     A.RIGHT: (A.BC_PRESSURE_OUTLET, None, (_p_out(),)), A.BOTTOM: A.BC_SLIP_WALL, A.TOP: A.BC_SLIP_WALL}
        kw.update(geometry=A.GEOM_WALL_PROFILE, profile=A.PROFILE_GAUSS_BUMP, geom_params=(-1.5, 0.0625, 25.0, 0.0), csd_eps=1e-30)
    else:
        kind = {"outflow": A.BC_OUTFLOW, "walls": A.BC_WALL, "periodic": A.BC_PERIODIC}[c["bc"]]
        kw["bcs"] = {f: kind for f in faces}
    if c["geom"] == "warp":
        kw.update(geometry=A.GEOM_SINE_WARP, geom_params=(0.1, 0.0, 0.0, 0.0))
    stab = c.get("stab", "none")
    if stab == "filter":
        kw.update(apply_filter=True, cut_off=min(2, c["p"] - 1), pp_limit=True)
    elif stab == "weno":
        kw.update(apply_weno=True, weno_gamma=0.998, threshold=0.8, theta=1.0, pp_limit=True)
    cfg = make_config(**kw)
    if c["bc"] == "bump":
        cfg.jvp_exact_bc = 1  # as the bump workload sets it
    return cfg


def _p_out():
    return P_TOTAL * (1.0 + 0.5 * (GAMMA - 1.0) * MACH * MACH) ** (-GAMMA / (GAMMA - 1.0))


def _gen(dev, seed):
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    return g


def _noise(shape, dev, gen):
    return 2.0 * torch.rand(shape, generator=gen, device=dev, dtype=torch.float64) - 1.0


def _energy(gas, rho, v2, p):
    if gas == "ideal":
        return p / (GAMMA - 1.0) + 0.5 * rho * v2
    a, b = VDW
    return (p + a * rho * rho) * (1.0 - b * rho) / (GAMMA - 1.0) - a * rho * rho + 0.5 * rho * v2


def _state(c, seed, dev):
    """(ny, nx, n, n, 4) conservative state: the case's flow, a seeded smooth modulation
    and nodal noise."""
    m = _Mesh(c, dev)
    x, y = m.x, m.y
    gen, r = _gen(dev, seed), np.random.RandomState(int(seed) % (2 ** 31))
    noise = _noise((4,) + tuple(x.shape), dev, gen)
    ph = r.uniform(0.0, 2.0 * math.pi, 4)
    wave = [torch.sin(2.0 * math.pi * (x / m.lx + y / m.ly) + float(q)) for q in ph]
    if c["flow"] == "blast":
        rad = torch.sqrt((x - 0.5 - 0.02 * float(r.uniform(-1, 1))) ** 2 + (y - 0.5) ** 2)
        inside = rad < 0.4 + 0.02 * float(r.uniform(-1, 1))
        rho, p = torch.where(inside, 1.0, 0.125).double(), torch.where(inside, 1.0, 0.1).double()
        u, v, amp = 0.3 * wave[0], 0.3 * wave[1], 0.01
    elif c["flow"] == "vortex":
        beta = 5.0 * float(r.uniform(0.8, 1.0))
        dx, dy = x - 5.0, y - 5.0
        ef = torch.exp(1.0 - dx * dx - dy * dy)
        rho = (1.0 - beta * beta * (GAMMA - 1.0) * ef * ef / (16.0 * GAMMA * math.pi ** 2)) ** (1.0 / (GAMMA - 1.0))
        u, v = 1.0 - beta * ef * dy / (2.0 * math.pi), 1.0 + beta * ef * dx / (2.0 * math.pi)
        p, amp = rho ** GAMMA, 1e-4
    else:
        fac = 1.0 + 0.5 * (GAMMA - 1.0) * MACH * MACH
        rho, p = torch.full_like(x, _p_out() * fac), torch.full_like(x, _p_out())
        u, v = MACH * torch.sqrt(GAMMA * p / rho) * (1.0 + 0.05 * wave[0]), 0.02 * wave[1]
        amp = 1e-3
    rho = rho * (1.0 + 0.02 * wave[2] + amp * noise[0])
    p = p * (1.0 + 0.02 * wave[3] + amp * noise[1])
    u, v = u + amp * noise[2], v + amp * noise[3]
    return torch.stack([rho, rho * u, rho * v, _energy(c["gas"], rho, u * u + v * v, p)], dim=-1).contiguous()


def _dt(c):
    """CFL 0.05 with the (2p + 1) rule on the case's fixed wave-speed bound."""
    lx, ly = dict(blast=(1.0, 1.0), vortex=(10.0, 10.0), bump=(3.0, 0.8))[c["flow"]]
    return 0.05 * min(lx / c["nx"], ly / c["ny"]) / ((2 * c["p"] + 1) * 3.0)


def _sigma(c):
    """1 / dt of the implicit cases: a few explicit time steps of the mesh."""
    return 0.2 * (c["nx"] / 3.0 + c["ny"] / 0.8) * (c["p"] + 1)


def _cfg1d(c):
    return make_config(dim=1, p=c["p"], n_elems=(c["nx"], 1), box=(1.0, 1.0), riemann="rusanov",
                       bcs={A.LEFT: A.BC_OUTFLOW, A.RIGHT: A.BC_OUTFLOW}, apply_filter=True,
                       cut_off=min(2, c["p"] - 1), pp_limit=True)


def _state1d(c, seed):
    """(nx, 3, n) Sod states, the jump and the levels varied by the seed."""
    r = np.random.RandomState(int(seed) % (2 ** 31))
    xi = _gll(c["p"])[0]
    x = (np.arange(c["nx"])[:, None] + 0.5 * (1.0 + xi[None, :])) / c["nx"]
    left = x < 0.5 + 0.05 * r.uniform(-1, 1)
    rho = np.where(left, 1.0, 0.125) * (1.0 + 0.01 * r.uniform(-1, 1, x.shape))
    p = np.where(left, 1.0, 0.1) * (1.0 + 0.01 * r.uniform(-1, 1, x.shape))
    u = 0.05 * np.sin(2.0 * math.pi * x)
    return np.stack([rho, rho * u, p / (GAMMA - 1.0) + 0.5 * rho * u * u], axis=1)


def _dt1d(c):
    return 0.1 / c["nx"] / ((2 * c["p"] + 1) * 1.3)


def _members(c):
    """The instances of a batch: circular explosions of uneven meshes, orders and gases."""
    r = np.random.RandomState(c["mesh_seed"])
    out = []
    for _ in range(c["count"]):
        ne, p, gas = int(r.choice([32, 48, 64, 96])), int(r.randint(2, 7)), str(r.choice(["ideal", "vdw"]))
        out.append(dict(kind="step", scheme="ssprk3", stab="filter", flow="blast", geom="cart", bc="outflow", gas=gas,
                        riemann="rusanov", p=p, nx=ne, ny=ne))
    return out


# ---------------------------------------------------------------- prepare and run
def prepare(case, seed):
    c, dev, kind = dict(case), torch.device("cuda"), case["kind"]
    s = dict(kind=kind, case=c)
    if kind == "run1d":
        s["solver"] = FRSolver(_cfg1d(c))
        s["U0"] = torch.from_numpy(_state1d(c, seed).reshape(-1)).to(dev)
        s["U"] = torch.empty_like(s["U0"])
        s["it"], s["dt"] = Integrator(s["solver"], "ssprk3"), _dt1d(c)
        return s
    if kind == "batch":
        members = _members(c)
        s["U0"] = torch.cat([_state(m, seed + 101 * k, dev).reshape(-1) for k, m in enumerate(members)])
        s["U"] = s["U0"].clone()
        items, at = [], 0
        for m in members:
            f = FRSolver(_config(m))
            items.append((f, s["U"][at:at + f.n_dofs], _dt(m), 1e9))
            at += f.n_dofs
        s["batch"] = DeviceBatch(items)
        return s
    f = s["solver"] = FRSolver(_config(c))
    U = s["U"] = _state(c, seed, dev).reshape(-1)
    if kind == "f32":
        s["U"] = U.float()
        s["out"] = torch.empty_like(s["U"])
    elif kind == "step":
        s["U0"], s["it"], s["dt"] = U.clone(), Integrator(f, c["scheme"]), _dt(c)
    elif kind == "newton":
        s["b"] = torch.empty_like(U)
        f.rhs_func(0.0, U, s["b"])
    elif kind == "blocks":
        nd = 4 * (c["p"] + 1) ** 2
        s["out"] = torch.empty(c["slots"] * f.n_elems * nd * nd, dtype=torch.float64, device=dev)
    else:
        s["out"] = torch.empty_like(U)
        if kind == "jvp" or c.get("form") == "ifunction":
            s["V"] = _noise(tuple(U.shape), dev, _gen(dev, seed + 7))
        if kind == "jvp":
            f.pre_jv_eval(0.0, U, _sigma(c))
    return s


def run(s):
    kind, c = s["kind"], s["case"]
    if kind == "run1d":
        s["U"].copy_(s["U0"])
        s["it"].run(s["U"], s["dt"], n_steps=c["steps"], graph=True)
        return s["U"]
    if kind == "batch":
        s["U"].copy_(s["U0"])
        s["batch"].run(max_steps=BATCH_STEPS)
        return s["U"]
    f = s["solver"]
    if kind == "rhs":
        if c["form"] == "ifunction":
            f.fun_implicit(0.0, s["U"], s["V"], s["out"])
        else:
            f.rhs_func(0.0, s["U"], s["out"])
        return s["out"]
    if kind == "f32":
        f.residual_kernel_f32(0.0, s["U"], s["out"])
        return s["out"]
    if kind == "step":
        s["U"].copy_(s["U0"])  # a step from the same state, so that every pass does the same work
        s["it"].step(s["U"], 0.0, s["dt"])
        return s["U"]
    if kind == "jvp":
        f.matmult(s["V"], s["out"])
        return s["out"]
    sigma = _sigma(c)
    if kind == "blocks":
        (f.jac_blocks5 if c["slots"] == 5 else f.jac_blocks)(0.0, sigma, s["U"], s["out"])
        return s["out"]
    # solved to rounding, so that the answer does not hang on the number of Krylov steps
    f.pre_jv_eval(0.0, s["U"], sigma)
    f.pc_setup_gs(0.0, sigma, s["U"])
    return gmres(f.matmult, f.pc_apply, s["b"], restart=RESTART, rtol=1e-12, max_iter=8 * RESTART)[0]


# ---------------------------------------------------------------- work
def work(case):
    c, kind = case, case["kind"]
    if kind == "run1d":
        n = c["p"] + 1
        nodes = c["nx"] * n
        return dict(bytes=2.0 * 8 * 3 * nodes, flops=c["steps"] * 3.0 * nodes * (120 + 6 * n))
    if kind == "batch":
        per = [work(m) for m in _members(c)]
        return dict(bytes=sum(w["bytes"] for w in per), flops=BATCH_STEPS * sum(w["flops"] for w in per))
    n = c["p"] + 1
    nel = c["nx"] * c["ny"]
    nodes, nd = nel * n * n, 4 * n * n
    vec = 8.0 * 4 * nodes                      # one FP64 vector
    curved = c["geom"] != "cart"
    geo = 32.0 * nodes if curved else 0.0      # metrics, read once
    res = nodes * (310.0 + (32 if curved else 16) * n)   # operations of one residual
    jvp = 3.0 * res
    if kind == "rhs":
        return dict(bytes=(3 if c["form"] == "ifunction" else 2) * vec + geo, flops=res)
    if kind == "f32":
        return dict(bytes=vec + geo, flops=res)
    if kind == "step":
        return dict(bytes=2 * vec + geo, flops=(3 if c["scheme"] == "ssprk3" else 4) * res)
    if kind == "jvp":
        return dict(bytes=3 * vec + geo, flops=jvp)
    if kind == "blocks":
        # the blocks are written whole; a flux Jacobian per node, two per face point
        return dict(bytes=vec + geo + 8.0 * c["slots"] * nd * nd * nel, flops=8.0 * res)
    # one cycle: the set-up's inversions; per step a product, a sweep over the FP32 inverses
    # and the basis, read once for the projections and once for the update
    inv = 4.0 * nd * nd * nel
    basis = sum(2 * (j + 1) for j in range(RESTART)) * vec
    return dict(bytes=RESTART * (inv + 3 * vec + geo) + basis,
                flops=2.0 * nd ** 3 * nel + RESTART * (jvp + 3.0 * nd * nd * nel) + basis / 4)


# ---------------------------------------------------------------- exact values: plain torch, FP64
def _gll(p):
    """GLL nodes, weights and differentiation matrix of order p."""
    L = np.polynomial.legendre.Legendre
    x = np.concatenate([[-1.0], np.sort(np.real(L.basis(p).deriv().roots())), [1.0]]) if p > 1 else np.array([-1.0, 1.0])
    x = 0.5 * (x - x[::-1])
    w = 2.0 / (p * (p + 1) * L.basis(p)(x) ** 2)
    n = p + 1
    lam = np.array([1.0 / np.prod([x[i] - x[k] for k in range(n) if k != i]) for i in range(n)])
    D = np.zeros((n, n))
    for i in range(n):
        for j in range(n):
            if i != j:
                D[i, j] = lam[j] / (lam[i] * (x[i] - x[j]))
        D[i, i] = sum(1.0 / (x[i] - x[k]) for k in range(n) if k != i)
    return x, w, D


def _lifts(p, x):
    """Derivatives of the DG correction functions (VCJH c = 0) at the nodes."""
    L = np.polynomial.legendre.Legendre
    a, b = L.basis(p).deriv()(x), L.basis(p + 1).deriv()(x)
    return (1.0 if p % 2 == 0 else -1.0) * 0.5 * (a - b), 0.5 * (a + b)


def _filter(p, x, w, cut):
    V = np.stack([np.polynomial.legendre.Legendre.basis(j)(x) for j in range(p + 1)], axis=1)
    i = np.arange(p + 1)
    sig = np.where(i < cut, 1.0, np.exp(-36.0 * (np.maximum(i - cut, 0) / (p - cut)) ** 32.0))
    gam = np.where(i < p, 2.0 / (2.0 * i + 1.0), 2.0 / p)
    return V @ np.diag(sig / gam) @ V.T @ np.diag(w)


class _Mesh:
    """Node coordinates, metrics (xi_x, xi_y, eta_x, eta_y), face normals and operators."""

    def __init__(self, c, dev):
        p, nx, ny = c["p"], c["nx"], c["ny"]
        self.c, self.p, self.n, self.nx, self.ny, self.dev = c, p, p + 1, nx, ny, dev
        self.lx, self.ly = dict(blast=(1.0, 1.0), vortex=(10.0, 10.0), bump=(3.0, 0.8))[c["flow"]]
        xi, w, D = _gll(p)
        t = lambda v: torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device=dev)
        self.w, self.D = t(w), t(D)
        self.dL, self.dR = (t(v) for v in _lifts(p, xi))
        self.xi, self.wn = xi, w
        xr = t(xi)
        i, j = torch.arange(nx, device=dev, dtype=torch.float64), torch.arange(ny, device=dev, dtype=torch.float64)
        cs = ((i[:, None] + 0.5 * (1 + xr)) / nx)[None, :, None, :]       # (1, nx, 1, k)
        et = ((j[:, None] + 0.5 * (1 + xr)) / ny)[:, None, :, None]       # (ny, 1, l, 1)
        self.curved = c["geom"] != "cart"
        self.x, self.y = self._map(*torch.broadcast_tensors(cs, et))
        if not self.curved:
            self.met = (2.0 * nx / self.lx, 0.0, 0.0, 2.0 * ny / self.ly)
            self.xn, self.yn = (1.0, 0.0), (0.0, 1.0)
            return
        xr_, yr_, xs_, ys_ = self._jac(*torch.broadcast_tensors(cs, et))
        a, b = 0.5 / nx, 0.5 / ny
        det = (xr_ * a) * (ys_ * b) - (xs_ * b) * (yr_ * a)
        self.met = (ys_ * b / det, -xs_ * b / det, -yr_ * a / det, xr_ * a / det)
        I, J = torch.arange(nx + 1, device=dev, dtype=torch.float64), torch.arange(ny + 1, device=dev, dtype=torch.float64)
        xf = self._jac(*torch.broadcast_tensors((I / nx)[None, :, None], et[:, :, :, 0]))
        yf = self._jac(*torch.broadcast_tensors(cs[:, :, 0, :], (J / ny)[:, None, None]))
        unit = lambda u, v: (u / torch.sqrt(u * u + v * v), v / torch.sqrt(u * u + v * v))
        self.xn, self.yn = unit(xf[3], -xf[2]), unit(-yf[1], yf[0])

    def _map(self, cs, et):
        if self.c["geom"] == "warp":
            d = 0.1 * torch.sin(2 * math.pi * cs) * torch.sin(2 * math.pi * et)
            return self.lx * cs + d, self.ly * et + d
        if self.c["geom"] == "bump":
            x = -1.5 + self.lx * cs
            return x, 0.0625 * torch.exp(-25.0 * x * x) * (1.0 - et) + self.ly * et
        return self.lx * cs, self.ly * et

    def _jac(self, cs, et):
        """dx/dcsi, dy/dcsi, dx/deta, dy/deta."""
        if self.c["geom"] == "warp":
            q = 2 * math.pi * 0.1
            dc = q * torch.cos(2 * math.pi * cs) * torch.sin(2 * math.pi * et)
            de = q * torch.sin(2 * math.pi * cs) * torch.cos(2 * math.pi * et)
            return self.lx + dc, dc, de, self.ly + de
        x = -1.5 + self.lx * cs
        h = 0.0625 * torch.exp(-25.0 * x * x)
        return (torch.full_like(h, self.lx), -50.0 * x * h * self.lx * (1.0 - et), torch.zeros_like(h), self.ly - h)


def _pressure(gas, rho, e):
    if gas == "ideal":
        return (GAMMA - 1.0) * rho * e
    a, b = VDW
    return (GAMMA - 1.0) * rho * (e + a * rho) / (1.0 - b * rho) - a * rho * rho


def _prim(gas, U):
    rho, E = U[..., 0], U[..., 3]
    u, v = U[..., 1] / rho, U[..., 2] / rho
    e = E / rho - 0.5 * (u * u + v * v)
    p = _pressure(gas, rho, e)
    if gas == "ideal":
        c2 = GAMMA * p / rho
    else:
        a, b = VDW
        q = (1.0 - b * rho) ** 2
        c2 = GAMMA * (GAMMA - 1.0) * (e + a * rho) / q + (GAMMA - 1.0) * a * rho * (2.0 - b * rho) / q - 2.0 * a * rho
    return rho, u, v, p, E, c2


def _sabs(x):
    return torch.sqrt(x * x + 1e-14) - 1e-7


def _smax(a, b):
    return 0.5 * (a + b + _sabs(a - b))


def _smin(a, b):
    return 0.5 * (a + b - _sabs(a - b))


def _sel(cond, a, b):
    return torch.where(cond, a, b)


def _riemann(c, UL, UR, nx, ny):
    rL, uL, vL, pL, EL, c2L = _prim(c["gas"], UL)
    rR, uR, vR, pR, ER, c2R = _prim(c["gas"], UR)
    cL, cR = torch.sqrt(c2L), torch.sqrt(c2R)
    nL, tL, nR, tR = uL * nx + vL * ny, vL * nx - uL * ny, uR * nx + vR * ny, vR * nx - uR * ny
    qL, qR = (rL, rL * nL, rL * tL, EL), (rR, rR * nR, rR * tR, ER)
    FL = (rL * nL, rL * nL * nL + pL, rL * nL * tL, (EL + pL) * nL)
    FR = (rR * nR, rR * nR * nR + pR, rR * nR * tR, (ER + pR) * nR)
    if c["riemann"] == "rusanov":
        s = _smax(_sabs(nL) + cL, _sabs(nR) + cR)
        f = [0.5 * (a + b) - 0.5 * s * (y - x) for a, b, x, y in zip(FL, FR, qL, qR)]
    else:
        re = lambda z: z.real if z.is_complex() else z
        sL, sR = _smin(nL - cL, nR - cR), _smax(nL + cL, nR + cR)
        dL, dR = rL * (sL - nL), rR * (sR - nR)
        sM = (pR - pL + nL * dL - nR * dR) / (dL - dR)
        left = re(sM) >= 0
        q = [_sel(left, x, y) for x, y in zip(qL, qR)]
        F = [_sel(left, x, y) for x, y in zip(FL, FR)]
        sK, nK, tK, pK = _sel(left, sL, sR), _sel(left, nL, nR), _sel(left, tL, tR), _sel(left, pL, pR)
        ps = pK + q[0] * (sK - nK) * (sM - nK)
        inv = 1.0 / (sK - sM)
        st0 = sM * (sK * q[0] - F[0]) * inv
        st = [st0, (sM * (sK * q[1] - F[1]) + sK * ps) * inv, tK * st0, (sM * (sK * q[3] - F[3]) + sK * ps * sM) * inv]
        takeL, star = re(sL) >= 0, left | (re(sR) >= 0)
        f = [_sel(takeL, a, _sel(star, s_, b)) for a, s_, b in zip(FL, st, FR)]
    return torch.stack([f[0], f[1] * nx - f[2] * ny, f[1] * ny + f[2] * nx, f[3]], dim=-1)


def _ghost(c, face, q, nx, ny):
    """Ghost state of a boundary face from the interior trace q."""
    kind = c["bc"]
    if kind == "outflow":
        return q
    r, ru, rv, E = q.unbind(-1)
    if kind == "walls":
        return torch.stack([r, -ru, rv, E] if face in "LR" else [r, ru, -rv, E], dim=-1)
    if face == "L":    # subsonic inflow: total pressure and temperature 1, R = 1, along x
        _, _, _, p, _, _ = _prim(c["gas"], q)
        p = torch.where((p.real if p.is_complex() else p) > P_TOTAL, torch.full_like(p, P_TOTAL), p)
        M2 = 2.0 / (GAMMA - 1.0) * ((P_TOTAL / p) ** ((GAMMA - 1.0) / GAMMA) - 1.0)
        rho = p * (1.0 + 0.5 * (GAMMA - 1.0) * M2)
        u = torch.sqrt(M2) * torch.sqrt(GAMMA * p / rho)
        return torch.stack([rho, rho * u, 0.0 * rho, p / (GAMMA - 1.0) + 0.5 * rho * u * u], dim=-1)
    if face == "R":    # static pressure outlet
        return torch.stack([r, ru, rv, _p_out() / (GAMMA - 1.0) + 0.5 * (ru * ru + rv * rv) / r], dim=-1)
    vn = (ru * nx + rv * ny) / r   # slip wall
    return torch.stack([r, ru - 2.0 * r * vn * nx, rv - 2.0 * r * vn * ny, E], dim=-1)


def _at(v, idx):
    return v[idx] if torch.is_tensor(v) else v


def _residual(m, U):
    """R(U) of a (ny, nx, l, k, 4) state (real or complex)."""
    c = m.c
    D, dL, dR = (v.to(U.dtype) for v in (m.D, m.dL, m.dR))
    rho, u, v, p, E, _ = _prim(c["gas"], U)
    F = torch.stack([U[..., 1], U[..., 1] * u + p, U[..., 1] * v, u * (E + p)], dim=-1)
    G = torch.stack([U[..., 2], U[..., 1] * v, U[..., 2] * v + p, v * (E + p)], dim=-1)
    xi = lambda q: torch.einsum("km,jilme->jilke", D, q)
    eta = lambda q: torch.einsum("lm,jimke->jilke", D, q)
    if m.curved:
        a, b, d, e = (v_[..., None] for v_ in m.met)
        R = a * xi(F) + b * xi(G) + d * eta(F) + e * eta(G)
    else:
        R = m.met[0] * xi(F) + m.met[3] * eta(G)
    per = c["bc"] == "periodic"
    col = lambda v_: v_[..., None] if torch.is_tensor(v_) else v_
    for axis in (0, 1):
        if axis == 0:     # traces (ny, nx, l, 4); faces along dim 1
            lo, hi, dim, (nx, ny), names = U[:, :, :, 0], U[:, :, :, -1], 1, m.xn, "LR"
            Fl, Fh, Gl, Gh = F[:, :, :, 0], F[:, :, :, -1], G[:, :, :, 0], G[:, :, :, -1]
        else:             # traces (ny, nx, k, 4); faces along dim 0
            lo, hi, dim, (nx, ny), names = U[:, :, 0], U[:, :, -1], 0, m.yn, "BT"
            Fl, Fh, Gl, Gh = F[:, :, 0], F[:, :, -1], G[:, :, 0], G[:, :, -1]
        N = lo.shape[dim]
        first, last = ((slice(None),) * dim + (slice(0, 1),)), ((slice(None),) * dim + (slice(N, N + 1),))
        end = (slice(None),) * dim + (slice(N - 1, N),)
        gl = hi[end] if per else _ghost(c, names[0], lo[first], _at(nx, first), _at(ny, first))
        gr = lo[first] if per else _ghost(c, names[1], hi[end], _at(nx, last), _at(ny, last))
        fs = _riemann(c, torch.cat([gl, hi], dim), torch.cat([lo, gr], dim), nx, ny)
        below, above = (slice(None),) * dim + (slice(0, N),), (slice(None),) * dim + (slice(1, N + 1),)
        g0, g1 = m.met[2 * axis], m.met[2 * axis + 1]
        sc = torch.sqrt(g0 * g0 + g1 * g1) if m.curved else abs(g0) + abs(g1)
        node = (lambda q, hi_: (q[..., -1 if hi_ else 0] if axis == 0 else q[:, :, -1 if hi_ else 0])) if m.curved else (lambda q, _: q)
        dl = col(node(sc, 0)) * (fs[below] - Fl * col(_at(nx, below)) - Gl * col(_at(ny, below)))
        dr = col(node(sc, 1)) * (fs[above] - Fh * col(_at(nx, above)) - Gh * col(_at(ny, above)))
        if axis == 0:
            R = R + dl.unsqueeze(3) * dL[:, None] + dr.unsqueeze(3) * dR[:, None]
        else:
            R = R + dl.unsqueeze(2) * dL[:, None, None] + dr.unsqueeze(2) * dR[:, None, None]
    return R


def _pp_limit(gas, U, w, eps0=1e-13):
    """Zhang-Shu scaling of an (elements, nodes, 4 or 3) state with weights w."""
    pres = lambda q: _pressure(gas, q[..., 0], (q[..., -1] - 0.5 * (q[..., 1:-1] ** 2).sum(-1) / q[..., 0]) / q[..., 0])
    need = ~((U[..., 0] > eps0 * (1 + 1e-10)) & (pres(U) > eps0 * (1 + 1e-10))).all(1)
    if not bool(need.any()):
        return U
    V = U[need]
    ub = (V * w[None, :, None]).sum(1) / w.sum()
    pb = pres(ub)
    ok = (ub[:, 0] > 0) & (pb > 0)
    eps = torch.minimum(torch.full_like(pb, eps0), torch.minimum(ub[:, 0], pb))
    rmin = V[..., 0].amin(1)
    th = torch.where(ok & (rmin < eps), (ub[:, 0] - eps) / (ub[:, 0] - rmin), torch.ones_like(rmin))
    V = V.clone()
    V[..., 0] = ub[:, None, 0] + th[:, None] * (V[..., 0] - ub[:, None, 0])
    lo, hi = torch.zeros_like(V[..., 0]), torch.ones_like(V[..., 0])
    bad = ~(pres(V) >= eps[:, None])
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        s = ub[:, None] + mid[..., None] * (V - ub[:, None])
        good = (s[..., 0] > 0) & (pres(s) >= eps[:, None])
        lo, hi = torch.where(good, mid, lo), torch.where(good, hi, mid)
    th2 = torch.where(bad, lo, torch.ones_like(lo)).amin(1)
    th2 = torch.where(ok, th2, torch.ones_like(th2))
    out = U.clone()
    out[need] = torch.where((th2 < 1)[:, None, None], ub[:, None] + th2[:, None, None] * (V - ub[:, None]), V)
    return out


def _weno_lines(m, U, axis):
    """WENO limiter with the shock sensor along one axis of a (ny, nx, l, k, 4) state."""
    per, D, w = m.c["bc"] == "periodic", m.D, m.w
    dim = 1 if axis == 0 else 0
    q = U if axis == 0 else U.transpose(2, 3)      # the line index last but one
    prev, nxt = torch.roll(q, 1, dim), torch.roll(q, -1, dim)
    if not per:
        prev, nxt = prev.clone(), nxt.clone()
        prev.select(dim, 0).zero_()
        nxt.select(dim, -1).zero_()
    along = lambda v: (v * w[:, None]).sum(-2)

    def smooth(v):
        beta, fac = 0.0, 4.0
        for _ in range(m.n - 1):
            v = torch.einsum("rc,jilce->jilre", D, v)
            beta = beta + fac * 0.5 * along(v * v)
            fac *= 4.0
        return beta

    gam = ((1 - 0.998) * 0.5, 0.998, (1 - 0.998) * 0.5)
    cg = [g / (1e-6 + smooth(v)) ** 2 for g, v in zip(gam, (prev, q, nxt))]
    tot = cg[0] + cg[1] + cg[2]
    cg = [v / tot for v in cg]
    num = sum((v / g - 1.0).abs() for v, g in zip(cg, gam))
    hit = (num / (abs(1.0 / min(gam) - 1.0) + 2.0)).abs() >= 0.8
    av = [0.5 * along(v) for v in (prev, q, nxt)]
    e = lambda v: v.unsqueeze(-2)
    lim = e(cg[0]) * (prev - e(av[0]) + e(av[1])) + e(cg[1]) * q + e(cg[2]) * (nxt - e(av[2]) + e(av[1]))
    out = torch.where(e(hit), lim, q)
    return out if axis == 0 else out.transpose(2, 3)


def _exact_step(c, U, dt, steps=1):
    m = _Mesh(c, U.device)
    n = m.n
    ww = (m.w[:, None] * m.w[None, :]).reshape(-1)
    pp = c["stab"] != "none"
    limit = (lambda q: _pp_limit(c["gas"], q.reshape(-1, n * n, 4), ww).reshape(q.shape)) if pp else (lambda q: q)
    Fm = torch.as_tensor(_filter(m.p, m.xi, m.wn, min(2, m.p - 1)), device=U.device) if c["stab"] == "filter" else None
    L = lambda q: -_residual(m, q)
    for _ in range(steps):
        if c["scheme"] == "ssprk3":
            a = limit(U + dt * L(U))
            b = limit(0.75 * U + 0.25 * a + 0.25 * dt * L(a))
            last = U / 3.0 + 2.0 / 3.0 * b + 2.0 * dt / 3.0 * L(b)
        else:
            k1 = L(U)
            k2 = L(limit(U + 0.5 * dt * k1))
            # each stage input is the limited output of the stage before
            a = limit(U + 0.5 * dt * k2)
            k3 = L(a)
            k4 = L(limit(U + dt * k3))
            last = U + dt / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
        if c["stab"] == "filter":
            last = 0.5 * (torch.einsum("rc,jilce->jilre", Fm, last) + torch.einsum("rc,jicke->jirke", Fm, last))
        elif c["stab"] == "weno":
            last = limit(last)
            last = 0.5 * (_weno_lines(m, last, 0) + _weno_lines(m, last, 1))
        U = limit(last)
    return U


def _exact_1d(c, U):
    p, N = c["p"], c["nx"]
    xi, w, D = _gll(p)
    dL, dR = _lifts(p, xi)
    t = torch.from_numpy
    F_, D_, dL_, dR_, w_ = t(_filter(p, xi, w, min(2, p - 1))), t(D), t(dL), t(dR), t(w)
    U, dt, jac = t(U), _dt1d(c), 2.0 * N

    def flux(q):
        u = q[:, 1] / q[:, 0]
        pr = (GAMMA - 1.0) * (q[:, 2] - 0.5 * q[:, 1] * u)
        return torch.stack([q[:, 1], q[:, 1] * u + pr, (q[:, 2] + pr) * u], dim=1), u, torch.sqrt(GAMMA * pr / q[:, 0])

    def rhs(q):
        F, u, a = flux(q)
        lo, hi = (lambda v: v[..., 0]), (lambda v: v[..., -1])
        ext = lambda v: (torch.cat([lo(v)[:1], hi(v)]), torch.cat([lo(v), hi(v)[-1:]]))   # left and right states of the faces
        (qL, qR), (fL, fR), (uL, uR), (aL, aR) = ext(q), ext(F), ext(u), ext(a)
        s = _smax(_sabs(uL) + aL, _sabs(uR) + aR)[:, None]
        fs = 0.5 * (fL + fR) - 0.5 * s * (qR - qL)
        R = torch.einsum("km,jem->jek", D_, F)
        R = R + (fs[:-1] - lo(F))[..., None] * dL_ + (fs[1:] - hi(F))[..., None] * dR_
        return -jac * R

    lim = lambda q: _pp_limit("ideal", q.transpose(1, 2), w_).transpose(1, 2)
    for _ in range(c["steps"]):
        a = lim(U + dt * rhs(U))
        b = lim(0.75 * U + 0.25 * a + 0.25 * dt * rhs(a))
        U = U / 3.0 + 2.0 / 3.0 * b + 2.0 * dt / 3.0 * rhs(b)
        U = lim(torch.einsum("rc,jec->jer", F_, U))
    return U


def _jvp(m, U, V, h=1e-30):
    return _sigma(m.c) * V + _residual(m, torch.complex(U, h * V)).imag / h


def _blocks(m, U, slots):
    """Blocks (element, slot, column, row) of the Jacobian; slots self, right, top, bottom, left."""
    ny, nx, nd = m.ny, m.nx, 4 * m.n * m.n
    dev = U.device
    B = torch.zeros((ny, nx, slots, nd, nd), dtype=torch.float64, device=dev)
    colour = (torch.arange(nx, device=dev)[None, :] + 2 * torch.arange(ny, device=dev)[:, None]) % 5
    for k in range(5):
        on = (colour == k).double()[:, :, None]
        slot = (k - colour) % 5
        for d in range(nd):
            V = torch.zeros((ny, nx, nd), dtype=torch.float64, device=dev)
            V[:, :, d:d + 1] = on
            J = _jvp(m, U, V.reshape(U.shape)).reshape(ny, nx, nd)
            for s in range(slots):
                hit = slot == s
                B[:, :, s, d][hit] = J[hit]
    return B


def _exact_solve(m, U, b):
    """J x = b by GMRES without restart, preconditioned by the diagonal blocks, in FP64."""
    ny, nx, nd = m.ny, m.nx, 4 * m.n * m.n
    inv = torch.linalg.inv(_blocks(m, U, 1)[:, :, 0].transpose(-1, -2))
    M = lambda v: torch.einsum("jiab,jib->jia", inv, v.reshape(ny, nx, nd)).reshape(-1)
    J = lambda v: _jvp(m, U, v.reshape(U.shape)).reshape(-1)
    x = torch.zeros_like(b)
    for _ in range(4):
        r = b - J(x)
        beta = float(r.norm())
        if beta <= 1e-14 * float(b.norm()):
            break
        V, Z, H = [r / beta], [], np.zeros((101, 100))
        for j in range(100):
            Z.append(M(V[j]))
            w = J(Z[j])
            for _pass in range(2):
                for i, v in enumerate(V):
                    h = float(v @ w)
                    H[i, j] += h
                    w = w - h * v
            H[j + 1, j] = float(w.norm())
            V.append(w / H[j + 1, j])
            e = np.zeros(j + 2)
            e[0] = beta
            y = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)[0]
            if np.linalg.norm(H[:j + 2, :j + 1] @ y - e) <= 1e-15 * float(b.norm()):
                break
        for yi, z in zip(y, Z):
            x = x + float(yi) * z
    return x


def exact(case, seed):
    c, kind = dict(case), case["kind"]
    dev = torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")
    if kind == "run1d":
        return _exact_1d(c, _state1d(c, seed)).reshape(-1).numpy()
    if kind == "batch":
        return torch.cat([_exact_step(m, _state(m, seed + 101 * k, dev), _dt(m), BATCH_STEPS).reshape(-1)
                          for k, m in enumerate(_members(c))])
    U = _state(c, seed, dev)
    if kind == "f32":
        return _residual(_Mesh(c, dev), U.float().double()).reshape(-1)
    if kind == "step":
        return _exact_step(c, U, _dt(c)).reshape(-1)
    m = _Mesh(c, dev)
    if kind == "rhs" and c["form"] == "rhs":
        return -_residual(m, U).reshape(-1)
    if kind == "blocks":
        return _blocks(m, U, c["slots"]).reshape(-1)
    if kind == "newton":
        return _exact_solve(m, U, -_residual(m, U).reshape(-1))
    V = _noise((U.numel(),), dev, _gen(dev, seed + 7))
    if kind == "rhs":
        return V + _residual(m, U).reshape(-1)
    return _jvp(m, U, V.reshape(U.shape)).reshape(-1)
