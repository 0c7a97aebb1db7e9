"""GPU: the complex-step product where HLLC's contact speed is exactly zero.  There the
reference's branch test on Re + Im picks the star state by the sign of the perturbation
(riemann_solver.hpp:314-341 on complex scalars), so the product is not linear in V; the
oracle computes Im(R(U + ihV)) / h as documented."""
import numpy as np
import pytest
import torch

from oracle.oracle import Oracle
from tests.helpers import TOL_JVP, rel_err

from fr_sdg_b200 import FRSolver
from fr_sdg_b200 import _abi as A
from fr_sdg_b200.workloads import make_config

pytestmark = pytest.mark.gpu


def _cfg(gas, p, n_elems, h):
    return make_config(dim=2, p=p, n_elems=n_elems, box=(1.0, 1.0), riemann="hllc", gas=gas, vdw=(0.05, 0.02), csd_eps=h,
                       bcs={f: A.BC_OUTFLOW for f in (A.LEFT, A.RIGHT, A.TOP, A.BOTTOM)})


def _state(cfg, flow):
    """Columns of elements in turn: a resting contact (densities 1 and 2) or a shear layer
    (tangential velocities +-1/2), uniform pressure; both sides' pressures have the same bits."""
    nx, ny, nn = cfg.n_elems[0], cfg.n_elems[1], (cfg.poly_deg + 1) ** 2
    odd = (np.arange(nx) % 2 == 1)[None, :, None] & np.ones((ny, nx, nn), dtype=bool)
    rho = np.where(odd, 2.0, 1.0) if flow == "contact" else np.ones(odd.shape)
    v = np.zeros(odd.shape) if flow == "contact" else np.where(odd, 0.5, -0.5)
    E = np.full(odd.shape, 2.5) + 0.5 * rho * v * v
    return np.stack([rho, np.zeros(odd.shape), rho * v, E], axis=-1).reshape(-1)


@pytest.mark.parametrize("gas,flow", [("ideal", "contact"), ("ideal", "shear"), ("vdw", "shear")])
@pytest.mark.parametrize("h", [1e-30, 1e-20])
@pytest.mark.parametrize("p", [1, 2, 5])
def test_product_follows_the_sign_of_the_perturbation(p, h, gas, flow, cuda):
    cfg = _cfg(gas, p, (4, 4), h)
    U = _state(cfg, flow)
    V = np.random.default_rng(p).normal(size=U.size)
    o = Oracle(cfg)
    plus, minus = o.jvp(0.0, 1.5, U, V), o.jvp(0.0, 1.5, U, -V)
    assert rel_err(-minus, plus) > 1e-3  # the tie is met
    with FRSolver(cfg) as s:
        Ud, out = torch.from_numpy(U).to(cuda), torch.empty(U.size, dtype=torch.float64, device=cuda)
        s.pre_jv_eval(0.0, Ud, 1.5)
        for W, ref in ((V, plus), (-V, minus)):
            s.matmult(torch.from_numpy(W).to(cuda), out)
            assert rel_err(out.cpu().numpy(), ref) <= TOL_JVP


@pytest.mark.parametrize("gas,flow", [("ideal", "contact"), ("vdw", "shear")])
def test_blocks_equal_single_seed_products(gas, flow, cuda):
    cfg = _cfg(gas, 1, (4, 3), 1e-30)
    U = _state(cfg, flow)
    o, nd, ne = Oracle(cfg), 16, 12
    ref = np.zeros((ne, nd, nd))
    for e in range(ne):
        for c in range(nd):
            V = np.zeros(U.size)
            V[e * nd + c] = 1.0
            ref[e, c] = o.jvp(0.0, 1.5, U, V)[e * nd:(e + 1) * nd]
    with FRSolver(cfg) as s:
        B = torch.empty(ne * nd * nd, dtype=torch.float64, device=cuda)
        s.jac_blocks(0.0, 1.5, torch.from_numpy(U).to(cuda), B)
    assert rel_err(B.cpu().numpy().reshape(ref.shape), ref) <= TOL_JVP


def test_inadmissible_node_is_not_plausible(cuda):
    """A negative pressure makes the sound speed imaginary: its value enters the imaginary part,
    and Im / h is of order 1 / h, in the oracle and here."""
    cfg = _cfg("ideal", 2, (4, 4), 1e-30)
    U = _state(cfg, "contact")
    U[4 * 9 * 5 + 2] = 5.0   # a boundary node of an inner element: kinetic energy above the total
    V = np.random.default_rng(3).normal(size=U.size)
    ref = np.abs(Oracle(cfg).jvp(0.0, 1.5, U, V)).max()
    with FRSolver(cfg) as s:
        out = torch.empty(U.size, dtype=torch.float64, device=cuda)
        s.pre_jv_eval(0.0, torch.from_numpy(U).to(cuda), 1.5)
        s.matmult(torch.from_numpy(V).to(cuda), out)
        got = float(out.abs().max())
    assert ref > 1e20 and not got < 1e20  # NaN counts as not plausible too


@pytest.mark.parametrize("flow", ["tangential", "isothermal"])
@pytest.mark.parametrize("p", [2, 3, 4])
def test_real_parts_round_as_complex_ones(p, flow, cuda):
    """Velocities along the y-faces of a curved mesh but for 1e-7, or one temperature and velocity at
    random densities: smooth_abs divides the rounding of the normal velocity, or of the
    difference of two equal wave speeds, by its 1e-7.  The first-order form has the complex form's
    real parts, but for one reciprocal in 3000 and one root in 25 (the complex root takes a
    hypot, which is not correctly rounded): an entry meets up to four face points, so most
    entries of the two differ by the rounding of their imaginary parts alone, a few units of
    2^-53 of their terms."""
    def product(h):
        cfg = make_config(dim=2, p=p, n_elems=(7, 6), box=(1.0, 1.0), riemann="rusanov", csd_eps=h,
                          geometry=A.GEOM_SINE_WARP, geom_params=(0.05, 0, 0, 0),
                          bcs={f: A.BC_PERIODIC for f in (A.LEFT, A.RIGHT, A.TOP, A.BOTTOM)})
        ex, ey = Oracle(cfg).node_metrics()[:, 2:4].T
        rng = np.random.default_rng(p)
        r = rng.uniform(-1, 1, (ex.size, 4))
        rho, pr, l = 1.0 + 0.1 * r[:, 0], 1.0 + 0.1 * r[:, 1], np.hypot(ex, ey)
        u, v = 0.5 * ey / l + 1e-7 * r[:, 2], -0.5 * ex / l + 1e-7 * r[:, 3]
        if flow == "isothermal":
            pr, u, v = rho, np.full_like(u, 0.5), np.full_like(v, 0.3)
        U = np.stack([rho, rho * u, rho * v, pr / 0.4 + 0.5 * rho * (u * u + v * v)], axis=1).reshape(-1)
        V = rng.normal(size=U.size)
        with FRSolver(cfg) as s:
            Ud, out = torch.from_numpy(U).to(cuda), torch.empty(U.size, dtype=torch.float64, device=cuda)
            s.pre_jv_eval(0.0, Ud, 1.0)
            s.matmult(torch.from_numpy(V).to(cuda), out)
        return out.cpu().numpy()
    a, b = product(1e-30), product(2e-20)  # first order, complex: second-order terms at 4e-40
    d = np.abs(a - b) / np.abs(b).max()
    assert np.median(d) <= 64 * 2.0 ** -53
