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
