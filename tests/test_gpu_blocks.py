"""GPU: the element-block preconditioners against dense FP64 sweeps over the blocks of
frsdg_jac_blocks5, at block sizes 16 to 144, with bounds derived from the FP32 storage of
the inverses and the couplings."""
import numpy as np
import pytest
import torch

from tests.helpers import random_state

from fr_sdg_b200 import FRSolver
from fr_sdg_b200 import _abi as A
from fr_sdg_b200.workloads import make_config

pytestmark = pytest.mark.gpu

U32 = 2.0 ** -24  # relative rounding error of an FP32 entry


def _cfg(p, n_elems, riemann="hllc", geometry=A.GEOM_WALL_PROFILE):
    return make_config(dim=2, p=p, n_elems=n_elems, box=(3.0, 0.8), riemann=riemann, geometry=geometry,
                       profile=A.PROFILE_GAUSS_BUMP, geom_params=(-1.5, 0.0625, 25.0, 0.0), csd_eps=1e-30,
                       bcs={A.LEFT: A.BC_OUTFLOW, A.RIGHT: A.BC_OUTFLOW, A.BOTTOM: A.BC_SLIP_WALL, A.TOP: A.BC_WALL})


def _blocks(s, cfg, U, sigma, cuda):
    """(ny, nx, 5, row, col) blocks of the Jacobian rows."""
    nx, ny = cfg.n_elems[0], cfg.n_elems[1]
    nd = s.n_dofs // s.n_elems
    B = torch.empty(s.n_elems * 5 * nd * nd, dtype=torch.float64, device=cuda)
    s.jac_blocks5(0.0, sigma, U, B)
    return B.view(ny, nx, 5, nd, nd).transpose(-1, -2)


def _sigma(cfg):
    """A few explicit time steps: diagonally heavy blocks, condition numbers of order 10."""
    p = cfg.poly_deg
    return 2.0 * (p + 1) ** 2 * (cfg.n_elems[0] / 3.0 + cfg.n_elems[1] / 0.8)


@pytest.mark.parametrize("p,n_elems", [(1, (7, 5)), (2, (6, 3)), (3, (5, 4)), (4, (3, 5)), (5, (3, 3))])
@pytest.mark.parametrize("geometry", [A.GEOM_WALL_PROFILE, A.GEOM_CARTESIAN])
def test_block_sweeps_match_dense(p, n_elems, geometry, cuda):
    cfg = _cfg(p, n_elems, "hllc" if p != 2 else "rusanov", geometry)
    sigma = _sigma(cfg)
    with FRSolver(cfg) as s:
        U = torch.from_numpy(random_state(cfg, 3 + p, amp=0.2)).to(cuda)
        B = _blocks(s, cfg, U, sigma, cuda)
        ny, nx, nd = B.shape[0], B.shape[1], B.shape[3]
        r = torch.randn(s.n_dofs, dtype=torch.float64, device=cuda, generator=torch.Generator(cuda).manual_seed(p))
        rv = r.view(ny, nx, nd)
        inv = torch.linalg.inv(B[:, :, 0])
        ap = lambda M, v: torch.einsum("jiab,jib->jia", M, v)

        def couple(M, z):
            out = torch.zeros_like(z)
            out[:, :-1] += ap(M[:, :-1, 1], z[:, 1:])
            out[:-1] += ap(M[:-1, :, 2], z[1:])
            out[1:] += ap(M[1:, :, 3], z[:-1])
            out[:, 1:] += ap(M[:, 1:, 4], z[:, :-1])
            return out

        # absolute forward errors: entries rounded to FP32 (U32 each), the FP64 inversion
        # and sums well below that
        Bi, Bo = inv.abs(), B.abs()
        z = torch.empty_like(r)
        s.pc_setup(0.0, sigma, U)
        s.pc_apply(r, z)
        ref = ap(inv, rv)
        bound = 1.01 * U32 * ap(Bi, rv.abs()) + 1e-11 * ref.abs().max()
        assert bool(((z.view_as(ref) - ref).abs() <= bound).all())

        red = ((torch.arange(nx, device=cuda)[None, :] + torch.arange(ny, device=cuda)[:, None]) % 2 == 0)[:, :, None]
        zero = torch.zeros_like(rv)
        z_r = torch.where(red, ap(inv, rv), zero)
        e_r = torch.where(red, U32 * ap(Bi, rv.abs()), zero)
        z_b = torch.where(red, zero, ap(inv, rv - couple(B, z_r)))
        t_b = rv.abs() + couple(Bo, z_r.abs())
        e_b = torch.where(red, zero, ap(Bi, U32 * t_b + couple(Bo, U32 * z_r.abs() + e_r)))
        c = couple(B, z_b)
        ref = torch.where(red, z_r - ap(inv, c), z_b)
        e_2 = ap(Bi, U32 * couple(Bo, z_b.abs()) + couple(Bo, U32 * z_b.abs() + e_b))
        bound = 1.05 * (torch.where(red, e_r + e_2, e_b)) + 1e-11 * ref.abs().max()
        s.pc_setup_gs(0.0, sigma, U)
        s.pc_apply(r, z)
        first = z.clone()
        assert bool(((z.view_as(ref) - ref).abs() <= bound).all())
        # the set-up is reproducible: the same blocks give the same bits
        s.pc_setup_gs(0.0, sigma, U)
        s.pc_apply(r, z)
        assert torch.equal(z, first)
