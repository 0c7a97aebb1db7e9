"""GPU: the block-Jacobi preconditioner under row windows.  The inverses stand at their
elements' global rows, so a window's products equal the whole mesh's rows bit for bit, ghost
rows give zero, and nothing of an earlier set-up is left in rows that the last one skipped."""
import pytest
import torch

from tests.helpers import random_state

from fr_sdg_b200 import FRSolver
from fr_sdg_b200 import _abi as A
from fr_sdg_b200.workloads import make_config

pytestmark = pytest.mark.gpu

NX, NY = 5, 6


def _cfg(p, periodic, geometry):
    y = A.BC_PERIODIC if periodic else A.BC_OUTFLOW
    return make_config(dim=2, p=p, n_elems=(NX, NY), box=(2.0, 1.5), riemann="hllc", geometry=geometry,
                       geom_params=(0.04, 0, 0, 0), csd_eps=1e-30,
                       bcs={A.LEFT: A.BC_PERIODIC, A.RIGHT: A.BC_PERIODIC, A.BOTTOM: y, A.TOP: y})


# (row_base, rows, row_begin, row_end); the second form holds two ghost rows beside the whole mesh
PERIODIC = [(-1, 5, 1, 4), (-1, NY + 2, 1, NY + 1), (2, 4, 1, 3), (3, 4, 1, 3)]
BOUNDED = [(0, 4, 0, 3), (2, 4, 1, 4), (1, 4, 1, 3), (0, NY, 0, NY)]


@pytest.mark.parametrize("p", [1, 3, 5])
@pytest.mark.parametrize("periodic", [False, True])
def test_windows_equal_the_whole_mesh(p, periodic, cuda):
    cfg = _cfg(p, periodic, A.GEOM_SINE_WARP if periodic else A.GEOM_CARTESIAN)
    sigma = 2.0 * (p + 1) ** 2 * NY
    row = NX * 4 * (p + 1) ** 2
    U = torch.from_numpy(random_state(cfg, 5, amp=0.2)).to(cuda)
    r = torch.randn(U.numel(), dtype=torch.float64, device=cuda, generator=torch.Generator(cuda).manual_seed(p))
    with FRSolver(cfg) as s:
        whole = torch.empty_like(r)
        s.pc_setup(0.0, sigma, U)
        s.pc_apply(r, whole)
        whole = whole.view(NY, row)
        for base, rows, begin, end in PERIODIC if periodic else BOUNDED:
            glob = [(base + j) % NY for j in range(rows)]
            Uw, rw = U.view(NY, row)[glob].reshape(-1), r.view(NY, row)[glob].reshape(-1)
            s.set_row_window(base, rows, begin, end)
            z = torch.full_like(rw, float("nan"))
            # the whole mesh's set-up seen through the window, then the window's own
            for own in (False, True):
                if own:
                    s.pc_setup(0.0, sigma, Uw)
                z.fill_(float("nan"))
                s.pc_apply(rw, z)
                v = z.view(rows, row)
                assert torch.equal(v[begin:end], whole[glob[begin:end]])
                assert not bool(v[:begin].any()) and not bool(v[end:].any())
            # the whole mesh after the window's set-up: its rows, zero elsewhere
            s.set_row_window(0, 0, 0, 0)
            z = torch.full_like(r, float("nan"))
            s.pc_apply(r, z)
            want = torch.zeros_like(whole)
            want[base + begin:base + end] = whole[base + begin:base + end]
            assert torch.equal(z.view(NY, row), want)
            s.pc_setup(0.0, sigma, U)


@pytest.mark.parametrize("p", [2, 6])
def test_blocks_under_a_window(p, cuda):
    cfg = _cfg(p, True, A.GEOM_CARTESIAN)
    nd = 4 * (p + 1) ** 2
    row = NX * nd
    U = torch.from_numpy(random_state(cfg, 8, amp=0.2)).to(cuda)
    with FRSolver(cfg) as s:
        B = torch.empty(NX * NY * nd * nd, dtype=torch.float64, device=cuda)
        s.jac_blocks(0.0, 3.0, U, B)
        B = B.view(NY, row * nd)
        for base, rows, begin, end in PERIODIC:
            glob = [(base + j) % NY for j in range(rows)]
            s.set_row_window(base, rows, begin, end)
            W = torch.empty(NX * rows * nd * nd, dtype=torch.float64, device=cuda)
            s.jac_blocks(0.0, 3.0, U.view(NY, row)[glob].reshape(-1), W)
            assert torch.equal(W.view(rows, row * nd)[begin:end], B[glob[begin:end]])


def test_gauss_seidel_sweep_refuses_a_window(cuda):
    """A sweep over a window's rows would take other elements' blocks."""
    cfg = make_config(dim=2, p=2, n_elems=(NX, NY), riemann="hllc", csd_eps=1e-30,
                      bcs={f: A.BC_OUTFLOW for f in (A.LEFT, A.RIGHT, A.TOP, A.BOTTOM)})
    U = torch.from_numpy(random_state(cfg, 2, amp=0.2)).to(cuda)
    with FRSolver(cfg) as s:
        s.pc_setup_gs(0.0, 50.0, U)
        s.set_row_window(2, 4, 1, 4)
        r = torch.zeros(s.n_dofs, dtype=torch.float64, device=cuda)
        with pytest.raises(A.FrsdgError):
            s.pc_apply(r, torch.empty_like(r))
        s.set_row_window(0, 0, 0, 0)
        s.pc_apply(U, torch.empty_like(U))
