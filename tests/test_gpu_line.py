"""GPU: the line-per-thread residual where its tiles can go wrong -- meshes around the tile
sizes, meshes large enough for the tuned tile (small ones take the variant with face warps),
16-byte aligned pointers, row windows that move tile edges, and the stage epilogues."""
import numpy as np
import pytest
import torch

from oracle.oracle import Oracle
from tests.helpers import TOL_FP32, TOL_FP64, poisoned_state, random_state, rel_err

from fr_sdg_b200 import FRSolver
from fr_sdg_b200 import _abi as A
from fr_sdg_b200.workloads import make_config

pytestmark = pytest.mark.gpu

PER = {f: A.BC_PERIODIC for f in (A.LEFT, A.RIGHT, A.TOP, A.BOTTOM)}
MIX = {A.LEFT: A.BC_WALL, A.RIGHT: A.BC_OUTFLOW, A.TOP: A.BC_OUTFLOW, A.BOTTOM: A.BC_WALL}


def _cfg(p, n_elems, curved, **kw):
    base = dict(dim=2, p=p, n_elems=n_elems, box=(2.0, 1.5), riemann="hllc" if p % 2 else "rusanov", bcs=MIX)
    if p % 3 == 0:
        base.update(gas="vdw", vdw=(0.05, 0.02))
    if curved:
        base.update(geometry=A.GEOM_SINE_WARP, geom_params=(0.05, 0, 0, 0), bcs=PER)
    base.update(kw)
    return make_config(**base)


# around the tiles (8 x 8 down to 3 x 2) and beyond one residency of the small variant
@pytest.mark.parametrize("n_elems", [(2, 2), (9, 5), (8, 17), (131, 83)])
@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("p", range(1, 10))
def test_residual_at_tile_edges(p, curved, n_elems, cuda):
    cfg = _cfg(p, n_elems, curved)
    U = random_state(cfg, 100 + p)
    ref = Oracle(cfg, threads=8).residual(0.0, U)
    with FRSolver(cfg) as s:
        Ud = torch.from_numpy(U).to(cuda)
        R = torch.full_like(Ud, float("nan"))
        s.residual_kernel(0.0, Ud, R)
        assert rel_err(R.cpu().numpy(), ref) <= TOL_FP64
        # 16-byte aligned vectors that are not 32-byte aligned: the same bits
        V, Q = torch.empty(U.size + 2, dtype=torch.float64, device=cuda), torch.empty(U.size + 2, dtype=torch.float64, device=cuda)
        V[2:].copy_(Ud)
        s.residual_kernel(0.0, V[2:], Q[2:])
        assert torch.equal(Q[2:], R)
        U32 = Ud.float()
        R32 = torch.full_like(U32, float("nan"))
        s.residual_kernel_f32(0.0, U32, R32)
        assert s.status() == 0
    ref32 = Oracle(cfg, threads=8).residual(0.0, U32.double().cpu().numpy())
    assert rel_err(R32.double().cpu().numpy(), ref32) <= TOL_FP32


@pytest.mark.parametrize("p", [2, 3, 5, 8])
def test_row_window_on_a_large_mesh(p, cuda):
    """Rows 30 to 60 of a mesh beyond one residency: bit for bit the whole mesh's rows."""
    cfg = _cfg(p, (131, 90), False)
    nd = 4 * (p + 1) ** 2
    U = torch.from_numpy(random_state(cfg, 7)).to(cuda)
    row = 131 * nd
    with FRSolver(cfg) as s:
        R = torch.empty_like(U)
        s.residual_kernel(0.0, U, R)
        s.set_row_window(29, 32, 1, 31)
        W = U[29 * row: 61 * row].clone()
        Q = torch.full_like(W, float("nan"))
        s.residual_kernel(0.0, W, Q)
        assert torch.equal(Q[row: 31 * row], R[30 * row: 60 * row])


@pytest.mark.parametrize("n_elems", [(7, 5), (131, 83)])
@pytest.mark.parametrize("p", [2, 4, 5, 7])
@pytest.mark.parametrize("filt", [False, True])
def test_stage_epilogue_on_both_variants(p, filt, n_elems, cuda):
    """The limiter and the filter in the stage's launch against the stage and the passes."""
    cfg = _cfg(p, n_elems, False, gas="ideal", apply_filter=filt, cut_off=1, pp_limit=True, pp_eps=1e-6)
    U = torch.from_numpy(random_state(cfg, 3)).to(cuda)
    # out = A + gamma rhs(U) with nodes of A below the floor in every third element
    bad = torch.from_numpy(poisoned_state(cfg, 5)).to(cuda)
    with FRSolver(cfg) as s:
        for flag in (A.STAGE_LIMIT, A.STAGE_POST_STEP):
            ref, got = torch.empty_like(U), torch.empty_like(U)
            s.rk_stage(0.0, U, ref, 1e-6, bad, 1.0)
            s.pp_limit(ref) if flag == A.STAGE_LIMIT else s.apply_stabilization(ref)
            s.rk_stage_fused(0.0, U, got, flag, 1e-6, bad, 1.0)
            assert rel_err(got.cpu().numpy(), ref.cpu().numpy()) <= 1e-13


def test_non_finite_densities_are_counted(cuda):
    cfg = _cfg(3, (131, 83), False)
    U = torch.from_numpy(random_state(cfg, 9)).to(cuda)
    for k, v in ((0, float("nan")), (4 * 16 * 700 + 8, -1.0), (4 * 16 * 5000 + 4, float("inf")), (4 * 16 * 9000, 0.0)):
        U[k] = v
    with FRSolver(cfg) as s:
        R = torch.empty_like(U)
        s.residual_kernel(0.0, U, R)
        assert s.status() == 4


@pytest.mark.parametrize("n", [3, 32, 33, 200])
@pytest.mark.parametrize("p", [2, 3, 6, 9])
@pytest.mark.parametrize("gas", ["ideal", "vdw"])
def test_1d_stage_epilogue(p, n, gas, cuda):
    cfg = make_config(dim=1, p=p, n_elems=(n, 1), riemann="rusanov", gas=gas, vdw=(0.05, 0.02), apply_filter=True,
                      cut_off=1, pp_limit=True, pp_eps=1e-6, bcs={A.LEFT: A.BC_OUTFLOW, A.RIGHT: A.BC_WALL})
    U = torch.from_numpy(random_state(cfg, p + n)).to(cuda)
    bad = torch.from_numpy(poisoned_state(cfg, p)).to(cuda)
    with FRSolver(cfg) as s:
        for flag in (A.STAGE_LIMIT, A.STAGE_POST_STEP):
            ref, got = torch.empty_like(U), torch.full_like(U, float("nan"))
            s.rk_stage(0.0, U, ref, 1e-6, bad, 1.0)
            s.pp_limit(ref) if flag == A.STAGE_LIMIT else s.apply_stabilization(ref)
            s.rk_stage_fused(0.0, U, got, flag, 1e-6, bad, 1.0)
            assert rel_err(got.cpu().numpy(), ref.cpu().numpy()) <= 1e-13


@pytest.mark.parametrize("gas", ["ideal", "vdw"])
def test_limited_nodes_pass_the_floor(gas, cuda):
    """Every limited element's nodes stand at or above the floor in the limiter's own
    arithmetic: a second pass changes nothing."""
    cfg = _cfg(4, (40, 30), False, gas=gas, vdw=(0.05, 0.02), pp_limit=True, pp_eps=1e-6)
    U = torch.from_numpy(poisoned_state(cfg, 11)).to(cuda)
    with FRSolver(cfg) as s:
        s.pp_limit(U)
        V = U.clone()
        s.pp_limit(V)
    assert torch.equal(U, V)
