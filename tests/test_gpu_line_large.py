"""GPU: the tuned tiles of the line-per-thread residual (meshes beyond one residency of the small
variant): curved and Van der Waals stage epilogues, the implicit form with and without the
change of variables, and columns redone with the checked functions."""
import numpy as np
import pytest
import torch

from oracle.oracle import Oracle
from tests.helpers import TOL_FP64, cons_to_prim, poisoned_state, random_state, rel_err

from fr_sdg_b200 import FRSolver
from fr_sdg_b200 import _abi as A
from fr_sdg_b200.workloads import make_config

pytestmark = pytest.mark.gpu

PER = {f: A.BC_PERIODIC for f in (A.LEFT, A.RIGHT, A.TOP, A.BOTTOM)}
OUT = {f: A.BC_OUTFLOW for f in (A.LEFT, A.RIGHT, A.TOP, A.BOTTOM)}
LARGE = (131, 83)


def _cfg(p, curved=False, **kw):
    base = dict(dim=2, p=p, n_elems=LARGE, box=(2.0, 1.5), riemann="hllc" if p % 2 else "rusanov", bcs=PER if curved else OUT)
    if curved:
        base.update(geometry=A.GEOM_SINE_WARP, geom_params=(0.05, 0, 0, 0))
    base.update(kw)
    return make_config(**base)


@pytest.mark.parametrize("p,filt", [(p, f) for p in (1, 2, 4, 5, 7, 9) for f in (False, True) if p > 1 or not f])
@pytest.mark.parametrize("curved,gas", [(True, "ideal"), (True, "vdw"), (False, "vdw")])
def test_stage_epilogue(p, filt, curved, gas, cuda):
    """In the stage's launch against the stage and the passes: the same values before the limiter,
    so equal up to the rounding of a filter sum and of the limiter's root."""
    cfg = _cfg(p, curved, gas=gas, vdw=(0.05, 0.02), apply_filter=filt, cut_off=1, pp_limit=True, pp_eps=1e-6)
    U = torch.from_numpy(random_state(cfg, 3)).to(cuda)
    bad = torch.from_numpy(poisoned_state(cfg, 5)).to(cuda)
    with FRSolver(cfg) as s:
        for flag in (A.STAGE_LIMIT, A.STAGE_POST_STEP):
            ref, got = torch.empty_like(U), torch.full_like(U, float("nan"))
            s.rk_stage(0.0, U, ref, 1e-6, bad, 1.0)
            s.pp_limit(ref) if flag == A.STAGE_LIMIT else s.apply_stabilization(ref)
            s.rk_stage_fused(0.0, U, got, flag, 1e-6, bad, 1.0)
            assert rel_err(got.cpu().numpy(), ref.cpu().numpy()) <= 1e-12


@pytest.mark.parametrize("cond", [False, True])
@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("p", [2, 4, 6, 8])
def test_implicit_form(p, curved, cond, cuda):
    cfg = _cfg(p, curved)
    U = random_state(cfg, 21, smooth=cond)
    if cond:
        cfg.cond_sys = 1
        U = cons_to_prim(cfg, U)
    Udot = np.random.default_rng(9).normal(size=U.size)
    ref = Oracle(cfg, threads=8).ifunction(0.1, U, Udot)
    with FRSolver(cfg) as s:
        Ud, out = torch.from_numpy(U).to(cuda), torch.empty(U.size, dtype=torch.float64, device=cuda)
        s.fun_implicit(0.1, Ud, torch.from_numpy(Udot).to(cuda), out)
        assert rel_err(out.cpu().numpy(), ref) <= TOL_FP64


@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("p", [1, 3, 5, 7, 9])
def test_columns_redone_with_the_checked_functions(p, curved, cuda):
    """Nodes of density 1e-40 (outside the fast reciprocal's range) and finite velocity and sound
    speed, in every kind of place: their columns are computed twice."""
    cfg = _cfg(p, curved)
    U = random_state(cfg, 17).reshape(-1, 4)
    pick = np.random.default_rng(p).random(len(U)) < 0.02
    U[pick] *= 1e-40 / U[pick, :1]
    U = U.reshape(-1)
    ref = Oracle(cfg, threads=8).residual(0.0, U)
    with FRSolver(cfg) as s:
        Ud = torch.from_numpy(U).to(cuda)
        R = torch.full_like(Ud, float("nan"))
        s.residual_kernel(0.0, Ud, R)
        assert s.status() == 0
    assert rel_err(R.cpu().numpy(), ref) <= TOL_FP64
