"""GPU: scratch vectors under the longest row window, a whole periodic mesh with a ghost row on
either side: the WENO post-step's copy of the state and the staging of host vectors."""
import pytest
import torch

from tests.helpers import random_state

from fr_sdg_b200 import FRSolver
from fr_sdg_b200 import _abi as A
from fr_sdg_b200.workloads import make_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [2, 4])
def test_whole_mesh_with_ghost_rows(p, cuda):
    nx, ny = 5, 6
    cfg = make_config(dim=2, p=p, n_elems=(nx, ny), riemann="hllc", apply_weno=True, threshold=0.3, pp_limit=True,
                      bcs={f: A.BC_PERIODIC for f in (A.LEFT, A.RIGHT, A.TOP, A.BOTTOM)})
    U = torch.from_numpy(random_state(cfg, 4)).to(cuda)
    row = U.numel() // ny
    with FRSolver(cfg) as s:
        want_post, want_rhs = U.clone(), torch.empty_like(U)
        s.apply_stabilization(want_post)
        s.rhs_func(0.0, U, want_rhs)
        s.set_row_window(-1, ny + 2, 1, ny + 1)
        W = torch.cat([U[-row:], U, U[:row]])
        host = torch.empty(W.numel(), dtype=torch.float64)
        s.rhs_func_host(0.0, W.cpu(), host)
        assert torch.equal(host[row:-row].to(cuda), want_rhs)
        s.apply_stabilization(W)
        assert torch.equal(W[row:-row], want_post)
