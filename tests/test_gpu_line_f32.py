"""GPU: FP32 residuals do not depend on where tiles cut the mesh, nodes included whose
reciprocals or roots leave the fast range (their neighbours keep the fast form in every tile)."""
import pytest
import torch

from tests.helpers import random_state

from fr_sdg_b200 import FRSolver
from fr_sdg_b200 import _abi as A
from fr_sdg_b200.workloads import make_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gas", ["ideal", "vdw"])
@pytest.mark.parametrize("p", [2, 3, 5, 7])
def test_row_window_equals_the_whole_mesh(p, gas, cuda):
    n, nx, ny = p + 1, 9, 23
    cfg = make_config(dim=2, p=p, n_elems=(nx, ny), box=(1.0, 2.0), riemann="hllc", gas=gas, vdw=(0.05, 0.02),
                      bcs={f: A.BC_OUTFLOW for f in (A.LEFT, A.RIGHT, A.TOP, A.BOTTOM)})
    U = torch.from_numpy(random_state(cfg, 40 + p)).to(cuda).float().view(ny, nx, n, n, 4)
    # a node off the elements' faces with kinetic above total energy: its root is not real, its
    # column's boundary nodes are ordinary
    U[::2, ::2, 1, 1, 1] = 4.0
    U = U.reshape(ny, -1)
    with FRSolver(cfg) as s:
        R = torch.empty_like(U).view(-1)
        s.residual_kernel_f32(0.0, U.view(-1), R)
        assert bool(torch.isfinite(R).all())
        R = R.view(ny, -1)
        for base, rows in ((0, 7), (3, 12), (6, 9), (11, 12)):
            begin, end = (1 if base else 0), (rows if base + rows == ny else rows - 1)
            s.set_row_window(base, rows, begin, end)
            W = U[base:base + rows].reshape(-1)
            Q = torch.full_like(W, float("nan"))
            s.residual_kernel_f32(0.0, W, Q)
            assert torch.equal(Q.view(rows, -1)[begin:end], R[base + begin:base + end])
