"""GPU: FP32 residuals do not depend on where tiles cut the mesh, also beside nodes whose
reciprocals or roots leave the fast range: their neighbours keep the fast form in every tile."""
import pytest
import torch

from tests.helpers import random_state

from fr_sdg_b200 import FRSolver
from fr_sdg_b200 import _abi as A
from fr_sdg_b200.workloads import make_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op,exponents", [(4, (-125, -100, 0, 37, 123)), (5, (-125, -112, -101, -100, -99, 0, 1, 38, 123))])
def test_fast_forms_equal_ieee(op, exponents, cuda):
    """Every mantissa (and either parity of the root's exponent): the fast FP32 reciprocal and root
    are the correctly rounded ones, so a redo with the IEEE operations leaves the same bits.  FP64
    rounded to FP32 is correctly rounded for both (53 >= 2 * 24 + 2)."""
    for e in exponents:
        x = ((1.0 + torch.arange(2 ** 23, dtype=torch.float64) * 2.0 ** -23) * 2.0 ** e).to(cuda)
        y = torch.empty_like(x)
        A.check(A.lib().frsdg_device_math(op, x.data_ptr(), y.data_ptr(), x.numel(), None), "frsdg_device_math")
        torch.cuda.synchronize()
        assert torch.equal(y.float(), (1.0 / x if op == 4 else torch.sqrt(x)).float())


@pytest.mark.parametrize("nx", [21, 600])  # both tile forms
@pytest.mark.parametrize("p", [2, 3, 5, 7])
def test_row_window_equals_the_whole_mesh(p, nx, cuda):
    n, ny = p + 1, 46
    cfg = make_config(dim=2, p=p, n_elems=(nx, ny), box=(1.0, 2.0), riemann="hllc",
                      bcs={f: A.BC_OUTFLOW for f in (A.LEFT, A.RIGHT, A.TOP, A.BOTTOM)})
    U = torch.from_numpy(random_state(cfg, 40 + p, amp=0.2)).to(cuda).float().view(ny, nx, n, n, 4)
    # nodes off the faces with kinetic above total energy in every second row: their roots are
    # not real, and their columns, ordinary boundary nodes among them, are computed twice
    U[::2, :, 1, 1:n - 1, 1] = 4.0
    U = U.reshape(ny, -1)
    with FRSolver(cfg) as s:
        R = torch.empty_like(U).view(-1)
        s.residual_kernel_f32(0.0, U.view(-1), R)
        assert bool(torch.isfinite(R).all())
        R = R.view(ny, -1)
        for base, rows in ((0, 7), (1, 9), (4, 12), (5, 39), (10, 36)):
            begin, end = (1 if base else 0), (rows if base + rows == ny else rows - 1)
            s.set_row_window(base, rows, begin, end)
            W = U[base:base + rows].reshape(-1)
            Q = torch.full_like(W, float("nan"))
            s.residual_kernel_f32(0.0, W, Q)
            assert torch.equal(Q.view(rows, -1)[begin:end], R[base + begin:base + end])
