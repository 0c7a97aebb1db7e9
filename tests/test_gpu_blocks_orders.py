"""GPU: the element blocks of the Jacobian at orders 6 to 9 (blocks of 196 to 400 DOFs, past the
preconditioner's range), complex and first-order steps: columns against the oracle's
single-seed products."""
import numpy as np
import pytest
import torch

from oracle.oracle import Oracle
from tests.helpers import TOL_JVP, random_state, rel_err

from fr_sdg_b200 import FRSolver
from fr_sdg_b200 import _abi as A
from fr_sdg_b200.workloads import make_config

pytestmark = pytest.mark.gpu

NX, NY = 4, 3


@pytest.mark.parametrize("h", [1e-30, 1e-7])
@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("p", [6, 7, 8, 9])
def test_columns_match_oracle(p, curved, h, cuda):
    kw = dict(geometry=A.GEOM_SINE_WARP, geom_params=(0.05, 0, 0, 0)) if curved else {}
    cfg = make_config(dim=2, p=p, n_elems=(NX, NY), box=(1.0, 0.8), riemann="hllc" if p % 2 else "rusanov", csd_eps=h,
                      gas="vdw" if p > 7 else "ideal", vdw=(0.05, 0.02),
                      bcs={A.LEFT: A.BC_OUTFLOW, A.RIGHT: A.BC_WALL, A.BOTTOM: A.BC_WALL, A.TOP: A.BC_OUTFLOW}, **kw)
    nd, ne = 4 * (p + 1) ** 2, NX * NY
    U = random_state(cfg, 3, amp=0.2)
    with FRSolver(cfg) as s:
        Ud = torch.from_numpy(U).to(cuda)
        B5 = torch.full((ne * 5 * nd * nd,), float("nan"), dtype=torch.float64, device=cuda)
        B1 = torch.full((ne * nd * nd,), float("nan"), dtype=torch.float64, device=cuda)
        s.jac_blocks5(0.1, 2.0, Ud, B5)
        s.jac_blocks(0.1, 2.0, Ud, B1)
    B5, B1 = B5.view(ne, 5, nd, nd).cpu().numpy(), B1.view(ne, nd, nd).cpu().numpy()
    assert np.array_equal(B5[:, 0], B1)
    o = Oracle(cfg, threads=8)
    rng = np.random.default_rng(p)
    n = p + 1
    corners = [0, 4 * (n - 1) + 1, 4 * n * (n - 1) + 2, nd - 1]  # face nodes, each variable
    for e in range(ne):
        i, j = e % NX, e // NX
        for c in (corners[e % 4], 4 * (e % n) + 3, 4 * n * (e % n) + 1, int(rng.integers(nd))):
            V = np.zeros(U.size)
            V[e * nd + c] = 1.0
            ref = o.jvp(0.1, 2.0, U, V).reshape(ne, nd)
            got = np.zeros_like(ref)
            # row element f, slot of the seeded element e in f's neighbourhood
            for f, slot in ((e, 0), (e - 1 if i > 0 else -1, 1), (e - NX, 2), (e + NX, 3), (e + 1 if i < NX - 1 else -1, 4)):
                if 0 <= f < ne:
                    got[f] = B5[f, slot, c]
            assert rel_err(got, ref) <= TOL_JVP
