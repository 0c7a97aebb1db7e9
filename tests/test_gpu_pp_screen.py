"""GPU: the 1D positivity limiter at pressures within rounding of its floor.  The nodes of
every element it leaves stand at or above the floor in its own arithmetic (quotients), which
plain numpy repeats bit for bit for an ideal gas: no product there can be contracted."""
import numpy as np
import pytest
import torch

from fr_sdg_b200 import FRSolver
from fr_sdg_b200 import _abi as A
from fr_sdg_b200.workloads import make_config

pytestmark = pytest.mark.gpu

EPS = 1e-13
G1 = np.float64(1.4) - 1.0


def _pressure(rho, m, E):
    return (G1 * rho) * ((E - 0.5 * (m * m) / rho) / rho)


@pytest.mark.parametrize("entry", ["pp_limit", "stage"])
@pytest.mark.parametrize("p", [1, 3, 6])
def test_nodes_stand_at_the_floor(p, entry, cuda):
    n, ne = p + 1, 8000
    cfg = make_config(dim=1, p=p, n_elems=(ne, 1), riemann="rusanov", pp_limit=True, pp_eps=EPS,
                      bcs={A.LEFT: A.BC_OUTFLOW, A.RIGHT: A.BC_OUTFLOW})
    rng = np.random.default_rng(p)
    # deviations of 1e-5 leave averages at pressures near 1e-10; the first node's lies within a
    # few roundings of the floor, the others' well above it
    rho = rng.uniform(0.6, 1.7, (ne, 1)) * (1.0 + 1e-5 * rng.uniform(-1, 1, (ne, n)))
    m = rng.uniform(0.5, 1.5, (ne, 1)) * (1.0 + 1e-5 * rng.uniform(-1, 1, (ne, n)))
    E = 0.5 * m * m / rho + 1e-12 / G1
    E[:, 0] = 0.5 * m[:, 0] ** 2 / rho[:, 0] + EPS / G1
    E[:, 0] += rng.integers(-2, 3, ne) * np.spacing(E[:, 0])
    U = np.stack([rho, m, E], axis=1)
    before = _pressure(rho, m, E)[:, 0]
    assert (before < EPS).sum() > ne // 10 and (before >= EPS).sum() > ne // 10
    with FRSolver(cfg) as s:
        X = torch.from_numpy(U.reshape(-1)).to(cuda)
        if entry == "pp_limit":
            s.pp_limit(X)
            out = X
        else:
            out = torch.empty_like(X)
            s.rk_stage_fused(0.0, X, out, A.STAGE_LIMIT, 0.0, X.clone(), 1.0)
        V = out.cpu().numpy().reshape(ne, 3, n)
    assert (_pressure(V[:, 0], V[:, 1], V[:, 2]) >= EPS).all()
