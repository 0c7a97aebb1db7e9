"""GPU: one Arnoldi step of frsdg_gmres_arnoldi against a restatement of it (classical
Gram-Schmidt, the second pass when the first leaves ||w||^2 below half its value, Givens
rotations), at sizes around the kernels' chunks of 512 and 2048 entries."""
import numpy as np
import pytest
import torch

from fr_sdg_b200 import _abi as A

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("near", [False, True])  # w nearly in the span of V: the second pass acts
@pytest.mark.parametrize("n,j", [(1, 0), (2, 0), (511, 0), (513, 6), (2047, 3), (2049, 9), (5000, 31), (4096, 255)])
def test_arnoldi_step(n, j, near, cuda):
    rng = np.random.default_rng(n + j)
    V = np.linalg.qr(rng.normal(size=(n, j + 1)))[0].T.copy()
    w = rng.normal(size=n)
    if near:
        w = V.T @ rng.normal(size=j + 1) + 1e-3 * w
    else:  # orthogonal to the span but for a little: one pass
        w = w - V.T @ (V @ w) + 1e-2 * (V.T @ rng.normal(size=j + 1))
    if n == j + 1:
        w = np.abs(w) + 1.0
    ldh, ldv = j + 2, n + 3
    ang = rng.uniform(0, 6, j)
    cs, sn, g = np.cos(ang), np.sin(ang), rng.normal(size=j + 1)
    # the restatement
    h = V @ w
    r = w - V.T @ h
    second = r @ r < 0.5 * (w @ w)
    if n > j + 1:
        assert second == near
    if second:
        h2 = V @ r
        h, r = h + h2, r - V.T @ h2
    hn = np.linalg.norm(r)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    Vd = torch.full((j + 1, ldv), float("nan"), dtype=torch.float64, device=cuda)
    Vd[:, :n] = d(V)
    wd, H = d(w), torch.full((j + 2, ldh), 7.0, dtype=torch.float64, device=cuda)
    c_, s_, g_ = (torch.zeros(j + 2, dtype=torch.float64, device=cuda) for _ in range(3))
    c_[:j], s_[:j], g_[:j + 1] = d(cs), d(sn), d(g)
    inv = torch.zeros(1, dtype=torch.float64, device=cuda)
    work = torch.empty(int(A.lib().frsdg_gmres_work_doubles(n)), dtype=torch.float64, device=cuda)
    A.check(A.lib().frsdg_gmres_arnoldi(Vd.data_ptr(), ldv, j, wd.data_ptr(), n, H.data_ptr(), ldh, c_.data_ptr(),
                                        s_.data_ptr(), g_.data_ptr(), inv.data_ptr(), work.data_ptr(), None), "arnoldi")
    torch.cuda.synchronize()
    H, got, c_, s_, g_ = (t.cpu().numpy() for t in (H, wd, c_, s_, g_))
    # each dot product of n terms is within n u of exact relative to ||v|| ||w||, in both
    tol = 4.0 * (n + j + 8) * U * np.linalg.norm(w) * np.sqrt(j + 1.0)
    assert np.abs(got - r).max() <= tol
    assert np.array_equal(H[:, :j], np.full((j + 2, j), 7.0))  # other columns stay
    # undo the rotations of the column: h and ||w||, then its last entry is 0
    col = H[:, j].copy()
    assert col[j + 1] == 0.0
    a, b = c_[j] * col[j], s_[j] * col[j]
    col[j], last = a, b
    for i in range(j - 1, -1, -1):
        x, y = col[i], col[i + 1]
        col[i], col[i + 1] = cs[i] * x - sn[i] * y, sn[i] * x + cs[i] * y
    assert np.abs(col[:j + 1] - h).max() <= 2.0 * tol and abs(last - hn) <= 2.0 * tol
    assert abs(c_[j] ** 2 + s_[j] ** 2 - 1.0) <= 8 * U
    assert abs(g_[j] - c_[j] * g[j]) <= 4 * U * abs(g[j]) and abs(g_[j + 1] + s_[j] * g[j]) <= 4 * U * abs(g[j])
    if n > j + 1:
        assert abs(float(inv[0]) * np.linalg.norm(got) - 1.0) <= 4.0 * n * U + 1e-12
        if second:
            assert np.abs(V @ got).max() <= tol
