"""FP64 calls whose columns and rows differ in magnitude: each keeps the accuracy of FP64 FMAs."""
import numpy as np
import pytest

import cacg_gb300 as cg
from gpu_util import ptr

pytestmark = pytest.mark.gpu


def _qr(torch, V):
    n, k = V.shape
    Q, R = torch.empty_like(V), torch.empty(k, k, dtype=torch.float64, device="cuda")
    assert cg.lib().cacg_k_tsqr(n, k, ptr(V), k, ptr(Q), k, ptr(R), None) == 0
    return Q.cpu().numpy(), R.cpu().numpy()


@pytest.mark.parametrize("M", [1.0 + 2.0 ** -19, 1.5 - 2.0 ** -19, 1.2345678, 1.9999])
@pytest.mark.parametrize("top", [0, 5, 13, 19, 21])
def test_products_that_cancel_exactly(torch_cuda, M, top):
    """V = [1, M or M +- 1, third]: every product and sum of the QR is exact in FP64 (norms 32
    and 16, M of 20 bits), and Q's second column is exactly 0 where V's is M.  The third
    column's magnitude differs from row to row, so the digits of 1 and M lie at many offsets."""
    torch = torch_cuda
    M = round(M * 2 ** 19) / 2 ** 19
    r = np.arange(1024)
    d = np.where(r % 8 == 0, 1.0, np.where(r % 8 == 4, -1.0, 0.0))  # 128 of each
    # signs orthogonal to 1 and d, magnitudes alike over the rows they pair
    third = np.where((r >> 3) % 2 == 0, 1.0, -1.0) * 2.0 ** ((r >> 4) % (top + 1))
    V = np.stack([np.ones(1024), M + d, third], 1)
    Q, R = _qr(torch, torch.from_numpy(V).cuda())
    assert np.array_equal(R[:2, :2], [[32.0, 32.0 * M], [0.0, 16.0]])
    assert np.array_equal(Q[:, 1], d / 16.0)
    assert np.array_equal(Q[:, 0], np.full(1024, 2.0 ** -5))


@pytest.mark.parametrize("kind,N,m", [("lap2d", 600, 8), ("st3d27", 40, 8), ("lap3d7", 60, 9)])
def test_fixed_point_spmm_point_values(kind, N, m):
    """B - A X where one element of a column is far above the others (its neighbours zero, so
    that their rows of A X are exact): the others' rows keep the accuracy of FMAs, 35 u of
    27 |c| max|x| of a row; the root of the sum over n rows."""
    rp, ci, v = cg.gen_matrix(kind, N, 0.0625)
    n = len(rp) - 1
    assert len(v) * m >= 1e7
    rng = np.random.default_rng(3)
    X = np.clip(rng.standard_normal((n, m)), -5.5, 5.5)
    mid = n // 2 + N // 2
    rows = np.repeat(np.arange(n), np.diff(rp))
    near = np.zeros(n, bool)
    near[mid] = True
    for _ in range(2):  # two rings
        near[ci[near[rows]]] = True
    X[:, 2] *= 2.0 ** -50
    X[near, 2] = 0.0
    X[mid, 2] = 1.0
    AX = np.stack([np.add.reduceat(v.astype(np.longdouble) * X[ci, c], rp[:-1])
                   for c in range(m)], 1)
    B = AX.astype(np.float64)
    hit = ci[rp[mid]:rp[mid + 1]]
    assert np.array_equal(AX[hit, 2], B[hit, 2])
    _, info = cg.solve(rp, ci, v, B, X0=X, s=4, bounds=("given", 0.05, 60.0), tol=1e-8, maxit=0)
    got = info["true_relres"][2] * np.linalg.norm(B[:, 2])
    assert got <= 35 * 2.0 ** -53 * 2 * 27 * 5.5 * 2.0 ** -50 * n ** 0.5
