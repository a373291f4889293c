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
