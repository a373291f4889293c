"""FP32-block kernels of the mixed mode at the edges of their tiles: the X/R update by
tiles and the tensor-core Gram, against FP64 sums of the same FP32 inputs."""
import numpy as np
import pytest

import cacg_gb300 as cg
from gpu_util import ptr

pytestmark = pytest.mark.gpu

F32, GRAM_TC5 = 1, 5


def _randn(torch, n, k, seed, dtype=None):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n, k, dtype=dtype or torch.float32, device="cuda", generator=g)


@pytest.mark.parametrize("n", [1, 84, 85, 86, 4097])
@pytest.mark.parametrize("k,m", [(4, 1), (8, 1), (44, 11), (24, 6), (64, 3), (36, 9), (40, 20),
                                 (200, 7), (256, 5)])
def test_xrupdate_tiles(torch_cuda, n, k, m):
    """k FP32 fused multiply-adds a product and alpha rounded to FP32: at most (k + 1) 2^-24 of
    |Q| |alpha|; X, R and the norms are FP64 (rows of tile: 256 / ceil(m / 4))."""
    torch = torch_cuda
    Q, AQ = _randn(torch, n, k, 1), _randn(torch, n, k, 2)
    al, X, R = (_randn(torch, a, m, 3 + i, torch.float64) for i, a in enumerate((k, n, n)))
    S0 = torch.full((n, k), 7.0, device="cuda")
    nr = torch.zeros(m, dtype=torch.float64, device="cuda")
    Xn, Rn = X.clone(), R.clone()
    rc = cg.lib().cacg_k_xrupdate(F32, n, k, m, ptr(Q), ptr(AQ), k, ptr(al), ptr(Xn), ptr(Rn),
                                  ptr(S0), k, ptr(nr), None)
    torch.cuda.synchronize()
    assert rc == 0
    for old, new, B, sign in ((X, Xn, Q, 1.0), (R, Rn, AQ, -1.0)):
        ref = old + sign * (B.double() @ al)
        bound = (k + 2) * 2.0 ** -24 * (B.double().abs() @ al.abs()) + 2.0 ** -50 * old.abs()
        assert bool(((new - ref).abs() <= bound).all())
    assert torch.equal(S0[:, :m], Rn.float()) and bool((S0[:, m:] == 7.0).all())
    ref = (Rn * Rn).sum(0)
    assert bool(((nr - ref).abs() <= (n + 2) * 2.0 ** -53 * ref).all())


@pytest.mark.parametrize("n", [1, 31, 33, 64, 95, 5000, 152 * 96 + 7, 60001])
@pytest.mark.parametrize("ka,kb1,kb2", [(8, 8, 1), (24, 24, 6), (44, 44, 11), (64, 64, 0),
                                        (80, 80, 16), (96, 96, 16), (112, 112, 0), (128, 120, 8),
                                        (128, 128, 16), (140, 136, 30)])
def test_gram_tc5_tiles(torch_cuda, n, ka, kb1, kb2):
    """Groups of 64 rows x 6 slice products accumulate in FP32 (at most 384 additions, each within
    2^-23 of the running sum), the groups' sums about 2^-44: 2^-14 of |L|^T |R| covers every
    output.  Three runs give the same bits (the ring, buffers and barriers have no race)."""
    torch = torch_cuda
    L, R1 = _randn(torch, n, ka, 1), _randn(torch, n, kb1, 2)
    ld2 = (kb2 + 3) // 4 * 4
    R2 = _randn(torch, n, max(ld2, 4), 3)
    R = torch.cat([R1, R2[:, :kb2]], 1).double()
    out = []
    for _ in range(3):
        C = torch.full((ka, kb1 + kb2), 7.0, dtype=torch.float64, device="cuda")
        rc = cg.lib().cacg_k_gram(F32, GRAM_TC5, n, ptr(L), ka, ka, ptr(R1), kb1, kb1,
                                  ptr(R2) if kb2 else None, max(ld2, 4), kb2, ptr(C), kb1 + kb2,
                                  None)
        torch.cuda.synchronize()
        assert rc == 0
        out.append(C)
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
    ref, bound = L.double().T @ R, L.double().abs().T @ R.abs()
    assert bool(((out[0] - ref).abs() <= 2.0 ** -14 * bound).all())


@pytest.mark.parametrize("kind,N,shift", [("st3d27", 58, 0.1), ("st3d27", 61, 0.0),
                                          ("lap2d", 1003, 0.05)])
def test_staged_spmm_one_value(torch_cuda, kind, N, shift):
    """Constant-coefficient stencils at sizes that read presence bits instead of the DIA values:
    the unstaged kernel reads the values, with the same FMAs in the same order."""
    rp, ci, v = cg.gen_matrix(kind, N, shift)
    n = len(rp) - 1
    assert {"st3d27": 27, "lap2d": 5}[kind] * n >= 5e6  # the branch's range
    B = cg.gen_rhs("normal", n, 16, 5)
    X = [cg.solve(rp, ci, v, B, s=3, bounds="gerschgorin", tol=1e-8, maxit=4, precision="mixed",
                  spmm_format=f)[0] for f in ("auto", "dia_unstaged")]
    assert np.all(np.isfinite(X[0])) and np.array_equal(X[0], X[1])
