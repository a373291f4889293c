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


def _stencil(kind, N, shift, m, seed=7):
    rp, ci, v = cg.gen_matrix(kind, N, shift)
    return rp, ci, v, cg.gen_rhs("normal", len(rp) - 1, m, seed)


def _relres(rp, ci, v, B, X):
    AX = np.stack([np.add.reduceat(v.astype(np.longdouble) * X[ci, c], rp[:-1])
                   for c in range(X.shape[1])], 1)
    return (np.sqrt(((B - AX) ** 2).sum(0)) / np.linalg.norm(B, axis=0)).astype(np.float64)


# exponents of the right-hand sides' scales, column 0 the smallest
SPREADS = [(0, 46, 10, 30), (0, 27, 33, 40), (-300, 100, 0, 200)]


@pytest.mark.parametrize("kind,N,m,s", [("lap2d", 256, 4, 4), ("lap3d7", 40, 8, 4)])
@pytest.mark.parametrize("spread", SPREADS)
def test_solve_columns_of_different_magnitude(kind, N, m, s, spread):
    """The block iteration is equivariant under a scale per right-hand side, exactly so for
    powers of two: X is the unscaled call's X scaled, bit for bit, in as many iterations."""
    rp, ci, v, B = _stencil(kind, N, 0.05, m)
    n = len(rp) - 1
    assert n * (s * m) ** 2 >= 2e6 and n * s * m * m >= 4e6  # the digit-plane updates' range
    d = 2.0 ** np.resize(spread, m).astype(np.float64)
    kw = dict(s=s, bounds="gerschgorin", tol=1e-9, maxit=300)
    X1, i1 = cg.solve(rp, ci, v, B, **kw)
    X2, i2 = cg.solve(rp, ci, v, B * d, **kw)
    assert i1["status"] == 0 and i2["status"] == 0
    assert i1["iterations"] == i2["iterations"]
    assert np.array_equal(X2, X1 * d)


@pytest.mark.parametrize("kind,N,m,s", [("lap2d", 256, 4, 4), ("lap3d7", 40, 8, 4)])
@pytest.mark.parametrize("spread", SPREADS)
def test_drop_in_columns_of_different_magnitude(kind, N, m, s, spread):
    """The reference's stop rule looks at column 0's recurrence alone: the true residual of
    every column has to agree with it (here: of column 0, the one the rule promises)."""
    rp, ci, v, B = _stencil(kind, N, 0.05, m)
    d = 2.0 ** np.resize(spread, m).astype(np.float64)
    eps = 1e-8 * float(np.linalg.norm(B[:, 0]))
    out = []
    for scale in (np.ones(m), d / d[0]):
        X = np.zeros_like(B)
        Bs = B * scale
        cg.bcbcg_v1(rp.astype(np.int64), ci.astype(np.int64), v, Bs, X, s, eps)
        assert cg.last_status() == 0
        out.append((X / scale, cg.last_iterations()))
        assert _relres(rp, ci, v, Bs, X)[0] <= 1.01e-8
    assert out[0][1] == out[1][1]
    assert np.array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("kind,N,m,s", [("lap2d", 400, 8, 4), ("lap3d7", 64, 8, 8)])
def test_solve_point_sources(kind, N, m, s):
    """Right-hand sides with one nonzero, alone and beside normal ones: columns whose elements
    fall off over hundreds of orders of magnitude.  The FMA variant's iterations and residual."""
    rp, ci, v, B = _stencil(kind, N, 0.5, m)
    n = len(rp) - 1
    assert n * (s * m) ** 2 >= 2e6 and n * s * m * m >= 4e6
    for point in (range(m), range(0, m, 2)):
        Bp = B.copy()
        for c in point:
            Bp[:, c] = 0.0
            Bp[(n // 2 + 977 * c) % n, c] = 1.0
        kw = dict(s=s, bounds="gerschgorin", tol=1e-11, maxit=200)
        X1, i1 = cg.solve(rp, ci, v, Bp, **kw)
        X2, i2 = cg.solve(rp, ci, v, Bp, gram="fma", **kw)
        assert i1["status"] == 0 and i2["status"] == 0
        assert abs(i1["iterations"] - i2["iterations"]) <= 1
        assert _relres(rp, ci, v, Bp, X1).max() <= 1.01e-11


@pytest.mark.parametrize("n,k", [(20000, 16), (20000, 2), (6000, 96), (3000, 128), (257, 5)])
@pytest.mark.parametrize("lo,hi", [(0, -7), (-7, 0), (-30, 30), (40, -40)])
def test_qr_columns_of_different_magnitude(torch_cuda, n, k, lo, hi):
    """QR of a block whose columns have magnitudes 10^lo .. 10^hi: CholeskyQR is equivariant
    under a scale per column, and so each *column* of Q R - V stays at rounding: a chain of k
    FMAs and the two passes, 100 k u of the column, u = 2^-53."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(3)
    V = torch.randn(n, k, dtype=torch.float64, device="cuda", generator=g)
    V *= 10.0 ** torch.linspace(lo, hi, k, device="cuda", dtype=torch.float64)
    Q, R = _qr(torch, V)
    v, u = V.cpu().numpy(), 100 * k * 2.0 ** -53
    E = (Q.astype(np.longdouble) @ R.astype(np.longdouble) - v).astype(np.float64)
    norm = np.linalg.norm(v, axis=0)
    assert np.all(np.linalg.norm(E / norm, axis=0) <= u)
    assert np.linalg.norm(Q.T @ Q - np.eye(k)) <= u * k ** 0.5


@pytest.mark.parametrize("n", [1000, 20000])
def test_qr_one_column_in_one_row(torch_cuda, n):
    """A column whose weight lies in one row beside spread ones: magnitudes by norm, not by the
    largest element."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(4)
    V = torch.randn(n, 24, dtype=torch.float64, device="cuda", generator=g)
    V[:, 7] *= 1e-9
    V[n // 3, 7] = 1.0
    Q, R = _qr(torch, V)
    v, u = V.cpu().numpy(), 100 * 24 * 2.0 ** -53
    E = (Q.astype(np.longdouble) @ R.astype(np.longdouble) - v).astype(np.float64)
    assert np.all(np.linalg.norm(E, axis=0) <= u * np.linalg.norm(v, axis=0))


def _gram(torch, L, R, variant=0):
    C = torch.empty(L.shape[1], R.shape[1], dtype=torch.float64, device="cuda")
    assert cg.lib().cacg_k_gram(0, variant, L.shape[0], ptr(L), L.shape[1], L.shape[1], ptr(R),
                                R.shape[1], R.shape[1], None, 0, 0, ptr(C), R.shape[1],
                                None) == 0
    return C.cpu().numpy()


@pytest.mark.parametrize("n,ka,kb", [(300, 20, 24), (2000, 24, 24), (5000, 96, 112),
                                     (40000, 17, 33), (3000, 130, 70)])
@pytest.mark.parametrize("kind", ["rows", "spikes", "tails", "zeros", "huge"])
def test_gram_rows_of_different_magnitude(torch_cuda, n, ka, kb, kind):
    """L^T R with rows of L and R graded against each other, with single large elements in
    different rows, with decaying columns: within n u of |L|^T |R| (n FMAs), u = 2^-53."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(8)
    L = torch.randn(n, ka, dtype=torch.float64, device="cuda", generator=g)
    R = torch.randn(n, kb, dtype=torch.float64, device="cuda", generator=g)
    if kind == "rows":
        d = 10.0 ** (torch.rand(n, 1, dtype=torch.float64, device="cuda", generator=g) * 12 - 6)
        L, R = L * d, R / d
    elif kind == "spikes":  # one large element a column, never in a row that both have
        L, R = L.sign(), R.sign()
        i = torch.arange(ka, device="cuda")
        L[2 * i % n, i] = 2.0 ** 60
        R[2 * i % n, :] = 0.0
        j = torch.arange(kb, device="cuda")
        R[(2 * j + 1) % n, j] = 2.0 ** 60
        L[(2 * j + 1) % n, :] = 0.0
    elif kind == "tails":  # a column's weight near its own row
        r = torch.arange(n, device="cuda", dtype=torch.float64)[:, None]
        at = torch.linspace(0, n - 1, ka, device="cuda", dtype=torch.float64)
        L = L * torch.exp(-40.0 * (r - at).abs() / n)
        at = torch.linspace(n - 1, 0, kb, device="cuda", dtype=torch.float64)
        R = R * torch.exp(-40.0 * (r - at).abs() / n)
    elif kind == "zeros":  # three rows in four are zero in one or the other
        r = torch.arange(n, device="cuda")
        L = L * 10.0 ** (-9.0 * (r % 4 == 0))[:, None]
        L[r % 4 == 1] = 0.0
        R[r % 4 >= 2] = 0.0
        R = R * 10.0 ** (-9.0 * (r % 4 == 1))[:, None]
    else:
        L = L * 1e300
        L[::7] = L[::7] * 1e-290
        R = R * 1e-300
        R[::7] = R[::7] * 1e290
    C = _gram(torch, L, R)
    l, r = L.cpu().numpy().astype(np.longdouble), R.cpu().numpy().astype(np.longdouble)
    ref, mag = np.zeros((ka, kb), np.longdouble), np.zeros((ka, kb), np.longdouble)
    for a in range(ka):
        ref[a] = l[:, a] @ r
        mag[a] = np.abs(l[:, a]) @ np.abs(r)
    assert np.all(np.abs(C - ref) <= n * 2.0 ** -53 * mag)


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
