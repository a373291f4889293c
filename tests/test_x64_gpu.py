"""FP64 products from fp16 digit planes (k_gram_x64.cu, k_tsm_x64.cu) against extended-precision sums.

Bound of an output: with M_i the largest magnitude of column i, a digit value is within
2^-55 M of its element, and the dropped plane products are below 2^-51 M_i M_j a row
(6 products of two digits of at most 2^7, 2^16 below the lowest kept weight's 2^48 unit,
against M_i M_j of at least 2^108); the chunk sums are FP64.  2^-50 M_i M_j a row covers
all of it.
"""
import numpy as np
import pytest

import cacg_gb300 as cg
import oracle as O
from gpu_util import ptr

pytestmark = pytest.mark.gpu


def _block(torch, n, k, ld, off, kind, seed):
    """An n x k view with row stride ld, off doubles into its allocation."""
    base = torch.zeros(n * ld + off + 2, dtype=torch.float64, device="cuda")
    v = torch.as_strided(base, (n, k), (ld, 1), off)
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(n, k, dtype=torch.float64, device="cuda", generator=g)
    if kind == "scaled":  # columns of very different magnitude, one of them zero
        x *= 10.0 ** torch.linspace(-120, 90, k, device="cuda", dtype=torch.float64)
        x[:, k // 2] = 0.0
    elif kind == "spike":
        x *= 1e-9
        x[n // 3] = -3.0
    elif kind == "edge":  # the largest significand at the top of every scale
        x = torch.full_like(x, -(2.0 - 2.0 ** -52))
    v.copy_(x)
    return v


def _gram(torch, L, R1, R2, variant=0):
    ka, kb1, kb2 = L.shape[1], R1.shape[1], 0 if R2 is None else R2.shape[1]
    C = torch.full((ka, kb1 + kb2), 7.0, dtype=torch.float64, device="cuda")
    rc = cg.lib().cacg_k_gram(0, variant, L.shape[0], ptr(L), L.stride(0), ka, ptr(R1),
                              R1.stride(0), kb1, ptr(R2), R2.stride(0) if kb2 else 0, kb2, ptr(C),
                              kb1 + kb2, None)
    assert rc == 0
    return C.cpu().numpy()


@pytest.mark.parametrize("n,ka,kb1,kb2", [
    (256, 8, 8, 1), (257, 9, 9, 3), (1000, 20, 20, 5), (2049, 64, 64, 8), (700, 96, 96, 16),
    (300, 128, 129, 0), (333, 129, 64, 7), (260, 256, 48, 16), (152 * 64 + 1, 12, 17, 0),
    (152 * 128 + 33, 8, 16, 0)])
@pytest.mark.parametrize("kind", ["normal", "scaled", "spike", "edge"])
@pytest.mark.parametrize("pad,off", [(0, 0), (3, 1)])
def test_gram_fp64_planes(n, ka, kb1, kb2, kind, pad, off):
    torch = pytest.importorskip("torch")
    L = _block(torch, n, ka, ka + pad, off, kind, 1)
    R1 = _block(torch, n, kb1, kb1 + pad, off, kind, 2)
    R2 = _block(torch, n, kb2, kb2 + pad, off, kind, 3) if kb2 else None
    C = _gram(torch, L, R1, R2)
    l = L.cpu().numpy().astype(np.longdouble)
    r = (R1 if R2 is None else torch.cat([R1, R2], 1)).cpu().numpy().astype(np.longdouble)
    tol = n * 2.0 ** -50 * np.abs(l).max(0)[:, None] * np.abs(r).max(0)[None, :]
    assert np.all(np.abs(C - l.T @ r) <= tol)


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("n,ka,kb1,kb2", [(7, 1, 1, 0), (1000, 4, 4, 1), (31, 5, 5, 3),
                                          (40000, 8, 8, 2), (700, 16, 16, 0), (1, 3, 9, 7),
                                          (3000, 16, 1, 15), (100, 17, 8, 0), (333, 24, 24, 6),
                                          (5000, 24, 32, 0), (700, 25, 31, 0), (90, 48, 32, 0),
                                          (2500, 49, 32, 0), (257, 96, 8, 8)])
def test_gram_fp64_few_outputs(n, ka, kb1, kb2, variant):
    """The FMA Gram around the output counts (768, 1536) where its thread layout changes, and
    the automatic variant's kernel for at most 16 columns a side: a chain of at most n FMAs
    and the partial sums (the planes' bound, taken past 16 columns, is test_gram_fp64_planes')."""
    torch = pytest.importorskip("torch")
    L = _block(torch, n, ka, ka, 0, "normal", 1)
    R1 = _block(torch, n, kb1, kb1 + 1, 1, "normal", 2)
    R2 = _block(torch, n, kb2, kb2, 0, "normal", 3) if kb2 else None
    if variant == 0 and (max(ka, kb1 + kb2) > 16 or n * ka * (kb1 + kb2) > 3e6 and ka * kb1 > 80):
        pytest.skip("not this kernel's shape")
    C = _gram(torch, L, R1, R2, variant)
    l = L.cpu().numpy().astype(np.longdouble)
    r = (R1 if R2 is None else torch.cat([R1, R2], 1)).cpu().numpy().astype(np.longdouble)
    assert np.all(np.abs(C - l.T @ r) <= (n + 40) * 2.0 ** -53 * (np.abs(l).T @ np.abs(r)))


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 4e-310])
def test_gram_fp64_planes_outside_range(value):
    """Values no scale holds: the reduction forms the product by FP64 FMAs."""
    torch = pytest.importorskip("torch")
    L = _block(torch, 1500, 24, 24, 0, "normal", 4)
    R = _block(torch, 1500, 24, 24, 0, "normal", 5)
    if np.isfinite(value):
        L[:, 3] = value
        R *= 1e200
    else:
        L[700, 3] = value
        R[900, 5] = value
    with np.errstate(all="ignore"):
        got, ref = _gram(torch, L, R, None), _gram(torch, L, R, None, variant=1)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    fin = np.isfinite(ref)
    assert np.array_equal(got[~fin & ~np.isnan(ref)], ref[~fin & ~np.isnan(ref)])
    # two FP64 sums of 1500 products in different orders
    scale = np.abs(L.cpu().numpy()).T @ np.abs(R.cpu().numpy())
    ok = fin & np.isfinite(scale)
    assert np.all(np.abs(got - ref)[ok] <= 2 * 1500 * 2.0 ** -53 * scale[ok])


def _qr(torch, V):
    n, k = V.shape
    Q = torch.empty(n, k, dtype=torch.float64, device="cuda")
    R = torch.empty(k, k, dtype=torch.float64, device="cuda")
    assert cg.lib().cacg_k_tsqr(n, k, ptr(V), V.stride(0), ptr(Q), k, ptr(R), None) == 0
    return Q.cpu().numpy(), R.cpu().numpy()


@pytest.mark.parametrize("n,k", [(256, 1), (300, 16), (129, 17), (1000, 31), (152 * 128 + 5, 33),
                                 (400, 64), (513, 65), (2000, 96), (700, 113), (640, 128)])
@pytest.mark.parametrize("pad,off", [(0, 0), (3, 1)])
def test_tall_small_product_in_qr(n, k, pad, off):
    """Y = A W at tile edges, through the QR: Q R = V and Q^T Q = I.  A product's error is
    below 2^-50 of its row's and column's largest magnitudes a term; two passes, k terms."""
    torch = pytest.importorskip("torch")
    V = _block(torch, n, k, k + pad, off, "normal", 6)
    V[:, :] *= 10.0 ** torch.linspace(-3, 3, n, device="cuda", dtype=torch.float64)[:, None]
    Q, R = _qr(torch, V)
    v = V.cpu().numpy()
    assert np.max(np.abs(Q.T @ Q - np.eye(k))) <= 4 * k * 2.0 ** -50
    assert np.linalg.norm(Q @ R - v) <= 4 * k * 2.0 ** -50 * np.linalg.norm(v)
    # rows of small magnitude keep their own relative accuracy (a scale per row)
    row = np.linalg.norm(Q @ R - v, axis=1) / np.linalg.norm(v, axis=1)
    cond = np.linalg.cond(R)
    assert np.max(row) <= 4 * k * 2.0 ** -50 * cond


@pytest.mark.parametrize("kind,N,m,s", [("lap2d", 24, 1, 2), ("lap3d7", 9, 3, 5),
                                        ("lap2d", 37, 5, 4), ("lap3d7", 17, 16, 4),
                                        ("lap2d", 40, 17, 3), ("lap3d7", 15, 32, 4),
                                        ("lap3d7", 16, 36, 4), ("lap2d", 45, 37, 2),
                                        ("lap3d7", 15, 12, 8)])
def test_solves_with_plane_products(kind, N, m, s):
    """Gram, Q and X / R updates together at the widths and row counts where their tiles end,
    against the oracle: the contract's +-1 iteration and 1e-6."""
    rp, ci, v = cg.gen_matrix(kind, N, 0.1)
    n = len(rp) - 1
    B = cg.gen_rhs("normal", n, m, 7)
    bounds = (0.1, 12.1 if kind == "lap3d7" else 8.1)
    eps = 1e-7 * float(np.linalg.norm(B[:, 0]))
    Xo, ito, _ = O.port_solve(rp, ci, v, B, np.zeros_like(B), s, eps, bounds, 200)
    X, info = cg.solve(rp, ci, v, B, s=s, bounds=("given",) + bounds, tol=eps,
                       tol_mode="abs_col0", maxit=200)
    assert info["status"] == 0
    assert abs(info["iterations"] - ito) <= 1
    assert np.linalg.norm(X - Xo) <= 1e-6 * np.linalg.norm(Xo)


def _residual_norms(rp, ci, v, B, X):
    """Column norms of B - A X, rows summed in extended precision."""
    AX = np.zeros(X.shape, np.longdouble)
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    for c in range(X.shape[1]):
        t = v.astype(np.longdouble) * X[ci, c]
        AX[:, c] = np.add.reduceat(t, rp[:-1])
    assert np.all(np.diff(rp) > 0) and len(rows) == len(v)
    return np.sqrt(((B - AX) ** 2).sum(0))


@pytest.mark.parametrize("kind,N,m", [("lap2d", 1423, 1), ("lap2d", 827, 3), ("lap2d", 360, 16),
                                      ("lap3d7", 67, 5), ("lap3d7", 40, 32), ("st3d27", 40, 7),
                                      ("st3d27", 32, 16), ("st3d27", 61, 2)])
@pytest.mark.parametrize("scale", [1.0, -0.3, 1e-30])
def test_fixed_point_spmm_residual(kind, N, m, scale):
    """B - A X of a one-value stencil matrix (no iterations: the residual alone).  An entry of
    A X is within (27 2^-58 + 35 2^-53) 27 max|X| |c|, max|X| < 5.5 and the residual's RMS
    above 4 |c|: 2e-13 of a column's norm."""
    rp, ci, v = cg.gen_matrix(kind, N, 0.05)
    v = v * scale  # another off-diagonal value, not a power of two
    n = len(rp) - 1
    assert len(v) * m >= 1e7  # the kernel's range
    rng = np.random.default_rng(3)
    X = np.clip(rng.standard_normal((n, m)), -5.5, 5.5)
    X[:, 0] *= 1e-9  # a scale per column
    B = rng.standard_normal((n, m)) * 2 * abs(scale)
    B[:, 0] *= 1e-9
    _, info = cg.solve(rp, ci, v, B, X0=X, s=4, bounds=("given", 0.05, 60.0), tol=1e-8, maxit=0)
    ref = _residual_norms(rp, ci, v, B, X).astype(np.float64)
    got = info["true_relres"] * np.linalg.norm(B, axis=0)
    assert np.all(np.abs(got - ref) <= 2e-13 * ref)


@pytest.mark.parametrize("kind,N,m,s", [("lap2d", 281, 9, 3), ("lap3d7", 33, 16, 4),
                                        ("st3d27", 24, 16, 5), ("st3d27", 26, 13, 3)])
def test_fixed_point_spmm_solves(kind, N, m, s):
    """Basis steps and A Q with it, even and odd widths: the solution's residual, in numpy."""
    rp, ci, v = cg.gen_matrix(kind, N, 0.1)
    n = len(rp) - 1
    B = cg.gen_rhs("normal", n, m, 11)
    X, info = cg.solve(rp, ci, v, B, s=s, bounds="gerschgorin", tol=1e-9, maxit=400)
    assert info["status"] == 0
    r = _residual_norms(rp, ci, v, B, X).astype(np.float64) / np.linalg.norm(B, axis=0)
    assert np.all(r <= 1.01e-9)
    assert np.all(np.abs(r - info["true_relres"]) <= 1e-13)


def test_fixed_point_spmm_outside_range():
    """An infinite entry: the FMA path's pattern of Inf and NaN (the solve breaks down)."""
    rp, ci, v = cg.gen_matrix("lap3d7", 73, 0.1)
    n = len(rp) - 1
    B = cg.gen_rhs("normal", n, 4, 5)
    X0 = np.zeros_like(B)
    X0[n // 2, 1] = np.inf
    for fmt in ("auto", "dia_unstaged"):
        _, info = cg.solve(rp, ci, v, B, X0=X0, s=4, bounds=("given", 0.1, 12.1), maxit=0,
                           spmm_format=fmt)
        assert np.array_equal(np.isfinite(info["true_relres"]), [True, False, True, True])
        # X0's other columns are zero: their residual is B, summed in another order only
        assert np.all(np.abs(info["true_relres"][[0, 2, 3]] - 1.0) <= n * 2.0 ** -53)


@pytest.mark.parametrize("k", [1, 2, 31, 33, 64, 97, 127, 128])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -300, 2.0 ** 300])
def test_qr_small_factor_edges(torch_cuda, k, scale):
    """The one-CTA Cholesky factor and inverse at the edges of its 32-lane columns and 16 warps of
    rows.  A well-conditioned block (cond < 3): each product and the factor are backward stable
    with k u of the norms, u = 2^-53; 100 k u covers the two passes."""
    torch = torch_cuda
    n = 40 * k + 7
    V = _block(torch, n, k, k, 0, "normal", 5) * scale
    Q, R = torch.empty_like(V), torch.empty(k, k, dtype=torch.float64, device="cuda")
    assert cg.lib().cacg_k_tsqr(n, k, ptr(V), k, ptr(Q), k, ptr(R), None) == 0
    torch.cuda.synchronize()
    u = 100 * k * 2.0 ** -53
    eye = torch.eye(k, dtype=torch.float64, device="cuda")
    assert float((Q.T @ Q - eye).norm()) <= u * k ** 0.5
    assert float((Q @ (R / scale) - V / scale).norm()) <= u * float((V / scale).norm())
    assert bool((torch.tril(R, -1) == 0).all()) and bool((torch.diagonal(R) > 0).all())


@pytest.mark.parametrize("kind,N,m,s", [("lap2d", 400, 2, 4), ("lap2d", 400, 3, 3), ("lap2d", 400, 4, 4),
                                        ("lap2d", 400, 4, 7), ("lap2d", 400, 3, 9), ("lap3d7", 37, 5, 4),
                                        ("lap3d7", 37, 1, 8), ("lap3d7", 37, 1, 10)])
def test_solves_around_the_updates_columns(kind, N, m, s):
    """Either side of the columns from which the updates take digit planes (k = 8 and 9; m = 3
    and 4, k m = 64, 100 and 112): the FMA kernels' iterations, and X to what two solutions of
    residual 1e-10 may differ by (a condition number of at most hi / lo)."""
    rp, ci, v = cg.gen_matrix(kind, N, 0.1)
    B = cg.gen_rhs("normal", len(rp) - 1, m, 11)
    lo, hi = 0.1, 8.1 if kind == "lap2d" else 12.1
    p = dict(s=s, bounds=("given", lo, hi), tol=1e-10, maxit=500)
    (X1, i1), (X2, i2) = (cg.solve(rp, ci, v, B, gram=g, **p) for g in ("auto", "fma"))
    assert i1["status"] == 0 and i2["status"] == 0 and abs(i1["iterations"] - i2["iterations"]) <= 1
    assert np.all(np.linalg.norm(X1 - X2, axis=0) <= 2e-10 * (hi / lo) * np.linalg.norm(X2, axis=0))
