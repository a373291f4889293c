"""The expiry path of the bounded device-side waits, exercised without a
fault: the tcgen05 Gram's pipeline waits are given a poll limit of zero
(cacg_set_pipeline_wait_limit), so every one of them runs out at once.  The
kernel must drain its own TMA loads and MMAs, free its tensor memory, set
its status word and return; the entry point reports CACG_ERR_TIMEOUT, the
context stays usable, and the next call with the default limit returns the
bit-identical product.  The same through a whole mixed solve."""
import numpy as np
import pytest

import cacg_gb300 as cg
import oracle as O
from gpu_util import dev, host, ptr

pytestmark = pytest.mark.gpu

F32, TC5 = 1, 5


def _gram_tc5(lib, torch, L, R1, R2):
    n, ka = L.shape
    kb1, kb2 = R1.shape[1], R2.shape[1]
    dL, d1, d2 = dev(torch, L), dev(torch, R1), dev(torch, R2)
    Cm = torch.zeros((ka, kb1 + kb2), dtype=torch.float64, device="cuda")
    rc = lib.cacg_k_gram(F32, TC5, n, ptr(dL), ka, ka, ptr(d1), kb1, kb1, ptr(d2), kb2, kb2,
                         ptr(Cm), kb1 + kb2, None)
    return rc, host(Cm)


@pytest.mark.parametrize("n", [100000, 3001])
def test_gram_pipeline_wait_expiry_then_recovery(lib, torch_cuda, n):
    torch = torch_cuda
    L = O.gen_rhs("normal", n, 96, 1).astype(np.float32)
    R1 = O.gen_rhs("normal", n, 96, 2).astype(np.float32)
    R2 = O.gen_rhs("normal", n, 16, 3).astype(np.float32)
    rc0, C0 = _gram_tc5(lib, torch, L, R1, R2)
    assert rc0 == 0
    lib.cacg_set_pipeline_wait_limit(0)
    try:
        rc1, _ = _gram_tc5(lib, torch, L, R1, R2)
    finally:
        lib.cacg_set_pipeline_wait_limit(-1)
    assert rc1 == -5  # CACG_ERR_TIMEOUT
    torch.cuda.synchronize()  # the context is intact
    rc2, C2 = _gram_tc5(lib, torch, L, R1, R2)
    assert rc2 == 0
    assert np.array_equal(C0, C2)


def test_solve_reports_timeout_and_next_solve_is_unchanged(lib, torch_cuda):
    rp, ci, v = cg.gen_matrix("st3d27", 16)
    n = len(rp) - 1
    B = cg.gen_rhs("uniform", n, 16, 2, -1.0, 1.0)
    kw = dict(s=6, bounds=("given", 0.05, 52.0), tol=1e-8, maxit=300, precision="mixed")
    X0, i0 = cg.solve(rp, ci, v, B, **kw)
    lib.cacg_set_pipeline_wait_limit(0)
    try:
        with pytest.raises(cg.CacgError) as e:
            cg.solve(rp, ci, v, B, **kw)
    finally:
        lib.cacg_set_pipeline_wait_limit(-1)
    assert e.value.code == -5
    X1, i1 = cg.solve(rp, ci, v, B, **kw)
    assert i1["status"] == 0 and i1["iterations"] == i0["iterations"]
    assert np.array_equal(X0, X1)


@pytest.mark.parametrize("n,k", [(5000, 48), (400, 20), (300, 128)])
def test_qr_wait_expiry_then_recovery(lib, torch_cuda, n, k):
    """The digit-plane products' waits run out: CACG_ERR_TIMEOUT, not the breakdown that the
    second pass meets in the first one's incomplete result.  (The digit-plane Gram recovers by
    itself: its reduction recomputes the outputs.)"""
    torch = torch_cuda
    V = dev(torch, O.gen_rhs("normal", n, k, 1))

    def qr():
        Q, R = torch.full_like(V, 7.0), torch.zeros(k, k, dtype=torch.float64, device="cuda")
        rc = lib.cacg_k_tsqr(n, k, ptr(V), k, ptr(Q), k, ptr(R), None)
        return rc, host(Q), host(R)

    rc0, Q0, R0 = qr()
    assert rc0 == 0
    lib.cacg_set_pipeline_wait_limit(0)
    try:
        rc1, _, _ = qr()
    finally:
        lib.cacg_set_pipeline_wait_limit(-1)
    assert rc1 == -5  # CACG_ERR_TIMEOUT
    rc2, Q2, R2 = qr()
    assert rc2 == 0 and np.array_equal(Q0, Q2) and np.array_equal(R0, R2)


@pytest.mark.parametrize("n,ka,kb", [(5000, 48, 64), (300, 20, 24), (2000, 130, 70)])
def test_fp64_gram_wait_expiry_is_recomputed(lib, torch_cuda, n, ka, kb):
    """A chain of FP64 FMAs and sixteen partial sums: (n + 16) u of |L|^T |R|, u = 2^-53."""
    torch = torch_cuda
    L, R = O.gen_rhs("normal", n, ka, 1), O.gen_rhs("normal", n, kb, 2)
    dL, dR = dev(torch, L), dev(torch, R)
    Cm = torch.zeros((ka, kb), dtype=torch.float64, device="cuda")
    lib.cacg_set_pipeline_wait_limit(0)
    try:
        rc = lib.cacg_k_gram(0, 0, n, ptr(dL), ka, ka, ptr(dR), kb, kb, None, 0, 0, ptr(Cm), kb,
                             None)
        C = host(Cm)
    finally:
        lib.cacg_set_pipeline_wait_limit(-1)
    assert rc == 0
    ref = L.astype(np.longdouble).T @ R.astype(np.longdouble)
    assert np.all(np.abs(C - ref) <= (n + 16) * 2.0 ** -53 * (np.abs(L).T @ np.abs(R)))
