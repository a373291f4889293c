"""Timed cases of the solver framework: what its users run, through its public entry points.

Families
  solve  Matrix.solve_device: a resident matrix, right-hand sides and solution on the GPU
  host   the drop-in bcbcg_v1: host arrays in and out, FP64, 64-bit indices, Gerschgorin bounds
  serve  a closed burst of requests through Server (host arrays in and out)
  gram   cacg_k_gram: L^T [R1 | R2] of FP64 tall blocks, the library's Gram entry point
  tsqr   cacg_k_tsqr: tall-skinny QR of an FP64 block

Matrices: the Laplacian and 27-point stencil families of the library's generators, which
``exact`` diagonalises by sine transforms, and two kinds without a constant stencil
(variable-coefficient diffusion, a random graph kept as CSR), which ``exact`` solves by FP64
conjugate gradients run down to rounding.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import cacg_gb300 as cg

TOL = 1e-8  # relative residual on every column, the tolerance of the solver's workloads


def listed():
    return [
        # one right-hand side, 128 x 128 Poisson, CBCG: the smallest solve, where launches and
        # the host's round trips count
        dict(name="solve_fp64_lap2d_128_m1", family="solve", kind="lap2d", N=128, shift=0.0, m=1,
             s=4, precision="fp64", bounds="analytic"),
        # block solve, 3-D 7-point 64^3, 8 right-hand sides, s = 8 (a 64-wide basis)
        dict(name="solve_fp64_lap3d7_64_m8", family="solve", kind="lap3d7", N=64, shift=0.0, m=8,
             s=8, precision="fp64", bounds="analytic"),
        # 27-point stencil, 16 right-hand sides, FP64: the largest FP64 work
        dict(name="solve_fp64_st3d27_96_m16", family="solve", kind="st3d27", N=96, shift=0.0,
             m=16, s=6, precision="fp64", bounds="stencil"),
        # the headline workload of bench.py: mixed precision, 128^3, 16 right-hand sides
        dict(name="solve_mixed_st3d27_128_m16", family="solve", kind="st3d27", N=128, shift=0.0,
             m=16, s=6, precision="mixed", bounds="stencil"),
        # a large request of the serving workload: an odd number of right-hand sides, a grid
        # that no tile divides
        dict(name="solve_mixed_lap2d_701_m11", family="solve", kind="lap2d", N=701, shift=0.043,
             m=11, s=4, precision="mixed", bounds="gerschgorin"),
        # the same in FP64, a middle size
        dict(name="solve_fp64_lap3d7_37_m5", family="solve", kind="lap3d7", N=37, shift=0.05, m=5,
             s=4, precision="fp64", bounds="gerschgorin"),
        # variable coefficients, 32 right-hand sides, a 128-wide basis, Lanczos bounds
        dict(name="solve_fp64_varcoef_256_m32", family="solve", kind="varcoef2d", N=256,
             shift=0.01, m=32, s=4, precision="fp64", bounds="lanczos"),
        # an unstructured matrix: no diagonals to use, the CSR kernels
        dict(name="solve_fp64_graph_50k_m6", family="solve", kind="graph", N=50021, shift=0.05,
             m=6, s=4, precision="fp64", bounds="gerschgorin"),
        # the reference's own call, on host arrays
        dict(name="host_bcbcg_lap3d7_32_m4", family="host", kind="lap3d7", N=32, shift=0.1, m=4,
             s=4),
        # the serving engine, both precisions
        dict(name="serve_fp64_16", family="serve", count=16, nmin=1000, nmax=40000, mix=1,
             precision="fp64"),
        dict(name="serve_mixed_24", family="serve", count=24, nmin=1000, nmax=60000, mix=2,
             precision="mixed"),
        # the tall-skinny QR as a library call (its drawn sibling is the Gram product)
        dict(name="tsqr_400k_48", family="tsqr", n=400000, k=48),
    ]


def draw(rng):
    """One more case of the same ranges."""

    def logu(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    u = rng.random()
    if u < 0.60:
        precision = "fp64" if rng.random() < 0.7 else "mixed"
        v = rng.random()
        if v < 0.70:  # the serving workload's matrices
            kind = "lap2d" if rng.random() < 0.5 else "lap3d7"
            m = rng.randint(1, 16)
            n = logu(1e3, min(1e6, 5.4e6 / m))
            N = max(4, round(n ** (0.5 if kind == "lap2d" else 1.0 / 3.0)))
            return dict(family="solve", kind=kind, N=N, shift=round(rng.uniform(0.01, 0.1), 4),
                        m=m, s=4, precision=precision, bounds="gerschgorin")
        if v < 0.85:
            return dict(family="solve", kind="st3d27", N=round(logu(12, 80)), shift=0.0,
                        m=rng.choice([4, 8, 10, 12, 16]), s=rng.choice([4, 5, 6]),
                        precision=precision, bounds="stencil")
        return dict(family="solve", kind="graph", N=round(logu(2e3, 1.2e5)), shift=0.05,
                    m=rng.randint(1, 12), s=4, precision=precision, bounds="gerschgorin")
    if u < 0.70:
        return dict(family="host", kind=rng.choice(["lap2d", "lap3d7"]), N=rng.randint(12, 40),
                    shift=0.1, m=rng.randint(1, 8), s=rng.choice([3, 4, 5]))
    if u < 0.80:
        nmax = round(logu(4e3, 6e4))
        return dict(family="serve", count=rng.randint(4, 24), nmin=1000, nmax=nmax,
                    mix=rng.randint(10, 10000), precision=rng.choice(["fp64", "mixed"]))
    if u < 0.90:
        ka = rng.randint(3, 128)
        kb2 = rng.randint(0, 16)
        return dict(family="gram", n=round(logu(2e3, 1.2e6)), ka=ka,
                    kb1=ka if rng.random() < 0.7 else rng.randint(2, 128), kb2=kb2)
    k = rng.randint(4, 96)
    return dict(family="tsqr", n=round(logu(2e3, 4e5)), k=k)


# ------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1 + int(seed))


@functools.lru_cache(maxsize=4)
def _matrix(kind, N, shift):
    """Host CSR of a case's matrix (the matrix is the problem, the seed draws the data)."""
    if kind == "graph":
        return _graph(N, shift)
    sigma = 0.3 if kind == "varcoef2d" else 0.0
    return cg.gen_matrix(kind, N, shift, sigma, 7)


def _graph(n, shift):
    """Weighted Laplacian of a random graph (each node joined to 4 others within a window, as
    meshes ordered for locality are) plus a shift, as CSR."""
    rng = np.random.default_rng(n)
    i = np.repeat(np.arange(n, dtype=np.int64), 4)
    j = (i + rng.integers(1, max(2, n // 40), i.size)) % n
    w = rng.uniform(0.5, 1.5, i.size)
    key = np.concatenate([i * n + j, j * n + i])
    val = np.concatenate([-w, -w])
    key, inv = np.unique(key, return_inverse=True)
    off = np.bincount(inv.ravel(), weights=val)
    keep = key // n != key % n
    key, off = key[keep], off[keep]
    diag = shift - np.bincount(key // n, weights=off, minlength=n)
    key = np.concatenate([key, np.arange(n, dtype=np.int64) * (n + 1)])
    off = np.concatenate([off, diag])
    order = np.argsort(key, kind="stable")
    key, off = key[order], off[order]
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(key // n, minlength=n), out=rp[1:])
    return rp, (key % n).astype(np.int32), off


def _rhs(kind, n, m, seed):
    g = _generator(seed)
    if kind == "st3d27":
        return torch.rand(n, m, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    return torch.randn(n, m, dtype=torch.float64, device="cuda", generator=g)


def _bounds(case):
    kind, N, b = case["kind"], case["N"], case["bounds"]
    if b == "analytic":  # extreme eigenvalues of the Dirichlet Laplacian
        d = {"lap2d": 2, "lap3d7": 3}[kind]
        t = math.pi / (N + 1)
        return ("given", case["shift"] + d * (2 - 2 * math.cos(t)),
                case["shift"] + d * (2 - 2 * math.cos(N * t)))
    if b == "stencil":
        return ("given", 0.05, 52.0)
    return ("lanczos", 50) if b == "lanczos" else "gerschgorin"


def _specs(case):
    """Shapes of a burst: the serving workload's distribution, from the case's mix."""
    from cacg_gb300.serving import request_specs

    return request_specs(case["count"], seed=case["mix"], nmin=case["nmin"], nmax=case["nmax"])


class _Burst:
    """A server and the requests it is sent; the server goes with the object."""

    def __init__(self, case, seed):
        self.server = cg.Server(8 << 30, max_active=16)
        self.params = cg.Params(s=4, bounds="gerschgorin", tol=TOL, maxit=1000,
                                precision=case["precision"])
        self.requests = []
        for i, sp in enumerate(_specs(case)):
            rp, ci, v = _matrix(sp["kind"], sp["N"], sp["shift"])
            B = _rhs(sp["kind"], len(rp) - 1, sp["m"], 1000 * int(seed) + i).cpu().numpy()
            self.requests.append((rp, ci, v, B))

    def __del__(self):
        self.server.close()


def prepare(case, seed):
    f = case["family"]
    if f == "solve":
        rp, ci, v = _matrix(case["kind"], case["N"], case["shift"])
        B = _rhs(case["kind"], len(rp) - 1, case["m"], seed)
        A = cg.Matrix(rp, ci, v, want_fp32=case["precision"] == "mixed")
        P = cg.Params(s=case["s"], bounds=_bounds(case), tol=TOL, maxit=2000,
                      precision=case["precision"])
        return dict(f=f, A=A, B=B, X=torch.zeros_like(B), P=P, m=case["m"])
    if f == "host":
        rp, ci, v = _matrix(case["kind"], case["N"], case["shift"])
        B = _rhs(case["kind"], len(rp) - 1, case["m"], seed).cpu().numpy()
        return dict(f=f, rp=rp.astype(np.int64), ci=ci.astype(np.int64), v=v, B=B, s=case["s"],
                    X=np.zeros_like(B), eps=TOL * float(np.linalg.norm(B[:, 0])))
    if f == "serve":
        return dict(f=f, burst=_Burst(case, seed))
    g = _generator(seed)
    n = case["n"]
    if f == "gram":
        ka, kb = case["ka"], case["kb1"] + case["kb2"]
        L = torch.randn(n, ka, dtype=torch.float64, device="cuda", generator=g)
        R1 = torch.randn(n, case["kb1"], dtype=torch.float64, device="cuda", generator=g)
        R2 = torch.randn(n, case["kb2"], dtype=torch.float64, device="cuda", generator=g)
        C = torch.empty(ka, kb, dtype=torch.float64, device="cuda")
        return dict(f=f, L=L, R1=R1, R2=R2, C=C)
    k = case["k"]
    V = torch.randn(n, k, dtype=torch.float64, device="cuda", generator=g)
    return dict(f=f, V=V, Q=torch.empty_like(V),
                R=torch.empty(k, k, dtype=torch.float64, device="cuda"))


# -------------------------------------------------------------------------- a pass
def _ok(rc, what):
    if rc != 0:
        raise RuntimeError("%s: %s" % (what, cg.status_string(rc)))


def run(state):
    f = state["f"]
    if f == "solve":
        X = state["X"].zero_()
        r = state["A"].solve_device(state["B"].data_ptr(), X.data_ptr(), state["m"], state["P"])
        _ok(r["status"], "solve_device")
        return X
    if f == "host":
        X = state["X"]
        X[:] = 0.0
        cg.bcbcg_v1(state["rp"], state["ci"], state["v"], state["B"], X, state["s"], state["eps"])
        _ok(cg.last_status(), "bcbcg_v1")
        return X
    if f == "serve":
        b = state["burst"]
        tickets = [b.server.submit(rp, ci, v, B, b.params) for rp, ci, v, B in b.requests]
        out = []
        for t in tickets:
            X, r = b.server.wait(t)
            _ok(r["status"], "request")
            out.append(X)
        return out
    vp = ctypes.c_void_p
    if f == "gram":
        L, R1, R2, C = state["L"], state["R1"], state["R2"], state["C"]
        two = R2.shape[1]
        _ok(cg.lib().cacg_k_gram(0, 0, L.shape[0], vp(L.data_ptr()), L.shape[1], L.shape[1],
                                 vp(R1.data_ptr()), R1.shape[1], R1.shape[1],
                                 vp(R2.data_ptr()) if two else None, two, two, vp(C.data_ptr()),
                                 C.shape[1], None), "cacg_k_gram")
        return C
    V, Q, R = state["V"], state["Q"], state["R"]
    k = V.shape[1]
    _ok(cg.lib().cacg_k_tsqr(V.shape[0], k, vp(V.data_ptr()), k, vp(Q.data_ptr()), k,
                             vp(R.data_ptr()), None), "cacg_k_tsqr")
    return [Q, R]


# ---------------------------------------------------------------------------- work
def _shape(kind, N):
    """(rows, nonzeros, condition number estimate without a shift)"""
    if kind == "graph":
        return N, 9 * N, 400.0
    n = N * N if kind in ("lap2d", "varcoef2d") else N ** 3
    per = {"lap2d": 5, "varcoef2d": 5, "lap3d7": 7, "st3d27": 27}[kind]
    return n, per * n, 0.41 * (N + 1) ** 2


def _solve_work(kind, N, shift, m, s, es):
    """Outer iterations that conjugate gradients needs (its bound on the condition number) times
    what each cannot do without: the matrix and the vectors once, the basis, Q and A Q written
    and read once; products, Gram matrices and updates as flops."""
    n, nnz, kappa = _shape(kind, N)
    top = 2.0 * nnz / n
    if shift > 0:
        kappa = min(kappa, (top + shift) / shift)
    steps = 0.35 * math.sqrt(kappa) * math.log(2.0 / TOL)
    its = max(2.0, steps / s / (1.0 + 0.1 * math.log2(m)))
    k = s * m
    by = nnz * (es + 4.0) + n * m * 8.0 * 4 + 6.0 * n * k * es
    fl = 2.0 * nnz * m * (2 * s - 1) + 2.0 * n * k * (3 * k + 3 * m) + k ** 3
    return its * by, its * fl


def work(case):
    f = case["family"]
    if f in ("solve", "host"):
        es = 4.0 if case.get("precision") == "mixed" else 8.0
        b, fl = _solve_work(case["kind"], case["N"], case["shift"], case["m"], case["s"], es)
        return {"bytes": b, "flops": fl}
    if f == "serve":
        es = 4.0 if case["precision"] == "mixed" else 8.0
        w = [_solve_work(sp["kind"], sp["N"], sp["shift"], sp["m"], 4, es) for sp in _specs(case)]
        return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}
    n = case["n"]
    if f == "gram":
        kb = case["kb1"] + case["kb2"]
        return {"bytes": 8.0 * (n * (case["ka"] + kb) + case["ka"] * kb),
                "flops": 2.0 * n * case["ka"] * kb}
    k = case["k"]
    return {"bytes": 8.0 * (2 * n * k + k * k), "flops": 4.0 * n * k * k}


# --------------------------------------------------------------------------- exact
def _sine_solve(kind, N, shift, B):
    """A^-1 B for the constant-coefficient stencils: A is diagonal in the sine basis."""
    t = math.pi / (N + 1) * torch.arange(1, N + 1, dtype=torch.float64, device=B.device)
    idx = torch.arange(1, N + 1, dtype=torch.float64, device=B.device)
    V = math.sqrt(2.0 / (N + 1)) * torch.sin(idx[:, None] * t[None, :])
    d = 2 if kind == "lap2d" else 3
    T = B.reshape((N,) * d + (-1,))

    def apply(T):
        for a in range(d):
            T = torch.movedim(torch.tensordot(V, T, dims=([1], [a])), 0, a)
        return T

    if kind == "st3d27":
        e = 1 + 2 * torch.cos(t)
        lam = 27 - e[:, None, None] * e[None, :, None] * e[None, None, :] + shift
    else:
        e = 2 - 2 * torch.cos(t)
        lam = e[:, None] + e[None, :] if d == 2 else (e[:, None, None] + e[None, :, None] +
                                                      e[None, None, :])
        lam = lam + shift
    return apply(apply(T) / lam[..., None]).reshape(B.shape).contiguous()


def _cg_solve(rp, ci, v, B):
    """A^-1 B by FP64 conjugate gradients, one refinement step, plain torch."""
    n = len(rp) - 1
    A = torch.sparse_csr_tensor(torch.from_numpy(rp).to(B.device), torch.from_numpy(ci).to(B.device),
                                torch.from_numpy(v).to(B.device), (n, n))
    X = torch.zeros_like(B)
    for _ in range(2):
        R = B - A @ X
        stop = 1e-13 * R.norm(dim=0)
        D, P, rr = torch.zeros_like(B), R.clone(), (R * R).sum(0)
        for it in range(6000):
            AP = A @ P
            a = rr / (P * AP).sum(0).clamp_min(1e-300)
            D += a * P
            R -= a * AP
            new = (R * R).sum(0)
            P = R + (new / rr.clamp_min(1e-300)) * P
            rr = new
            if it % 20 == 19 and bool((rr.sqrt() <= stop).all()):
                break
        X = X + D
    return X


def _solution(kind, N, shift, B):
    if kind in ("lap2d", "lap3d7", "st3d27"):
        return _sine_solve(kind, N, shift, B)
    return _cg_solve(*_matrix(kind, N, shift), B)


def exact(case, seed):
    f = case["family"]
    if f in ("solve", "host"):
        n = _shape(case["kind"], case["N"])[0]
        X = _solution(case["kind"], case["N"], case["shift"],
                      _rhs(case["kind"], n, case["m"], seed))
        return X.cpu().numpy() if f == "host" else X
    if f == "serve":
        out = []
        for i, sp in enumerate(_specs(case)):
            n = _shape(sp["kind"], sp["N"])[0]
            B = _rhs(sp["kind"], n, sp["m"], 1000 * int(seed) + i)
            out.append(_sine_solve(sp["kind"], sp["N"], sp["shift"], B).cpu().numpy())
        return out
    st = prepare(case, seed)
    if f == "gram":
        return st["L"].T @ torch.cat([st["R1"], st["R2"]], dim=1)
    Q, R = torch.linalg.qr(st["V"])
    sign = torch.where(R.diagonal() < 0, -1.0, 1.0).to(R.dtype)
    return [Q * sign[None, :], R * sign[:, None]]
