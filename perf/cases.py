"""Timed cases of the dense LU engine, through its public entry points.

Each case is one call (or the two or three calls that belong together) of a program that uses
the package: factor and solve, a solve with factors it keeps, the mixed-precision solve, a batch
of small uneven systems, the differentiable solve, Cholesky and the complex factorization.
Inputs are dense seeded matrices; all of them make the pivot search and the interchanges work
(only the reference's own benchmark input, randn + n I, is diagonally dominant).
"""
import math

import numpy as np
import torch

import __graft_entry__

oxi = __graft_entry__.load_package()

DEV = "cuda"


def listed():
    return [
        # OxiBLAS.lu + ldiv at the reference benchmark's middle size: latency and launches
        dict(name="lu_256", kind="lu", n=256, nrhs=1, input="kappa", kappa=1e3),
        # the reference's published headline: randn + n I, n = 1024, one right-hand side
        dict(name="lu_1024", kind="lu", n=1024, nrhs=1, input="shifted", kappa=0.0),
        # an ordinary system of odd order with a few right-hand sides
        dict(name="lu_3001x8", kind="lu", n=3001, nrhs=8, input="kappa", kappa=1e4),
        # the largest plain FP64 factor + solve of the benchmark
        dict(name="lu_16384", kind="lu", n=16384, nrhs=1, input="kappa", kappa=1e4),
        # time stepping, adjoint sweeps: factors kept, transposed solve of several right-hand sides
        dict(name="solve_t_4096x8", kind="solve", n=4096, nrhs=8, trans="T", kappa=1e4),
        # the benchmark's headline: mixed precision, kappa = 1e4, one right-hand side
        dict(name="mixed_16384", kind="mixed", n=16384, nrhs=1, precision="fp16x3", kappa=1e4),
        # the benchmark's second configuration: sixteen right-hand sides
        dict(name="mixed_8192x16", kind="mixed", n=8192, nrhs=16, precision="fp16x3", kappa=1e4),
        # many small uneven systems in one launch, FP64 (factors and solutions in place)
        dict(name="batched_fp64_4096", kind="batched", count=4096, nmin=16, nmax=256, kmax=8, prec="fp64"),
        # the same batch with FP32 factors and FP64 refinement
        dict(name="batched_fp32_4096", kind="batched", count=4096, nmin=16, nmax=256, kmax=8, prec="fp32"),
        # differentiable A \ b: forward and backward through torch.autograd
        dict(name="autograd_2048", kind="autograd", n=2048, nrhs=1, kappa=1e3),
        # symmetric positive definite system of odd order
        dict(name="cholesky_4999x4", kind="cholesky", n=4999, nrhs=4),
        # ComplexF64 factor + solve
        dict(name="complex_2048", kind="complex", n=2048, nrhs=1, kappa=1e3),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["lu", "lu", "solve", "mixed", "mixed", "batched", "batched", "autograd", "cholesky",
                       "complex"])
    if kind == "lu":
        return dict(kind=kind, n=_log_int(rng, 100, 12000), nrhs=rng.choice([1, 1, 3, 8, 16]),
                    input=rng.choice(["kappa", "kappa", "shifted"]), kappa=rng.choice([1e2, 1e3, 1e4]))
    if kind == "solve":
        return dict(kind=kind, n=_log_int(rng, 256, 12000), nrhs=rng.randint(1, 16), trans=rng.choice(["N", "T"]),
                    kappa=rng.choice([1e2, 1e3, 1e4]))
    if kind == "mixed":
        precision = rng.choice(["fp16x3", "fp16x3", "fp32", "bf16x3"])
        return dict(kind=kind, n=_log_int(rng, 500, 12000), nrhs=rng.choice([1, 1, 5, 16]), precision=precision,
                    kappa=rng.choice([1e2, 1e3] if precision == "bf16x3" else [1e2, 1e3, 1e4]))
    if kind == "batched":
        nmin = rng.choice([1, 16, 32, 64])
        return dict(kind=kind, count=_log_int(rng, 256, 4096), nmin=nmin, nmax=rng.randint(max(2 * nmin, 32), 256),
                    kmax=rng.choice([1, 4, 8]), prec=rng.choice(["fp64", "fp32"]))
    if kind == "autograd":
        return dict(kind=kind, n=_log_int(rng, 100, 6000), nrhs=rng.choice([1, 1, 4]), kappa=rng.choice([1e2, 1e3]))
    if kind == "cholesky":
        return dict(kind=kind, n=_log_int(rng, 200, 12000), nrhs=rng.choice([1, 4, 16]))
    return dict(kind="complex", n=_log_int(rng, 100, 4000), nrhs=rng.choice([1, 3]), kappa=rng.choice([1e2, 1e3]))


# ---- inputs ----

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, dtype=torch.float64, device=DEV, generator=g)


def _hartley(X, g):
    """The orthogonal Hartley transform of the rows' order, after random signs."""
    n = X.shape[0]
    s = torch.sign(torch.rand(n, 1, dtype=torch.float64, device=DEV, generator=g) - 0.5)
    Y = torch.fft.fft(X * s, dim=0)
    return (Y.real - Y.imag) / math.sqrt(n)


def _fourier(X, g):
    n = X.shape[0]
    t = 2 * math.pi * torch.rand(n, 1, dtype=torch.float64, device=DEV, generator=g)
    return torch.fft.fft(X * torch.polar(torch.ones_like(t), t), dim=0) / math.sqrt(n)


def _kappa_matrix(n, kappa, g, mix=_hartley, dtype=torch.float64):
    """U diag(sigma) V, sigma log-uniform on [1/kappa, 1], U and V products of orthogonal
    transforms and random signs: dense, with the wanted condition number."""
    sigma = kappa ** -torch.rand(n, dtype=torch.float64, device=DEV, generator=g)
    sigma[0], sigma[-1] = 1.0, 1.0 / kappa
    X = torch.diag(sigma).to(dtype)
    for _ in range(2):
        X = mix(mix(X, g), g).t()
    return X.contiguous()


def _matrix(case, g):
    n = case["n"]
    if case["kind"] == "complex":
        return _kappa_matrix(n, case["kappa"], g, _fourier, torch.complex128)
    if case["kind"] == "cholesky":
        G = _randn(g, n, n)
        A = torch.addmm(torch.eye(n, dtype=torch.float64, device=DEV), G, G.t(), alpha=1.0 / n)
        return torch.tril(A) + torch.tril(A, -1).t()
    if case.get("input") == "shifted":
        A = _randn(g, n, n)
        A.diagonal().add_(float(n))
        return A
    return _kappa_matrix(n, case["kappa"], g)


def _rhs(case, g):
    n, k = case["n"], case["nrhs"]
    B = _randn(g, n) if k == 1 else _randn(g, n, k)
    return torch.complex(B, torch.randn(B.shape, dtype=torch.float64, device=DEV, generator=g)) \
        if case["kind"] == "complex" else B


def _batch_shapes(case, seed):
    r = np.random.RandomState(seed % (1 << 31))
    return r.randint(case["nmin"], case["nmax"] + 1, case["count"]), r.randint(1, case["kmax"] + 1, case["count"])


def _batch_values(case, seed):
    """Orders, right-hand-side counts, the offsets of the problems and the values of both pools:
    N(0, 1) plus 1.5 sqrt(n) on a random permutation of the diagonal."""
    n, k = _batch_shapes(case, 1)  # one batch shape; the values are the seed's
    offA = np.concatenate([[0], np.cumsum((n * n + 1) // 2 * 2)])
    offB = np.concatenate([[0], np.cumsum((n * k + 1) // 2 * 2)])
    g = _gen(seed)
    a, b = _randn(g, int(offA[-1])), _randn(g, int(offB[-1]))
    r = np.random.RandomState((seed + 1) % (1 << 31))
    at = np.concatenate([o + np.arange(m) * m + r.permutation(m) for o, m in zip(offA, n)])
    a[torch.from_numpy(at).to(DEV)] += 1.5 * torch.from_numpy(np.repeat(np.sqrt(n), n)).to(DEV)
    return n, k, offA, offB, a, b


def prepare(case, seed):
    g = _gen(seed)
    if case["kind"] == "batched":
        n, k, offA, offB, a, b = _batch_values(case, seed)
        P = oxi.BatchedLU(n, k)
        P.poolA[:a.numel()].copy_(a)
        P.poolB[:b.numel()].copy_(b)
        s = dict(case=case, P=P)
        if case["prec"] == "fp64":  # factored in place: the next pass takes the matrices from here
            s.update(a=P.poolA.clone(), b=P.poolB.clone())
        return s
    A, B = _matrix(case, g), _rhs(case, g)
    if case["kind"] == "solve":
        return dict(case=case, F=oxi.lu(A), B=B)
    if case["kind"] == "autograd":
        return dict(case=case, A=A.requires_grad_(), B=B.requires_grad_(), xbar=_rhs(case, g))
    return dict(case=case, A=A, B=B)


# ---- one pass ----

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("lu", "complex"):
        F = oxi.lu(state["A"])
        return F.factors, F.ipiv, oxi.ldiv(F, state["B"])
    if kind == "solve":
        F = state["F"]
        return oxi.ldiv(F.T if case["trans"] == "T" else F, state["B"])
    if kind == "mixed":
        r = oxi.mixed_solve(state["A"], state["B"], maxiter=30, rtol=1e-14, normwise=True,
                            precision=case["precision"], refine="auto")
        return r["x"], r["converged"]
    if kind == "batched":
        P = state["P"]
        if case["prec"] == "fp64":
            P.poolA.copy_(state["a"])
            P.poolB.copy_(state["b"])
            info = P.gesv("fp64")["info"]
            return P.poolA, P.poolP, P.poolB, info
        r = P.gesv("fp32")
        return P.poolX, r["info"], r["backward_error"] <= 1e-13
    if kind == "autograd":
        x = oxi.solve(state["A"], state["B"])
        Abar, bbar = torch.autograd.grad(x, (state["A"], state["B"]), state["xbar"])
        return x.detach(), Abar, bbar
    F = oxi.cholesky(state["A"])
    return F.factors, F.solve(state["B"])


# ---- what a pass cannot do without ----

def work(case):
    kind = case["kind"]
    if kind == "batched":
        n, k = (v.astype(np.float64) for v in _batch_shapes(case, 1))
        # fp64: A and B read, factors and solutions written; fp32: the matrices are only read
        moved = 16.0 * (n * n + n * k) if case["prec"] == "fp64" else 8.0 * n * n + 16.0 * n * k
        return dict(bytes=float(moved.sum()), flops=float((2.0 / 3.0 * n ** 3 + 2.0 * n * n * k).sum()))
    n, k = float(case["n"]), float(case["nrhs"])
    if kind == "lu":
        return dict(bytes=16.0 * (n * n + n * k) + 8.0 * n, flops=2.0 / 3.0 * n ** 3 + 2.0 * n * n * k)
    if kind == "solve":
        return dict(bytes=8.0 * n * n + 16.0 * n * k, flops=2.0 * n * n * k)
    if kind == "mixed":
        return dict(bytes=8.0 * n * n + 16.0 * n * k, flops=2.0 / 3.0 * n ** 3 + 4.0 * n * n * k)
    if kind == "autograd":  # A read and its gradient written; factor, two solves and the outer product
        return dict(bytes=16.0 * n * n + 32.0 * n * k, flops=2.0 / 3.0 * n ** 3 + 6.0 * n * n * k)
    if kind == "cholesky":
        return dict(bytes=16.0 * (n * n + n * k), flops=n ** 3 / 3.0 + 2.0 * n * n * k)
    return dict(bytes=32.0 * (n * n + n * k) + 8.0 * n, flops=8.0 / 3.0 * n ** 3 + 8.0 * n * n * k)


def tolerance(case):
    """About four times the difference from 64-bit torch measured over the ranges of draw()."""
    kind = case["kind"]
    if kind == "mixed":  # both stop at a normwise backward error of 1e-14
        return dict(rel=5e-13 * math.sqrt(case["kappa"]))
    if kind == "batched":  # fp32: refined to a componentwise backward error of 1e-13
        return dict(rel=1e-14 if case["prec"] == "fp64" else 5e-13)
    if kind == "cholesky" or case.get("input") == "shifted":
        return dict(rel=2e-14)
    # rounding grows with the order and the condition number; whole numbers (pivots) are the same
    return dict(rel=(2.5e-17 if kind == "complex" else 1.5e-17) * case["kappa"] ** 0.75 * max(case["n"], 256))


# ---- the same in plain 64-bit torch ----

def _lu_outputs(A, B):
    LU, piv = torch.linalg.lu_factor(A)
    X = torch.linalg.lu_solve(LU, piv, B.reshape(B.shape[0], -1)).reshape(B.shape)
    return LU, piv.to(torch.int64), X


def _lu_complex(A, B, width=32):
    """Blocked elimination with the pivot of largest |re|^2 + |im|^2 (LAPACK's complex routines,
    and so torch's, take the largest |re| + |im|)."""
    n = A.shape[0]
    A, piv = A.clone(), torch.empty(n, dtype=torch.int64, device=DEV)
    perm = torch.arange(n, device=DEV)
    for f in range(0, n, width):
        l = min(n, f + width)
        for j in range(f, l):
            a = torch.view_as_real(A[j:, j]).square().sum(1)
            p = torch.argmax(a) + j
            piv[j] = p + 1
            both = torch.stack([torch.full_like(p, j), p])
            A[both] = A[both.flip(0)]
            perm[both] = perm[both.flip(0)]
            A[j + 1:, j] /= A[j, j].clone()
            A[j + 1:, j + 1:l] -= torch.outer(A[j + 1:, j], A[j, j + 1:l])
        if l < n:
            A[f:l, l:] = torch.linalg.solve_triangular(A[f:l, f:l], A[f:l, l:], upper=False, unitriangular=True)
            A[l:, l:] -= A[l:, f:l] @ A[f:l, l:]
    Y = torch.linalg.solve_triangular(A, B.reshape(n, -1)[perm], upper=False, unitriangular=True)
    return A, piv, torch.linalg.solve_triangular(A, Y, upper=True).reshape(B.shape)


def _exact_batched(case, seed):
    n, k, offA, offB, a, b = _batch_values(case, seed)
    offP = np.concatenate([[0], np.cumsum(n)])
    A, X = torch.zeros(a.numel() + 2, dtype=a.dtype, device=DEV), torch.zeros(b.numel() + 2, dtype=b.dtype, device=DEV)
    P = torch.zeros(int(n.sum()) + 1, dtype=torch.int64, device=DEV)
    A[:-2], X[:-2] = a, b  # the words between two problems keep what they hold
    kmax = int(k.max())
    for m in np.unique(n):
        ids = np.nonzero(n == m)[0]
        m = int(m)
        ia = torch.from_numpy(offA[ids][:, None] + np.arange(m * m)).to(DEV)
        M = a[ia].view(-1, m, m).mT.contiguous()
        cols = np.minimum(np.arange(kmax)[None, :], k[ids][:, None] - 1)  # short problems repeat their last column
        ib = torch.from_numpy(offB[ids][:, None, None] + cols[:, :, None] * m + np.arange(m)).to(DEV)
        LU, piv = torch.linalg.lu_factor(M)
        S = torch.linalg.lu_solve(LU, piv, b[ib].mT.contiguous())
        A[ia] = LU.mT.reshape(len(ids), m * m)
        P[torch.from_numpy(offP[ids][:, None] + np.arange(m)).to(DEV)] = piv.to(torch.int64)
        X[ib] = S.mT
    info = np.zeros(len(n), dtype=np.int32)
    if case["prec"] == "fp64":
        return A, P, X, info
    for i in np.nonzero((n * k) % 2)[0]:  # only the solutions are written to this pool
        X[int(offB[i] + n[i] * k[i])] = 0.0
    return X, info, np.ones(len(n), dtype=bool)


def exact(case, seed):
    if case["kind"] == "batched":
        return _exact_batched(case, seed)
    g = _gen(seed)
    A, B = _matrix(case, g), _rhs(case, g)
    kind = case["kind"]
    if kind == "complex":
        return _lu_complex(A, B)
    if kind == "lu":
        return _lu_outputs(A, B)
    if kind == "solve":
        return _lu_outputs(A.t().contiguous() if case["trans"] == "T" else A, B)[2]
    if kind == "mixed":
        LU, piv = torch.linalg.lu_factor(A)
        b = B.reshape(case["n"], -1)
        x = torch.linalg.lu_solve(LU, piv, b)
        return (x + torch.linalg.lu_solve(LU, piv, b - A @ x)).reshape(B.shape), True
    if kind == "autograd":
        xbar = _rhs(case, g)
        n = case["n"]
        x = _lu_outputs(A, B)[2]
        bbar = _lu_outputs(A.t().contiguous(), xbar)[2]
        return x, -bbar.reshape(n, -1) @ x.reshape(n, -1).t(), bbar
    L = torch.linalg.cholesky(A)
    return L, torch.cholesky_solve(B.reshape(case["n"], -1), L).reshape(B.shape)
