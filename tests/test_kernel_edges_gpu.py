"""The kernels at the sizes where their tiles, remainders and branches change,
against the oracle or a 64-bit NumPy solve.

FP64 LU factors are the oracle's bits.  Solves: a backward stable solve leaves
max|b - A x| <= c n eps (|A||x| + |b|) with a moderate c; the bound below is 30 n
eps of the normwise terms, the bar the reference's own solves are held to,
whatever the condition of the matrix and of its factors' diagonal blocks.
"""
import numpy as np
import pytest
import scipy.linalg as sl
import torch

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _np(t):
    return t.detach().cpu().numpy()


def _backward(A, x, b):
    r = np.abs(b - A @ x).max()
    return r / (np.abs(A).sum(1).max() * np.abs(x).max() + np.abs(b).max()) / (A.shape[0] * EPS)


@pytest.mark.parametrize("m", [5, 31, 33, 255, 256, 257, 513, 4095, 4096, 4097, 8191, 8193])
def test_leaf_heights_bit_identical(pkg, oracle, m):
    """Rows per CTA and cluster sizes of the leaf change with the height; 40
    columns leave a whole leaf and a narrow one.  Values of equal magnitude make
    the arg-max resolve ties by position."""
    rng = np.random.default_rng(m)
    for A in (rng.standard_normal((m, 40)), rng.integers(-2, 3, (m, 40)).astype(float)):
        F = pkg.lu(A, check=False)
        Fo, ipo, info = oracle.getrf(A, check=False)
        assert F.info == info
        assert np.array_equal(_np(F.ipiv), ipo)
        assert np.array_equal(_np(F.factors), Fo)


@pytest.mark.parametrize("m", [129, 191, 192, 193, 257, 513, 1111, 4096, 4097, 4161])
def test_wide_leaf_bit_identical(pkg, oracle, m):
    """A panel of 128 columns takes two FP64 leaves of 64 columns (the recursion's
    step from 32 to 64 inside the launch) where 64 <= rows <= 4096; the 32 columns
    behind the panel take the narrow one."""
    rng = np.random.default_rng(m)
    Z = rng.standard_normal((m, 160))
    Z[:, 9] = 0.0                        # zero pivots in both halves of a leaf
    Z[:, 45] = 0.0
    Z[m // 2:, 70] = np.nan
    for A in (rng.standard_normal((m, 160)), rng.integers(-2, 3, (m, 160)).astype(float), Z):
        F = pkg.lu(A, check=False)
        Fo, ipo, info = oracle.getrf(A, check=False)
        assert F.info == info
        assert np.array_equal(_np(F.ipiv), ipo)
        assert np.array_equal(_np(F.factors), Fo, equal_nan=True)


@pytest.mark.parametrize("m,n,k", [(1, 2, 2), (63, 30, 16), (64, 32, 18), (65, 34, 64), (130, 66, 128), (569, 128, 128)])
def test_gemm_tiles_same_bits(pkg, m, n, k):
    """Few 128 x 64 tiles: the update runs on 64 x 32 ones.  Every element is one
    chain over k, so the rows of a taller update, which takes the large tiles, are
    the same bits; and they are within k eps of the exact product."""
    g = torch.Generator(device="cuda").manual_seed(m)
    rows = 128 * 105
    C, A = (torch.randn(rows, c, dtype=torch.float64, device="cuda", generator=g) for c in (n, k))
    B = torch.randn(k, n, dtype=torch.float64, device="cuda", generator=g)
    small = pkg.gemm_update(C[:m].clone(), A[:m].contiguous(), B)
    assert torch.equal(small, pkg.gemm_update(C.clone(), A, B)[:m])
    err = (small - (C[:m] - A[:m] @ B)).abs()
    assert bool((err <= 2 * (k + 1) * EPS * (C[:m].abs() + A[:m].abs() @ B.abs())).all())


@pytest.mark.parametrize("power", [2, 3])
def test_float32_block_row_by_substitution(pkg, power):
    """U12 of an FP32 panel whose triangle's 32 x 32 blocks are ill-conditioned, its
    columns the products of L with random ones: |P A - L U| <= k u |L||U| with k
    terms an element, which substitution keeps (a product with the blocks'
    inverses left 2.3 and 2.9 times that)."""
    rng = np.random.default_rng(power)
    m, w = 600, 128
    T = np.linalg.matrix_power(2 * np.eye(m) - np.eye(m, k=1) - np.eye(m, k=-1), power)[:, :w].astype(np.float32)
    P, L, _ = sl.lu(T)
    A = np.hstack([T, (P @ L @ rng.standard_normal((w, 64))).astype(np.float32)])
    F = pkg.lu(torch.from_numpy(A), check=False)  # the rows below have nothing left to factor
    LU, PA = _np(F.factors).astype(float), A[F.p].astype(float)
    n = A.shape[1]
    Lf, U = np.tril(LU, -1) + np.eye(m, n), np.triu(LU[:n])
    k = np.minimum(np.arange(m)[:, None], np.arange(n)) + 1
    assert (np.abs(PA - Lf @ U) <= (k + 1) * 2.0 ** -24 * (np.abs(Lf) @ np.abs(U))).all()


def test_repeated_factorization_same_bits(pkg):
    """Both streams of the lookahead and all pipelines under load: every repetition
    gives the same factors."""
    g = torch.Generator(device="cuda").manual_seed(2048)
    A = torch.randn(2048, 2048, dtype=torch.float64, device="cuda", generator=g)
    F0 = pkg.lu(A).factors.clone()
    for _ in range(400):
        assert torch.equal(pkg.lu(A).factors, F0)


def test_repeated_products_same_bits(pkg):
    """The slabs' refills of the complex product and of both tile sizes."""
    g = torch.Generator(device="cuda").manual_seed(7)

    def randn(*shape, dtype=torch.float64):
        return torch.randn(*shape, dtype=dtype, device="cuda", generator=g)
    Z, S = randn(1500, 1500, dtype=torch.complex128), randn(1500, 1500)
    S = S @ S.T + 1500 * torch.eye(1500, dtype=S.dtype, device="cuda")
    C, A, B = randn(3000, 128), randn(3000, 128), randn(128, 128)
    for count, f in ((150, lambda: pkg.lu(Z).factors), (300, lambda: pkg.cholesky(S).factors),
                     (4000, lambda: pkg.gemm_update(C.clone(), A, B))):
        first = f().clone()
        assert all(torch.equal(f(), first) for _ in range(count))


def test_leaf_zero_nan_and_extreme_pivots(pkg, oracle):
    rng = np.random.default_rng(7)
    A = rng.standard_normal((300, 64))
    A[:, 11] = 0.0                       # a zero pivot inside a group
    A[:, 20] = A[:, 3] * 2.0             # rank deficiency found by elimination
    A[40:, 33] = np.nan                  # a NaN below never wins
    B = rng.standard_normal((300, 64)) * 10.0 ** rng.uniform(-250, 250, (300, 1))
    C = rng.standard_normal((300, 64))
    C[rng.uniform(size=C.shape) < 0.3] = -0.0
    for M in (A, B, C):
        F = pkg.lu(M, check=False)
        Fo, ipo, info = oracle.getrf(M, check=False)
        assert F.info == info
        assert np.array_equal(_np(F.ipiv), ipo)
        assert np.array_equal(_np(F.factors), Fo, equal_nan=True)


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 511, 513, 1100])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 7, 8, 17])
def test_superblock_solves(pkg, n, nrhs):
    rng = np.random.default_rng(1000 * n + nrhs)
    A = rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, nrhs))
    F = pkg.lu(A)
    assert _backward(A, _np(F.solve(B)), B) <= 30
    assert _backward(A.T, _np(F.T.solve(B)), B) <= 30
    S = A @ A.T / n + np.eye(n)
    S = (S + S.T) / 2
    assert _backward(S, _np(pkg.cholesky(S).solve(torch.from_numpy(B))), B) <= 30


@pytest.mark.parametrize("n", [1, 33, 127, 128, 129, 300])
@pytest.mark.parametrize("nrhs", [1, 2, 5])
def test_superblock_solves_complex(pkg, n, nrhs):
    rng = np.random.default_rng(1000 * n + nrhs)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    F = pkg.lu(A)
    assert _backward(A, _np(F.solve(B)), B) <= 30
    assert _backward(A.T, _np(F.T.solve(B)), B) <= 30
    assert _backward(A.conj().T, _np(F.H.solve(B)), B) <= 30


@pytest.mark.parametrize("m", [15, 16, 17, 255, 257, 4096, 4097, 8193])
def test_complex_leaf_heights(pkg, oracle, m):
    """Pivots as the oracle's; the overflow rule (abs2 not finite) inside a group."""
    rng = np.random.default_rng(m)
    A = rng.standard_normal((m, 20)) + 1j * rng.standard_normal((m, 20))
    A[m // 2, 2] = 1e200 + 1e200j
    A[m // 3, 2] = 2e200
    F = pkg.lu(A, check=False)
    Fo, ipo, info = oracle.zgetrf(A)
    assert F.info == info
    assert np.array_equal(_np(F.ipiv), ipo)
    assert np.linalg.norm(_np(F.factors) - Fo) <= 1e-11 * np.linalg.norm(Fo)


@pytest.mark.parametrize("n", [8, 9, 31, 121, 127, 129, 136, 257, 385])
def test_cholesky_blocks_and_first_failing_column(pkg, oracle, n):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n))
    A = G @ G.T + n * np.eye(n)
    Lo, _ = oracle.potrf(A)
    assert np.linalg.norm(_np(pkg.cholesky(A).L) - Lo) <= 1e-13 * np.linalg.norm(Lo)
    for bad in sorted({0, 7, 8, n // 2, n - 1}):
        if bad >= n:
            continue
        M = A.copy()
        M[bad, bad] = -1.0
        assert pkg.cholesky(M, check=False).info == oracle.potrf(M)[1] == bad + 1


def test_cholesky_roots_and_quotients_are_the_rounded_ones(pkg):
    """The diagonal block forms roots and quotients from an approximate reciprocal
    root by fused corrections: the values of sqrt and of the division, over the
    exponents where that form is taken.  (It could miss one in 2^50: a result
    whose exact value lies within 2^-103 of the middle of two numbers.)"""
    rng = np.random.default_rng(11)
    for _ in range(10):
        a = rng.uniform(1, 2, 1024) * 2.0 ** rng.integers(-899, 899, 1024)
        assert np.array_equal(_np(pkg.cholesky(np.diag(a)).L).diagonal(), np.sqrt(a))
    for _ in range(40):
        a = rng.uniform(1, 4) * 2.0 ** rng.integers(-200, 200)
        v = np.sqrt(a) * rng.uniform(-1, 1, 127) * 2.0 ** rng.integers(-60, 60, 127)
        A = np.diag(np.concatenate([[a], 256 * (v / np.sqrt(a)) ** 2]))
        A[0, 1:] = A[1:, 0] = v
        # the other columns see u_0i u_0j of both signs and sizes: only the first row is exact
        A[1:, 1:] += np.outer(v, v) / a
        assert np.array_equal(_np(pkg.cholesky(A).L)[1:, 0], v / np.sqrt(a))


@pytest.mark.parametrize("n", [8, 127, 300])
def test_cholesky_pivots_out_of_the_fast_range(pkg, n):
    """Scaling by 2^-960 (exact) brings the pivots under 2^-900, where roots and
    quotients are computed by the library functions.  |L L' - A| <= (n + 1) eps
    |L||L'| elementwise, whose diagonal is that of A; twice that for the products
    with inverted blocks."""
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n))
    A = G @ G.T + n * np.eye(n)
    L = _np(pkg.cholesky(A * 2.0 ** -960).L) * 2.0 ** 480
    assert np.abs(L @ L.T - A).max() <= 2 * (n + 1) * EPS * A.diagonal().max()


@pytest.mark.parametrize("nrhs", [4, 5, 8, 9, 16])
@pytest.mark.parametrize("n", [130, 300, 1027])
def test_mixed_solve_right_hand_sides(pkg, n, nrhs):
    """The residual's tensor-core pass (more than four right-hand sides) and the
    narrow block solve of the FP32 panels, whole and ragged."""
    rng = np.random.default_rng(n + nrhs)
    A = rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, nrhs))
    r = pkg.mixed_solve(A, B, maxiter=20, rtol=1e-14, precision="fp16x3", refine="auto", normwise=True)
    x = _np(r["x"])
    assert r["converged"]
    res = np.abs(B - A @ x).max(0) / (np.abs(A).sum(1).max() * np.abs(x).max(0) + np.abs(B).max(0))
    assert res.max() <= 1e-14 + 4 * n * EPS  # the report's value up to the rounding of this residual
    xe = sl.solve(A, B)
    assert np.linalg.norm(x - xe) <= 1e-10 * np.linalg.norm(xe)


def _gauss(n, w, reg=0.0):
    i = np.arange(n)
    return np.exp(-((i[:, None] - i[None]) / w) ** 2) + reg * np.eye(n)


def _smooth(kind, n):
    """Matrices whose factors' diagonal blocks have inverses of large norm: the fourth
    difference and kernel matrices."""
    if kind == "difference":
        T = 2 * np.eye(n) - np.eye(n, k=1) - np.eye(n, k=-1)
        return T @ T
    w, reg = kind
    return _gauss(n, w, reg)


SMOOTH = [("difference", 256), ("difference", 512), ("difference", 2048), ((2.0, 0.0), 1024), ((2.5, 0.0), 1024),
          ((3.0, 0.0), 1024), ((3.0, 0.0), 2048)] + [((8.0, r), n) for r in (1e-4, 1e-6, 1e-10) for n in (128, 256, 257, 1024)]


def _rhs_of(M, n, rng, dtype):
    """b = M x for x of ones and for random x: x stays small, so the error of a
    product with an inverse of large norm shows."""
    X = np.stack([np.ones(n), rng.standard_normal(n)], 1)
    return (M.astype(np.clongdouble if np.iscomplexobj(M) else np.longdouble) @ X).astype(dtype)


def _normwise(M, x, b, eps):
    r = np.abs(b - M @ x).max(0)
    return (r / (np.abs(M).sum(1).max() * np.abs(x).max(0) + np.abs(b).max(0))).max() / (M.shape[0] * eps)


@pytest.mark.parametrize("kind,n", SMOOTH)
def test_solves_with_ill_conditioned_blocks(pkg, kind, n):
    """Substitution leaves 30 n eps whatever the condition of the diagonal blocks;
    so do the superblock solves: corrected products, or substitution by strips."""
    rng = np.random.default_rng(n)
    A = _smooth(kind, n)
    F = pkg.lu(A)
    for Fv, M in ((F, A), (F.T, A.T)):
        b = _rhs_of(M, n, rng, np.float64)
        assert _normwise(M, _np(pkg.ldiv(Fv, torch.from_numpy(b))), b, EPS) <= 30
    if kind == "difference" or kind[1] >= 1e-6 or kind[0] <= 2.5:  # positive definite to rounding
        b = _rhs_of(A, n, rng, np.float64)
        assert _normwise(A, _np(pkg.cholesky(A).solve(torch.from_numpy(b))), b, EPS) <= 30


@pytest.mark.parametrize("kind,n", [s for s in SMOOTH if s[1] <= 1024])
def test_solves_with_ill_conditioned_blocks_complex(pkg, kind, n):
    rng = np.random.default_rng(n)
    t = np.exp(2j * np.pi * rng.uniform(size=n))
    A = t[:, None] * _smooth(kind, n) * np.exp(2j * np.pi * rng.uniform(size=n))
    F = pkg.lu(A)
    for Fv, M in ((F, A), (F.T, A.T), (F.H, A.conj().T)):
        b = _rhs_of(M, n, rng, np.complex128)
        assert _normwise(M, _np(pkg.ldiv(Fv, torch.from_numpy(b))), b, EPS) <= 30


@pytest.mark.parametrize("kind,n", [s for s in SMOOTH if s[1] <= 1024])
def test_solves_with_ill_conditioned_blocks_float32(pkg, kind, n):
    rng = np.random.default_rng(n)
    A = _smooth(kind, n).astype(np.float32)
    A64 = A.astype(np.float64)
    F = pkg.lu(torch.from_numpy(A))
    for Fv, M in ((F, A64), (F.T, A64.T)):
        b = _rhs_of(M, n, rng, np.float32)
        x = _np(pkg.ldiv(Fv, torch.from_numpy(b))).astype(np.float64)
        assert _normwise(M, x, b.astype(np.float64), np.finfo(np.float32).eps) <= 30


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [256, 600])
def test_solve_where_the_inverse_overflows(pkg, dtype, n):
    """Ones on the diagonal, -1 below: L is the matrix, its inverse has elements up to
    2^(n-2).  Substitution of the right-hand side of x = ones only sees small whole
    numbers, so it is exact."""
    A = (np.eye(n) - np.tril(np.ones((n, n)), -1)).astype(dtype)
    b = (A.astype(np.float64) @ np.ones(n)).astype(dtype)
    F = pkg.lu(torch.from_numpy(A))
    assert np.array_equal(_np(pkg.ldiv(F, torch.from_numpy(b))), np.ones(n))
    bt = (A.T.astype(np.float64) @ np.ones(n)).astype(dtype)
    assert np.array_equal(_np(pkg.ldiv(F.T, torch.from_numpy(bt))), np.ones(n))


@pytest.mark.parametrize("dtype,e", [(np.float64, 1005), (np.float64, -1000), (np.float32, 118), (np.float32, -110)])
def test_solve_at_the_ends_of_the_range(pkg, dtype, e):
    """Scaled by a power of two, the inverses of a block are subnormal or near overflow."""
    rng = np.random.default_rng(9)
    n = 300
    A = (rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)).astype(dtype)
    b = (A.astype(np.longdouble) @ rng.uniform(0.5, 1, n)).astype(dtype) / dtype(64)
    x = _np(pkg.ldiv(pkg.lu(torch.from_numpy(np.ldexp(A, e))), torch.from_numpy(np.ldexp(b, e)))).astype(np.float64)
    A, b = A.astype(np.float64), b.astype(np.float64)
    assert _normwise(A, x[:, None], b[:, None], np.finfo(dtype).eps) <= 30


def test_infinite_right_hand_side_stays_in_its_column(pkg):
    rng = np.random.default_rng(5)
    n = 600
    A = rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((n, 3))
    B[300, 1] = np.inf
    X = _np(pkg.lu(A).solve(B))
    assert not np.isfinite(X[:, 1]).any()
    assert _backward(A, X[:, [0, 2]], B[:, [0, 2]]) <= 30
