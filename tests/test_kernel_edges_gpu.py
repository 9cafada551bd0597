"""The kernels at the sizes where their tiles, remainders and branches change,
against the oracle or a 64-bit NumPy solve.

FP64 LU factors are the oracle's bits.  Solves: a backward stable solve leaves
max|b - A x| <= c n eps (|A||x| + |b|) with c of the order of the growth of the
blocks' inverses; the bound below is 30 n eps of the normwise terms, the bar
the reference's own solves are held to.
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
