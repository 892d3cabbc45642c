"""FP64 contractions: on the tensor cores' exact BF16 slices (SliceEngine) and, for
small products, on the FP64 units; the tuning key f64 selects either for any size.

Sizes sit where the kernels can go wrong: tiles of 128 x 128, of 16 to 80 columns
(other accumulators) and K blocks of 32 with remainders, one narrow side, K beyond what one unit's integer sum takes
(16384: split), few tiles (split K) and many.

Tolerance: an output is one rounding of a sum whose operands are cut 60 bits
below their row's largest value and whose products below 2^-63 of
|row max| |column max| are dropped: |error| <= 2^-53 |c| + K 2^-57 rowmax colmax
holds with room for any values; integers small enough for exact sums must come
out exactly.
"""
import numpy as np
import pytest

from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu

@pytest.fixture
def sliced(monkeypatch):
    monkeypatch.setenv('SCESS_TUNE', 'f64=1')


SHAPES = [(1, 1, 1), (3, 2, 5), (129, 128, 1217), (128, 127, 1300), (2000, 17, 600), (8, 4001, 700), (1025, 641, 33),
          (600, 520, 65), (300, 31, 16401), (24, 24, 36000), (2111, 1301, 8),
          (700, 45, 300), (260, 60, 100), (20000, 75, 200), (200, 136, 1000)]


def reference(A, B):
    """A.B in extended precision, and the error scale K |row max| |column max|."""
    c = A.astype(np.longdouble) @ B.astype(np.longdouble) if A.shape[1] * A.shape[0] * B.shape[1] < 2e8 else None
    scale = A.shape[1] * np.abs(A).max(axis=1)[:, None] * np.abs(B).max(axis=0)[None, :]
    return c, scale


@pytest.mark.parametrize('M,N,K', SHAPES)
def test_integers_are_exact(gctx, sliced, M, N, K):
    rng = np.random.default_rng(M + N + K)
    lim = 1 << 18
    A = rng.integers(-lim, lim + 1, (M, K)).astype(float)
    B = rng.integers(-lim, lim + 1, (K, N)).astype(float)
    A[:, 0] = lim * 2.0**-3  # a fractional column: exact in FP64 as well
    want = A @ B  # every partial sum is a multiple of 2^-3 below 2^52: exact in any order
    got = gctx.einsum('mk,kn->mn', A, B, out_shape=(M, N))
    assert np.array_equal(got, want)


@pytest.mark.parametrize('M,N,K', [(129, 128, 1217), (2000, 17, 600), (1025, 641, 33), (24, 24, 36000)])
def test_random_values_round_once(gctx, sliced, M, N, K):
    rng = np.random.default_rng(K)
    A = rng.standard_normal((M, K)) * np.exp(2.0 * rng.standard_normal((M, 1)))
    B = rng.standard_normal((K, N)) * np.exp(2.0 * rng.standard_normal((1, N)))
    rows = rng.choice(M, 8, replace=False)  # extended precision is slow: some rows
    want, scale = reference(A[rows], B)
    got = gctx.einsum('mk,kn->mn', A, B, out_shape=(M, N))[rows]
    err = np.abs(got.astype(np.longdouble) - want)
    assert np.all(err <= 2.0**-53 * np.abs(want) + 2.0**-57 * scale)


@pytest.mark.parametrize('alpha,beta', [(1.0, 0.0), (-2.0, 1.0), (0.3, 1.0), (-0.5, 0.7), (1.5, 0.0)])
def test_alpha_beta_and_permuted_output(gctx, sliced, alpha, beta):
    rng = np.random.default_rng(5)
    A = rng.integers(-512, 513, (20, 90, 45)).astype(float)       # (i, a, k)
    B = rng.integers(-512, 513, (45, 33, 21)).astype(float)       # (k, b, j)
    C0 = rng.integers(-512, 513, (33, 20, 21, 90)).astype(float)  # (b, i, j, a)
    got = gctx.einsum('iak,kbj->bija', A, B, C_init=C0, alpha=alpha, beta=beta)
    want = alpha * np.einsum('iak,kbj->bija', A, B, optimize=True) + beta * C0
    assert np.max(np.abs(got - want)) <= 2.0**-50 * np.max(np.abs(want))


SMALL = [(9, 8, 3), (10, 10, 2000), (16, 4, 33), (17, 5, 260), (7, 9, 128), (8, 8, 129), (25, 19, 361), (5, 5, 9025), (90, 10, 90), (361, 25, 131),
         (2, 3, 1), (700, 700, 11)]


@pytest.mark.parametrize('M,N,K', SMALL)
@pytest.mark.parametrize('spec', ['mk,kn->mn', 'km,nk->nm'])
def test_small_products_are_exact(gctx, monkeypatch, M, N, K, spec):
    monkeypatch.setenv('SCESS_TUNE', 'f64=2')
    # tiles of up to 64 outputs, K ranges of 128 with remainders, one tile split over many CTAs
    rng = np.random.default_rng(M * N + K)
    A = rng.integers(-1000, 1001, (M, K)).astype(float)
    B = rng.integers(-1000, 1001, (K, N)).astype(float)
    C0 = rng.integers(-1000, 1001, (M, N)).astype(float)
    want = 2.0 * (A @ B) - 3.0 * C0
    if spec == 'km,nk->nm':
        got = gctx.einsum(spec, A.T, B.T, C_init=C0.T, alpha=2.0, beta=-3.0).T
    else:
        got = gctx.einsum(spec, A, B, C_init=C0, alpha=2.0, beta=-3.0)
    assert np.array_equal(got, want)


@pytest.mark.parametrize('M,K', [(1, 600), (95, 1805), (1215, 513), (1216, 700), (1217, 511), (3000, 33)])
def test_matrix_vector_products_are_exact(gctx, M, K):
    rng = np.random.default_rng(M + K)
    A = rng.integers(-1000, 1001, (M, K)).astype(float)
    x = rng.integers(-1000, 1001, (K, 1)).astype(float)
    assert np.array_equal(gctx.einsum('mk,kn->mn', A, x, out_shape=(M, 1)), A @ x)


def test_zero_tiny_and_huge_rows(gctx, sliced):
    rng = np.random.default_rng(6)
    M, N, K = 140, 150, 1000
    A = rng.integers(-999, 1000, (M, K)).astype(float)
    B = rng.integers(-999, 1000, (K, N)).astype(float)
    A[3] = 0.0
    B[:, 4] = 0.0
    A[5] *= 2.0**-1060  # subnormal values
    A[6] *= 2.0**960
    B[:, 7] *= 2.0**-960
    want = A @ B        # integers times powers of two: exact (or overflow / underflow alike)
    got = gctx.einsum('mk,kn->mn', A, B, out_shape=(M, N))
    assert np.array_equal(got, want)


def test_infinities_and_nans_reach_their_outputs(gctx, sliced):
    rng = np.random.default_rng(7)
    M, N, K = 200, 170, 700
    A = rng.integers(-99, 100, (M, K)).astype(float)
    B = rng.integers(1, 100, (K, N)).astype(float)
    C0 = rng.integers(-99, 100, (M, N)).astype(float)
    A[11, 3] = np.inf
    A[150, 9] = np.nan
    B[20, 130] = -np.inf
    A[:, 20] = np.abs(A[:, 20]) + 1.0
    with np.errstate(invalid='ignore'):
        want = 2.0 * (A @ B) + C0
    got = gctx.einsum('mk,kn->mn', A, B, C_init=C0, alpha=2.0, beta=1.0)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    fin = ~np.isnan(want)
    assert np.array_equal(got[fin], want[fin])
