"""FP64 contractions on the FP64 units (tuning key f64 = 2): the short-K form against a long
side (K <= 32, a small side of at most 256) and the finely cut one, at the edges of their
tiles; split sums of the mixed engine.

Tolerance: a sum of K products in any order, alpha and beta applied once each, is within
(K + 3) 2^-53 (|alpha| sum |a b| + |beta C|) of the exact value.
"""
import numpy as np
import pytest

from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('alpha,beta', [(1.0, 1.0), (-2.0, 0.0), (0.3, 0.75)])
@pytest.mark.parametrize('order', ['C', 'F'])
@pytest.mark.parametrize('M,N,K', [(1, 3001, 1), (10, 8101, 10), (8101, 9, 32), (256, 4097, 7), (90, 900, 16), (33, 80000, 3),
                                   (300, 257, 9), (5, 6, 127), (17, 16, 129), (7, 65, 4000)])
def test_products(gctx, monkeypatch, M, N, K, order, alpha, beta):
    monkeypatch.setenv('SCESS_TUNE', 'f64=2')
    rng = np.random.default_rng(M + N + K)
    A, B, C = (np.array(rng.standard_normal(s), order=order) for s in ((M, K), (K, N), (M, N)))
    got = gctx.einsum('mk,kn->mn', A, B, C_init=C, alpha=alpha, beta=beta)
    A, B, C = (x.astype(np.longdouble) for x in (A, B, C))
    tol = (K + 3) * 2.0**-53 * (abs(alpha) * (abs(A) @ abs(B)) + abs(beta * C))
    assert np.all(abs(got - (alpha * (A @ B) + beta * C)) <= tol)


@pytest.mark.parametrize('M,N,K', [(10, 90, 9000), (129, 33, 2000), (130, 10, 700), (900, 127, 300)])
@pytest.mark.parametrize('alpha,beta', [(1.0, 1.0), (-2.0, 0.0), (0.3, 0.75)])
def test_mixed_narrow_and_split(gctx, M, N, K, alpha, beta):
    # operands of 22 bits, FP32 sums of a K block: 2e-6 of the largest value, as for every mixed product
    rng = np.random.default_rng(K)
    A, B, C = rng.standard_normal((M, K)), rng.standard_normal((N, K)), rng.standard_normal((M, N))
    got = gctx.einsum('mk,nk->mn', A, B, C_init=C, alpha=alpha, beta=beta, precision='mixed')
    ref = alpha * (A @ B.T) + beta * C
    assert abs(got - ref).max() <= 2e-6 * abs(ref).max()
