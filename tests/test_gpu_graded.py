"""FP64 contractions of operands whose values differ widely inside a row or column: what
the tensor cores' fixed-point slices cannot hold goes to the FP64 units.

Tolerance: a chain of K fused multiply-adds has |error| <= K 2^-53 sum_k |a_k b_k| and,
with roundings of either sign, about sqrt(K) of them; every output has to be within
(sqrt(K) + 2) 2^-53 sum_k |a_k b_k| of the exact sum, whichever unit computed it.
"""
import math

import numpy as np
import pytest

from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu


def exact_dot(a, b):
    """The correctly rounded sum of products (Dekker's error-free products, then fsum)."""
    p = a * b
    def split(x):
        c = 134217729.0 * x
        h = c - (c - x)
        return h, x - h
    ah, al = split(a)
    bh, bl = split(b)
    e = al * bl - (((p - ah * bh) - al * bh) - ah * bl)
    return math.fsum(np.concatenate([p, e]))


def operands(kind, M, N, K, rng):
    A = rng.standard_normal((M, K))
    B = rng.standard_normal((K, N))
    if kind.startswith('large'):  # one large value a row, which meets zeros of every column
        g = int(kind[5:])
        dead = rng.choice(K, max(1, K // 20), replace=False)
        A[np.arange(M), rng.choice(dead, M)] = 2.0**g
        B[dead] = 0.0
    elif kind == 'half':  # large values that meet zeros of half of the columns
        dead = rng.choice(K, max(1, K // 20), replace=False)
        A[:, dead] *= 2.0**45
        B[np.ix_(dead, rng.choice(N, N // 2, replace=False))] = 0.0
    elif kind == 'opposite':  # graded along k, A one way and B the other
        s = rng.integers(-60, 61, K)
        A *= 2.0**s[None, :]
        B *= 2.0**-s[:, None]
    elif kind == 'wide':  # every value of its own size
        A *= 2.0**rng.integers(-50, 1, (M, K))
        B *= 2.0**rng.integers(-50, 1, (K, N))
    elif kind == 'sparse':
        A[rng.random((M, K)) < 0.9] = 0.0
        B[rng.random((K, N)) < 0.5] = 0.0
    elif kind == 'disjoint':  # no common index but one, of tiny values
        A[:, ::2] = 0.0
        B[1::2] = 0.0
        A[:, 0] = 2.0**-70
        A[M // 2:, 0] = 0.0
        B[0] = 2.0**-50
    return A, B


KINDS = ['plain', 'large12', 'large25', 'large40', 'large60', 'half', 'opposite', 'wide', 'sparse', 'disjoint']
# few tiles (K split over CTAs) and many, narrow sides, short and long K, remainders
SHAPES = [(140, 150, 700), (33, 20, 5000), (65, 129, 40), (1300, 1100, 96), (2000, 17, 600), (900, 1500, 33)]


@pytest.mark.parametrize('kind', KINDS)
@pytest.mark.parametrize('M,N,K', SHAPES)
def test_every_output_is_as_accurate_as_fused_multiply_adds(gctx, monkeypatch, M, N, K, kind):
    monkeypatch.setenv('SCESS_TUNE', 'f64=1')
    rng = np.random.default_rng(M + N + K + KINDS.index(kind))
    A, B = operands(kind, M, N, K, rng)
    C0 = rng.standard_normal((M, N)) * np.abs(A).mean() * np.abs(B).mean()
    got = gctx.einsum('mk,kn->mn', A, B, out_shape=(M, N))
    acc = gctx.einsum('mk,nk->nm', A, B.T, C_init=C0.T, alpha=-2.0, beta=1.0).T
    ms, ns = rng.choice(M, min(M, 24), replace=False), rng.choice(N, min(N, 24), replace=False)
    tol = (math.sqrt(K) + 2) * 2.0**-53
    for m in ms:
        for n in ns:
            want, scale = exact_dot(A[m], B[:, n]), float(np.abs(A[m]) @ np.abs(B[:, n]))
            assert abs(got[m, n] - want) <= tol * scale, (m, n, got[m, n], want)
            both = math.fsum([C0[m, n], -2.0 * want])
            assert abs(acc[m, n] - both) <= 2.0 * tol * scale + 2.0**-52 * (abs(both) + abs(C0[m, n])), (m, n)
