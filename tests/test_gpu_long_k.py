"""FP64 products with K beyond the slices' coordinates (their planes of K values in 31 bits)
run on the FP64 units."""
import numpy as np
import pytest

from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('K', [(1 << 31) // 7 + 100])
def test_a_sum_of_more_terms_than_the_slices_can_address(gctx, monkeypatch, K):
    monkeypatch.setenv('SCESS_TUNE', 'f64=1')  # (the slices wherever they can)
    A = np.empty((2, K), order='F')
    A[0] = 1.0
    A[1] = np.arange(K) % 5
    B = np.empty((K, 2), order='F')
    B[:, 0] = 2.0
    B[:, 1] = A[1]
    s, q = float(A[1].sum()), float((A[1] * A[1]).sum())  # (exact: integers below 2^53)
    got = gctx.einsum('mk,kn->mn', A, B, out_shape=(2, 2))
    assert np.array_equal(got, [[2.0 * K, s], [2.0 * s, q]])
