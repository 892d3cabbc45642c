"""Integer contractions whose terms cancel to small results of either sign: exact on the FP64
units (every partial sum is an integer below 2^53) and on the slices."""
import numpy as np
import pytest

from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('tune', ['f64=1', 'f64=2'])
@pytest.mark.parametrize('M,N,K', [(130, 140, 300), (40, 30, 1000), (33, 20, 5000), (900, 700, 40)])
def test_small_results_of_either_sign_are_exact(gctx, monkeypatch, M, N, K, tune):
    monkeypatch.setenv('SCESS_TUNE', tune)
    rng = np.random.default_rng(M + K)
    A = rng.integers(-4095, 4096, (M, K)).astype(float)
    B = rng.integers(-4095, 4096, (K, N)).astype(float)
    want_row = rng.integers(-9, 10, N).astype(float)  # the first row's results
    A[0, -1] = 1.0
    B[-1] = want_row - A[0, :-1] @ B[:-1]
    want = A @ B
    assert np.array_equal(want[0], want_row)
    assert np.array_equal(gctx.einsum('mk,kn->mn', A, B, out_shape=(M, N)), want)
    got = gctx.einsum('mk,kn->mn', A, B, out_shape=(M, N), alpha=-3.0)
    assert np.array_equal(got, -3.0 * want)
