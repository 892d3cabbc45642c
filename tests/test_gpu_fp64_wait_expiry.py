"""Expired pipeline waits of the FP64 slice GEMM: a launch whose first operand stage is
never filled gives up its bounded waits and returns, the call fails with SCESS_ERR_CUDA, and
the next call is right. Wide and narrow tiles, one unit and several per CTA, split K."""
import numpy as np
import pytest

from scess_gb300 import cc
from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('M,N,K', [(64, 80, 96), (2000, 17, 600), (3000, 2000, 300), (40000, 30, 90), (24, 24, 36000)])
def test_expired_wait_returns_an_error_and_the_next_call_is_right(gctx, monkeypatch, M, N, K):
    monkeypatch.setenv('SCESS_TUNE', 'f64=1')
    rng = np.random.default_rng(K)
    A = rng.integers(-99, 100, (M, K)).astype(float)
    B = rng.integers(-99, 100, (K, N)).astype(float)
    for _ in range(2):
        gctx.arm_wait_expiry(1 << 20)  # ~0.5 ms at 2 GHz
        with pytest.raises(cc.ScessError) as e:
            gctx.einsum('mk,kn->mn', A, B, out_shape=(M, N))
        assert e.value.status == cc.SCESS_ERR_CUDA and 'wait expired' in str(e.value)
        assert np.array_equal(gctx.einsum('mk,kn->mn', A, B, out_shape=(M, N)), A @ B)
