"""Expired pipeline waits of the mixed tensor-core GEMM on products of several units per CTA
and of a split K: the call fails with SCESS_ERR_CUDA and the next one is right."""
import numpy as np
import pytest

from scess_gb300 import cc
from tests.gpu_common import gctx, rel_err  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('M,N,K', [(3000, 2000, 300), (40000, 30, 90), (40, 24, 36000)])
def test_expired_wait_returns_an_error_and_the_next_call_is_right(gctx, M, N, K):
    rng = np.random.default_rng(K)
    A, B = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    for _ in range(2):
        gctx.arm_wait_expiry(1 << 20)  # ~0.5 ms at 2 GHz
        with pytest.raises(cc.ScessError) as e:
            gctx.einsum('mk,kn->mn', A, B, precision='mixed', out_shape=(M, N))
        assert e.value.status == cc.SCESS_ERR_CUDA and 'wait expired' in str(e.value)
        assert rel_err(gctx.einsum('mk,kn->mn', A, B, precision='mixed', out_shape=(M, N)), A @ B) < 1e-6
