"""A product and its transpose take the same FP64 route: the estimate that chooses it is of
the launch that is made, whichever side the operands come on."""
import numpy as np
import pytest

from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu

UNITS = {'dgemm_small', 'skinny64', 'dgemm_table'}


def route(gctx, spec, A, B, shape):
    gctx.profile(True)
    gctx.einsum(spec, A, B, out_shape=shape)
    names = {k.split('[')[0] for k in gctx.profile_report()}
    gctx.profile(False)
    return 'slices' if 'slice_gemm' in names else (names & UNITS).pop()


@pytest.mark.parametrize('M,N,K', [(6, 5766, 1116), (10, 81000, 90), (17, 3000, 400), (40, 900, 700), (3, 3, 40),
                                   (64, 64, 900), (65, 200, 300)])
def test_a_product_and_its_transpose_take_one_route(gctx, M, N, K):
    rng = np.random.default_rng(M)
    A, B = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    a = route(gctx, 'mk,kn->mn', A, B, (M, N))
    b = route(gctx, 'nk,km->nm', B.T, A.T, (N, M))
    assert a == b
