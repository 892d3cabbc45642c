"""(T) without amplitudes is exactly zero, on the form that (T) prefers."""
import numpy as np
import pytest

from scess_gb300.synthetic import make_workload
from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('o,v', [(3, 7), (6, 21)])
def test_zero_amplitudes(gctx, o, v):
    w = make_workload(o, v, seed=1)
    gctx.profile(True)
    e = gctx.triples(w.eri(), w.eps, o, np.zeros((o, v)), np.zeros((o, o, v, v)))
    names = gctx.profile_report()
    gctx.profile(False)
    assert e == 0.0 and any(k.startswith('slice_gemm[triples]') for k in names)
