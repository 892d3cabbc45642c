"""A solve whose tensor-core wait expires fails one way or another (the expiry, or an energy
that is not finite by then); the next call on the context must not hear of it."""
import pytest

import oracle
from scess_gb300 import cc
from scess_gb300.synthetic import make_workload
from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
@pytest.mark.parametrize('iterations', [1, 100])
def test_the_call_after_a_failed_solve_is_right(gctx, monkeypatch, precision, iterations):
    monkeypatch.setenv('SCESS_TUNE', 'f64=1')
    w = make_workload(5, 19, seed=0)
    eri = w.eri()
    ref = oracle.solve_rccsd_diis(eri, w.eps, 5)
    gctx.arm_wait_expiry(1 << 20)
    with pytest.raises(cc.ScessError):
        gctx.solve(eri, w.eps, 5, precision=precision, max_iterations=iterations)
    got = gctx.solve(eri, w.eps, 5, precision=precision)
    assert got.converged and abs(got.E_CCSD - ref.E_CCSD) < (1e-9 if precision == 'fp64' else 1e-6)
