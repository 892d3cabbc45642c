"""Mixed (T) energies over the forms of the orbit energy kernel: pairs or quads of pairs
per thread (o % 4), (Y, W) pairs in shared memory (o <= 23) or V recomputed (o >= 24), one
W buffer that is cleared behind the kernel or three.

Tolerance: as everywhere for the mixed form, FP32 sums of at most 256 products between
drains and operands of 22 bits: 2e-6 relative to FP64 (E_T here is of order one or less).
"""
import pytest

from scess_gb300.synthetic import convergent_sigma, make_workload
from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('wbuf', [1, 3])
@pytest.mark.parametrize('o,v,nb', [(1, 6, 4), (4, 9, 4), (9, 11, 5), (20, 9, 4), (23, 7, 4), (24, 7, 4), (25, 6, 3)])
def test_mixed_energy_forms(gctx, monkeypatch, o, v, nb, wbuf):
    monkeypatch.setenv('SCESS_TUNE', f't_nb={nb},t_wbuf={wbuf}')
    w = make_workload(o, v, seed=o, with_amplitudes=True, sigma=convergent_sigma(o, v))
    got = gctx.triples(None, w.eps, o, w.t1, w.t2, B=w.B, precision='mixed')
    monkeypatch.setenv('SCESS_TUNE', f't_nb={nb}')
    ref = gctx.triples(None, w.eps, o, w.t1, w.t2, B=w.B, precision='fp64')
    assert abs(got - ref) <= 2e-6 * max(1.0, abs(ref))
