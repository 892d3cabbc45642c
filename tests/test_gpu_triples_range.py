"""FP64 (T) of inputs whose values differ widely: amplitudes far below the integrals, and
integrals that meet vanishing amplitudes."""
import pytest

from scess_gb300.synthetic import make_workload
from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('o,v', [(3, 7), (5, 19), (8, 33)])
@pytest.mark.parametrize('shift', [-45, -30, -15, 15, 40])
def test_energy_is_homogeneous_in_the_amplitudes(gctx, o, v, shift):
    # E_T is quadratic in (t1, t2), and a power of two scales every FP64 operation exactly:
    # both energies are sums of the same numbers, to rounding
    w = make_workload(o, v, seed=1, with_amplitudes=True)
    eri = w.eri()
    e = gctx.triples(eri, w.eps, o, w.t1, w.t2)
    s = gctx.triples(eri, w.eps, o, w.t1 * 2.0**shift, w.t2 * 2.0**shift) * 2.0**(-2 * shift)
    assert abs(s - e) <= 1e-13 * abs(e)


@pytest.mark.parametrize('o,v', [(5, 19), (8, 33)])
@pytest.mark.parametrize('power', [20, 45, 70])
def test_large_integrals_that_meet_zero_amplitudes(gctx, o, v, power):
    # t2 has no component along the virtual f: <ib|af> of that f do not count
    w = make_workload(o, v, seed=2, with_amplitudes=True)
    eri, t2, f = w.eri(), w.t2.copy(), 3
    t2[:, :, f, :] = 0.0
    t2[:, :, :, f] = 0.0
    e = gctx.triples(eri, w.eps, o, w.t1, t2)
    big = eri.copy()
    big[:o, o:, o:, o + f] *= 2.0**power
    g = gctx.triples(big, w.eps, o, w.t1, t2)
    assert abs(g - e) <= 1e-13 * abs(e)
