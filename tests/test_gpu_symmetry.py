"""FP64 iterations choose between the literal and the reassociated contraction list
by the symmetry of their inputs: t2(ijab) = t2(jiba), the driver likewise and
<ab|cd> = <ba|dc>.  Inputs without it follow the reference's literal list."""
import numpy as np
import pytest

import oracle
from scess_gb300.synthetic import convergent_sigma, make_workload
from tests.gpu_common import gctx, rel_err  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('o,v', [(3, 7), (5, 19)])
@pytest.mark.parametrize('broken', ['none', 't2', 'driver', 'vvvv'])
def test_iteration_matches_literal_oracle(gctx, o, v, broken):
    w = make_workload(o, v, seed=3, with_amplitudes=True, sigma=convergent_sigma(o, v))
    rng = np.random.default_rng(8)
    eri, t1, t2 = w.eri(), w.t1, w.t2.copy()
    drv = 1e-3 * rng.standard_normal(t2.shape)
    drv = 0.5 * (drv + drv.transpose(1, 0, 3, 2))
    if broken == 't2':
        t2[0, 1, 2, 3] += 1e-3
    if broken == 'driver':
        drv[1, 0, 2, 3] += 1e-3
    if broken == 'vvvv':
        eri[o + 1, o + 2, o, o + 3] += 1e-2
    ints = oracle.make_integral_blocks(eri, o)
    eia, eijab = oracle.rccsd.denominators(w.eps, o)
    u1, u2 = oracle.update_amplitudes(ints, eia, eijab, drv, t1, t2)
    from scess_gb300 import RCCSD_F12Coupling
    st = gctx.state(eri, w.eps, o, f12=RCCSD_F12Coupling(residual=drv, energy=np.zeros_like(drv)))
    st.set_amplitudes(t1, t2)
    st.iterate(1)
    g1, g2 = st.amplitudes()
    st.close()
    assert rel_err(g1, u1) < 1e-12 and rel_err(g2, u2) < 1e-12
