"""Memory caps under a live state: an iteration that cannot allocate returns SCESS_ERR_OOM, and
the state goes on when there is room again."""
import numpy as np
import pytest

import oracle
import scess_gb300 as s
from scess_gb300 import cc
from scess_gb300.synthetic import convergent_sigma, make_workload
from tests.gpu_common import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_cap_below_what_is_held_on_a_context_without_engines(precision):
    o, v = 4, 11
    w = make_workload(o, v, seed=5, with_amplitudes=True, sigma=convergent_sigma(o, v))
    eri = w.eri()
    ints = oracle.make_integral_blocks(eri, o)
    eia, eijab = oracle.rccsd.denominators(w.eps, o)
    u1, u2 = oracle.update_amplitudes(ints, eia, eijab, None, w.t1, w.t2)
    with s.Context(0) as ctx:
        st = ctx.state(eri, w.eps, o, precision=precision)
        st.set_amplitudes(w.t1, w.t2)
        ctx.set_memory_limit(1 << 12)
        with pytest.raises(cc.ScessError) as e:
            st.iterate(1)
        assert e.value.status == cc.SCESS_ERR_OOM
        ctx.set_memory_limit(0)
        st.set_amplitudes(w.t1, w.t2)
        st.iterate(1)
        g1, g2 = st.amplitudes()
        st.close()
    tol = 1e-12 if precision == 'fp64' else 1e-5
    assert rel_err(g1, u1) < tol and rel_err(g2, u2) < tol
    assert np.all(np.isfinite(g2))
