"""FP64 (T) of amplitudes that are not finite (a state takes any): no energy, as from the
FP64 units, and none of it left behind for the next call."""
import numpy as np
import pytest

from scess_gb300.synthetic import make_workload
from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('value', [np.nan, np.inf])
def test_amplitudes_that_are_not_finite_give_no_energy(gctx, value):
    o, v = 5, 19
    w = make_workload(o, v, seed=1, with_amplitudes=True)
    st = gctx.state(w.eri(), w.eps, o)
    st.set_amplitudes(w.t1, w.t2)
    good = st.triples()[0]
    t2 = w.t2.copy()
    t2[1, 2, 3, 4] = value
    st.set_amplitudes(w.t1, t2)
    bad = st.triples()[0]
    st.set_amplitudes(w.t1, w.t2)
    again = st.triples()[0]
    st.close()
    assert np.isfinite(good) and not np.isfinite(bad) and again == good
