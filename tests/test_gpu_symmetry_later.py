"""FP64 iterations on integrals that leave t2 symmetric at the start but break its
symmetry in the first iteration: the later ones follow the reference's literal list too."""
import pytest

import oracle
from scess_gb300.synthetic import convergent_sigma, make_workload
from tests.gpu_common import gctx, rel_err  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('o,v', [(3, 7), (5, 19)])
@pytest.mark.parametrize('broken', ['none', 'oooo', 'oovv'])
def test_integrals_that_break_the_symmetry_of_t2_later(gctx, o, v, broken):
    # <kl|ij> and <ij|ab> enter t2 outside the symmetrised terms: it loses its symmetry in
    # the first iteration, and the next ones need the literal list
    w = make_workload(o, v, seed=3, with_amplitudes=True, sigma=convergent_sigma(o, v))
    eri, t1, t2 = w.eri(), w.t1, w.t2
    if broken == 'oooo':
        eri[0, 1, 2, 0] += 1e-1
    if broken == 'oovv':
        eri[0, 1, o, o + 3] += 1e-1
    ints = oracle.make_integral_blocks(eri, o)
    eia, eijab = oracle.rccsd.denominators(w.eps, o)
    st = gctx.state(eri, w.eps, o, diis_start=100)  # (no extrapolation)
    st.set_amplitudes(t1, t2)
    st.iterate(4)
    g1, g2 = st.amplitudes()
    st.close()
    for _ in range(4):
        t1, t2 = oracle.update_amplitudes(ints, eia, eijab, None, t1, t2)
    assert rel_err(g1, t1) < 1e-12 and rel_err(g2, t2) < 1e-12
