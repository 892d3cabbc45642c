"""What fits a memory cap in the form that needs least is done, whichever form is preferred:
FP64 iterations whose combined integrals don't fit take the literal list."""
import numpy as np
import pytest

import oracle
import scess_gb300 as s
from scess_gb300 import cc
from scess_gb300.synthetic import convergent_sigma, make_workload
from tests.gpu_common import rel_err

pytestmark = pytest.mark.gpu


def iterate_at(eri, w, o, room):
    """Amplitudes after two iterations with `room` bytes beyond what the state holds, or None."""
    with s.Context(0) as ctx:
        st = ctx.state(eri, w.eps, o)
        st.set_amplitudes(w.t1, w.t2)
        ctx.set_memory_limit(ctx.memory_held() + room)
        try:
            st.iterate(2)
            return st.amplitudes()
        except cc.ScessError as e:
            assert e.status == cc.SCESS_ERR_OOM
            return None
        finally:
            ctx.set_memory_limit(0)
            st.close()


def test_iterations_with_few_virtuals_under_a_cap():
    o, v = 20, 6  # the combined integrals and the ladder's pairs are larger than <ab|cd> here
    w = make_workload(o, v, seed=6, with_amplitudes=True, sigma=convergent_sigma(o, v))
    eri = w.eri()
    broken = eri.copy()
    broken[o + 1, o + 2, o, o + 3] += 1e-2  # (takes the literal list from the start)
    room = next(r for r in range(1 << 18, 1 << 24, 1 << 16) if iterate_at(broken, w, o, r))
    got = iterate_at(eri, w, o, room + (200 << 10))  # (the first attempt's offset tables stay)
    assert got is not None
    want = iterate_at(eri, w, o, 1 << 30)
    assert rel_err(got[0], want[0]) < 1e-12 and rel_err(got[1], want[1]) < 1e-12
    ints = oracle.make_integral_blocks(eri, o)
    eia, eijab = oracle.rccsd.denominators(w.eps, o)
    t1, t2 = w.t1, w.t2
    for _ in range(2):  # (no extrapolation yet)
        t1, t2 = oracle.update_amplitudes(ints, eia, eijab, None, t1, t2)
    assert rel_err(got[0], t1) < 1e-12 and rel_err(got[1], t2) < 1e-12
    assert np.all(np.isfinite(got[1]))


@pytest.mark.parametrize('precision,tol', [('mixed', 1e-5), ('fp64', 1e-12)])
def test_triples_under_a_cap_take_smaller_blocks(monkeypatch, precision, tol):
    o, v = 13, 40
    w = make_workload(o, v, seed=7, with_amplitudes=True)

    def energy(cap, tune):
        monkeypatch.setenv('SCESS_TUNE', tune)
        with s.Context(0) as ctx:
            ctx.set_memory_limit(cap)
            try:
                return ctx.triples(None, w.eps, o, w.t1, w.t2, B=w.B, precision=precision)
            except cc.ScessError as e:
                assert e.status == cc.SCESS_ERR_OOM
                return None

    ample = energy(0, '')
    small = 'f64=2,t_nb=2'  # (blocks of two virtuals; FP64: the form without packs)
    cap = next(c for c in range(8 << 20, 1 << 30, 2 << 20) if energy(c, small) is not None)
    got = energy(cap + (2 << 20), '')
    assert got is not None and abs(got - ample) <= tol * abs(ample)
