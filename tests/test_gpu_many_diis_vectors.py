"""DIIS subspaces larger than the context's 64 scalars: the Gram row of an iteration is read in
parts."""
import numpy as np
import pytest

import oracle
from scess_gb300.synthetic import convergent_sigma, make_workload
from tests.gpu_common import gctx, rel_err  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('vectors', [47, 48, 49, 64, 65, 90])
def test_iterations_beyond_64_vectors(gctx, vectors):
    o, v = 2, 4
    w = make_workload(o, v, seed=2, sigma=0.4 * convergent_sigma(o, v))  # (converges without extrapolation)
    eri = w.eri()
    ref = oracle.solve_rccsd_diis(eri, w.eps, o)
    st = gctx.state(eri, w.eps, o, max_diis_vectors=vectors, max_iterations=100, diis_start=1000,
                    energy_convergence=0.0, amplitude_convergence=0.0)  # (never converged, never extrapolated)
    st.set_amplitudes(ref.t1, ref.t2)
    st.iterate(95)
    t1, t2 = st.amplitudes()
    st.close()
    # a fixed point: 95 updates stay where the converged amplitudes are
    assert rel_err(t2, ref.t2) < 1e-6 and np.all(np.isfinite(t1))
    got = gctx.solve(eri, w.eps, o, max_diis_vectors=vectors)
    assert got.converged and abs(got.E_CCSD - ref.E_CCSD) < 1e-9
