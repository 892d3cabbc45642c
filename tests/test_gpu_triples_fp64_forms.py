"""The FP64 (T) in its forms: the grouped slice launch, the 12 table products a block triple on
slices or on the FP64 units (tuning key f64 = 2), and those that a memory cap leads to."""
import numpy as np
import pytest

import oracle
import scess_gb300 as s
from scess_gb300 import cc
from scess_gb300.synthetic import make_workload
from tests.gpu_common import gctx  # noqa: F401

pytestmark = pytest.mark.gpu

SIZES = [(2, 5), (5, 19), (7, 33), (10, 40)]


@pytest.fixture(scope='module')
def workloads():
    out = {}
    for o, v in SIZES:
        w = make_workload(o, v, seed=4, with_amplitudes=True)
        eri = w.eri()
        out[o, v] = w, eri, oracle.rccsd_triples_correction(eri, w.eps, o, w.t1, w.t2)
    return out


@pytest.mark.parametrize('tune', ['', 'f64=1', 'f64=2', 'f64=2,t_nb=4', 't_nb=4'])
@pytest.mark.parametrize('o,v', SIZES)
def test_forms_agree_with_the_oracle(gctx, monkeypatch, workloads, o, v, tune):
    w, eri, ref = workloads[o, v]
    monkeypatch.setenv('SCESS_TUNE', tune)
    gctx.profile(True)
    et = gctx.triples(eri, w.eps, o, w.t1, w.t2)
    names = gctx.profile_report()
    gctx.profile(False)
    # sums of up to some 10^6 terms: 1e-12 of the total, as for the other FP64 (T) tests (o = 1 is left
    # out: r3 of a single occupied orbital is 4 + 1 + 1 - 6 = 0, so that total is rounding alone)
    assert abs(et - ref) <= 1e-12 * abs(ref)
    grouped = any(k.startswith('slice_gemm[triples]') for k in names)
    assert grouped == ('f64=2' not in tune)


@pytest.mark.parametrize('precision,tol', [('fp64', 1e-12), ('mixed', 1e-5)])
def test_every_cap_gives_the_energy_or_no_memory(workloads, precision, tol):
    o, v = 7, 33
    w, eri, ref = workloads[o, v]
    seen = []
    with s.Context(0) as ctx:
        for cap in np.geomspace(18e6, 200e6, 24):
            ctx.set_memory_limit(int(cap))
            try:
                et = ctx.triples(eri, w.eps, o, w.t1, w.t2, precision=precision)
            except cc.ScessError as e:
                assert e.status == cc.SCESS_ERR_OOM and not any(seen)  # (more room is never worse)
                seen.append(False)
                continue
            assert abs(et - ref) <= tol * abs(ref), cap
            seen.append(True)
    assert not seen[0] and seen[-1]
