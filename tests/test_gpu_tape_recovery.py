"""A gradient call that runs out of memory while it records its forward operations leaves no
recording behind: the next call on the context does not write to it."""
import numpy as np
import pytest

import scess_gb300 as s
from scess_gb300 import cc
from scess_gb300.synthetic import make_workload

pytestmark = pytest.mark.gpu


def test_calls_after_gradients_without_memory():
    o, v = 4, 12
    w = make_workload(o, v, seed=8, with_amplitudes=True)
    rng = np.random.default_rng(0)
    A, B = rng.integers(-9, 10, (30, 40)).astype(float), rng.integers(-9, 10, (40, 20)).astype(float)
    failed = 0
    with s.Context(0) as ctx:
        want = ctx.triples_vjp(None, w.eps, o, w.t1, w.t2, B=w.B, want_integrals=True)
        for room in range(1 << 18, 6 << 20, 1 << 18):
            ctx.set_memory_limit(room)
            try:
                ctx.triples_vjp(None, w.eps, o, w.t1, w.t2, B=w.B, want_integrals=True)
            except cc.ScessError as e:
                assert e.status == cc.SCESS_ERR_OOM
                failed += 1
            ctx.set_memory_limit(0)
            assert np.array_equal(ctx.einsum('mk,kn->mn', A, B, out_shape=(30, 20)), A @ B)
        again = ctx.triples_vjp(None, w.eps, o, w.t1, w.t2, B=w.B, want_integrals=True)
    assert failed > 3
    for x, y in zip(want, again):
        assert np.allclose(x, y, rtol=1e-10, atol=1e-14)
