"""scess_einsum_static on a captured stream: its launches follow copies, fills and kernels of the
same graph, and kernels follow them."""
import numpy as np
import pytest

from scess_gb300 import cc

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('M,N,K', [(5, 7, 3), (64, 65, 40), (200, 30, 2000)])
def test_capture_and_replay(M, N, K):
    rng = np.random.default_rng(K)
    dev = torch.device('cuda:0')

    def values(*shape):  # integers: exact sums in any order
        return torch.from_numpy(rng.integers(-99, 100, shape).astype(float)).to(dev)

    a0, b0 = values(K, M), values(N, K)  # (column-major A(m,k), B(k,n))
    a, b = torch.empty_like(a0), torch.empty_like(b0)
    c, d = torch.empty((N, M), dtype=torch.float64, device=dev), torch.empty((N, M), dtype=torch.float64, device=dev)

    def body(stream):
        a.copy_(a0)       # a copy, then
        b.copy_(b0)
        c.zero_()         # a fill before the first contraction
        cc.einsum_static('mk,kn->mn', a.data_ptr(), (M, K), b.data_ptr(), (K, N), c.data_ptr(), (M, N), stream=stream)
        a.mul_(2.0)       # a kernel that writes what the contraction before has read
        cc.einsum_static('mk,kn->mn', a.data_ptr(), (M, K), b.data_ptr(), (K, N), c.data_ptr(), (M, N), 1.0, 1.0,
                         stream)
        d.copy_(c)

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        body(s.cuda_stream)
    s.synchronize()
    want = 3.0 * (b0 @ a0)
    assert torch.equal(d, want)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        body(s.cuda_stream)
    for q in range(3):
        a0.copy_(values(K, M))
        d.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(d, 3.0 * (b0 @ a0))
