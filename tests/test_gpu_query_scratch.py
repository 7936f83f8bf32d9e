"""A query call allocates only when it brings more queries than any call before:
neither k, nor the rows' alignment, nor the memory they come from asks for more.
So such a call can be captured, and a captured one replayed after later calls.
Needs a B200."""
import numpy as np
import pytest

from drpt_b200 import build_index, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as _t
    if not _t.cuda.is_available():
        pytest.skip("no CUDA device")
    return _t


@pytest.mark.parametrize("nq", [1, 40, 700])
def test_other_calls_of_as_many_queries_allocate_nothing(torch, nq):
    X = torch.from_numpy(synth.clustered_f32(3_700, 36, n_clusters=7, seed=4)).cuda()
    Q = X[3_000:3_000 + nq].clone()
    index = build_index(X[:3_000].contiguous(), 3, 10, 5, leaf_size=256)[0]
    fresh = build_index(X[:3_000].contiguous(), 3, 10, 5, leaf_size=256)[0]
    off = torch.empty(Q.numel() + 1, device="cuda")[1:].view_as(Q)  # off a 16-byte boundary
    off.copy_(Q)
    want = [fresh.query(q, k) for q, k in ((Q, 32), (off, 32), (Q, 7))]
    index.query(Q, 1)  # the only call that may allocate
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [index.query(q, k) for q, k in ((Q, 32), (off, 32), (Q, 7))]
    host = index.query(Q.cpu().numpy(), 32)
    assert np.array_equal(host[0], want[0][0].cpu().numpy())
    for _ in range(2):
        for i, d in got:
            i.fill_(-9)
            d.fill_(-9.0)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for g, w in zip(got, want) for a, b in zip(g, w))
