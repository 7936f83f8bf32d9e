"""What a query call finds in its index's scratch.  It allocates only when it
brings more queries than any call before: neither k, nor the rows' alignment, nor
the memory they come from asks for more, so such a call can be captured, and a
captured one replayed after later calls.  And nothing that an earlier call left in
the tickets by which a query's last block is told is counted.  Needs a B200."""
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


def test_nothing_left_in_a_ticket_is_counted(torch):
    from cuda.bindings import runtime as rt

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r
        return r[1:]

    X = torch.from_numpy(synth.clustered_f32(3_050, 36, n_clusters=7, seed=4)).cuda()
    Q = X[3_000:].clone()
    index = build_index(X[:3_000].contiguous(), 3, 10, 5, leaf_size=256)[0]
    want = index.query(Q, 10)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        got = index.query(Q, 10)
    graph.instantiate()
    # the captured call clears the tickets: where they lie
    g = rt.cudaGraph_t(graph.raw_cuda_graph())
    nodes = ok(rt.cudaGraphGetNodes(g, ok(rt.cudaGraphGetNodes(g))[1]))[0]
    clears = [ok(rt.cudaGraphMemsetNodeGetParams(v))[0] for v in nodes
              if ok(rt.cudaGraphNodeGetType(v))[0] ==
              rt.cudaGraphNodeType.cudaGraphNodeTypeMemset]
    assert len(clears) == 1 and clears[0].width * clears[0].elementSize >= 8 * len(Q)
    tickets, t = int(clears[0].dst), np.zeros(len(Q), np.uint64)

    def leave(change):
        torch.cuda.synchronize()
        ok(rt.cudaMemcpy(t.ctypes.data, tickets, t.nbytes,
                         rt.cudaMemcpyKind.cudaMemcpyDeviceToHost))
        t[:] = change(t)
        ok(rt.cudaMemcpy(tickets, t.ctypes.data, t.nbytes,
                         rt.cudaMemcpyKind.cudaMemcpyHostToDevice))

    for change in (lambda v: v - np.uint64(2), lambda v: v + np.uint64(3), lambda v: 0 * v):
        for nq in (len(Q), 1):
            leave(change)
            i, d = index.query(Q[:nq], 10)
            assert torch.equal(i, want[0][:nq]) and torch.equal(d, want[1][:nq])
        leave(lambda v: v + np.uint64(1 << 40))  # of a later turn than the captured one
        got[0].fill_(-9)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
