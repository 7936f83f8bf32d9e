"""Routes of a query call beside the usual ones: rows that start off the boundary
that the grouped forms read from, with and without a ticket for each query, and
calls that are cut into blocks.  The lists are the same bit for bit.  Needs a
B200."""
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


@pytest.mark.parametrize("dtype,d,k", [("f32", 36, 10), ("f32", 132, 32), ("u8", 36, 7),
                                       ("u8", 100, 32)])
def test_rows_off_the_boundary(torch, dtype, d, k):
    n, most = 2_500, 4_097  # one more than there are tickets
    if dtype == "u8":
        Z = torch.from_numpy(synth.clustered_u8(n + most, d, seed=3)).cuda()
    else:
        Z = torch.from_numpy(synth.clustered_f32(n + most, d, n_clusters=7, seed=3)).cuda()
    Q = Z[n:].contiguous()
    Q[5] = Z[17]
    index = build_index(Z[:n].contiguous(), 3, min(k, 10), 5, leaf_size=256)[0]
    flat = torch.empty(Q.numel() + 1, dtype=Q.dtype, device="cuda")
    view = flat[1:].view_as(Q)  # f32: 4 bytes past the boundary, u8: 1 byte
    view.copy_(Q)
    for nq in (3, 40, 300, most - 1, most):
        i, dist = index.query(Q[:nq], k)
        vi, vd = index.query(view[:nq], k)
        assert torch.equal(vi, i) and torch.equal(vd, dist)


def test_call_cut_into_blocks(torch):
    # lists of 32 trees and 32 neighbours: blocks of 2^26 / (32 * 32) queries
    n, d, T, k, block = 1_500, 8, 32, 32, 1 << 16
    nq = 2 * block + 5
    Z = torch.from_numpy(synth.clustered_f32(n + nq, d, n_clusters=7, seed=8)).cuda()
    index = build_index(Z[:n].contiguous(), T, 10, 5, leaf_size=512)[0]
    Q = Z[n:].contiguous()
    parts = [index.query(Q[a:a + 10_000], k) for a in range(0, nq, 10_000)]
    want = [torch.cat(p) for p in zip(*parts)]
    for q in (Q, Q.cpu().numpy()):
        got = index.query(q, k)
        assert all(np.array_equal(torch.as_tensor(g).cpu().numpy(), w.cpu().numpy())
                   for g, w in zip(got, want))
    got = index.query(Q, 1)
    assert torch.equal(got[0], want[0][:, :1]) and torch.equal(got[1], want[1][:, :1])
