"""The forms of a query call (few queries, each reading its leaves; queries
grouped by leaf, 16 or 64 at a time) return the same lists bit for bit, at
sizes around their edges.  Needs a B200."""
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


def _brute(torch, X, Q, k):
    """k nearest rows of X by (distance, id), distances in 64 bits."""
    d = (X.double()[None] - Q.double()[:, None]).square().sum(-1).sqrt()
    v, i = torch.sort(d, dim=1, stable=True)
    return i[:, :k], v[:, :k]


@pytest.mark.parametrize("n,d,dtype,k,leaf", [
    (4_001, 4, "f32", 1, 256), (4_001, 44, "f32", 32, 256), (9_000, 132, "f32", 10, 1024),
    (3_000, 36, "u8", 16, 128), (700, 100, "u8", 7, 1024)])
def test_forms_agree(torch, n, d, dtype, k, leaf):
    nq = 1_500
    if dtype == "u8":
        Z = torch.from_numpy(synth.clustered_u8(n + nq, d, seed=3)).cuda()
    else:
        Z = torch.from_numpy(synth.clustered_f32(n + nq, d, n_clusters=7, seed=3)).cuda()
    X, Q = Z[:n].contiguous(), Z[n:].contiguous()
    Q[5] = X[17]  # an indexed row, and ties from repeated rows
    Q[6] = Q[7]
    index = build_index(X, 3, min(k, 10), 5, leaf_size=leaf)[0]
    one = [index.query(Q[i:i + 1], k) for i in range(40)]
    want_i = torch.cat([o[0] for o in one])
    want_d = torch.cat([o[1] for o in one])
    for m in (3, 40, 200, 1_500):
        i, dist = index.query(Q[:m], k)
        r = min(m, 40)
        assert torch.equal(i[:r], want_i[:r]) and torch.equal(dist[:r], want_d[:r])
    # rows that start off a 16-byte boundary take the few-queries form
    if dtype == "u8":
        flat = torch.empty(Q.numel() + 4, dtype=Q.dtype, device="cuda")
        view = flat[4:].view_as(Q)
        view.copy_(Q)
        vi, vd = index.query(view, k)
        assert torch.equal(vi, i) and torch.equal(vd, dist)
    # distances of the returned rows, sorted and distinct
    ii, dd = i.cpu().numpy(), dist.cpu().numpy()
    assert (dd[:, 1:] >= dd[:, :-1]).all()
    for q in (0, 5, 6, 1_499):
        ids = ii[q][ii[q] >= 0]
        assert len(np.unique(ids)) == len(ids)
        ref = (X[ids].double() - Q[q].double()).square().sum(1).sqrt().cpu().numpy()
        # FP32 sums of d squares in order: at most d + 3 roundings each
        assert np.allclose(dd[q][:len(ids)], ref, rtol=(d + 3) * 2.0 ** -24, atol=0)
    if n <= 1024:  # one leaf: the call is an exact search
        bi, bd = _brute(torch, X, Q[:64], k)
        assert torch.allclose(dist[:64].double(), bd, rtol=(d + 3) * 2.0 ** -24, atol=0)
