"""Builds on device rows that start off the boundary which the whole-leaf forms read
from (16 bytes, 8-bit rows 4): the graphs are those of the same rows elsewhere.  Needs
a B200."""
import numpy as np
import pytest

from drpt_b200 import build_graph, build_graph_batched, build_index, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as _t
    if not _t.cuda.is_available():
        pytest.skip("no CUDA device")
    return _t


def _rows(torch, n, d, dtype):
    X = synth.clustered_u8(n, d, seed=3) if dtype == "u8" else \
        synth.clustered_f32(n, d, n_clusters=7, seed=3)
    X = torch.from_numpy(X).cuda()
    off = torch.empty(X.numel() + 1, dtype=X.dtype, device="cuda")[1:].view_as(X)
    off.copy_(X)
    return X, off


@pytest.mark.parametrize("kw", [dict(mode="mixed"), dict(mode="mixed", precision="fp8"),
                                dict(mode="fp32_gram"), dict(mode="fp32_leaf"),
                                dict(mode="mixed", learned_trees=1, learn_iters=2)])
@pytest.mark.parametrize("dtype,d", [("f32", 40), ("u8", 104)])
def test_rows_off_the_boundary(torch, kw, dtype, d):
    X, off = _rows(torch, 4_001, d, dtype)
    want = build_graph(X, 3, 10, 5, leaf_size=512, **kw)[:2]
    got = build_graph(off, 3, 10, 5, leaf_size=512, **kw)[:2]
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("dtype,d", [("f32", 40), ("u8", 104)])
def test_batches_and_indexes(torch, dtype, d):
    X, off = _rows(torch, 6_000, d, dtype)
    offs = np.array([0, 1_000, 4_001, 6_000])
    for kw in (dict(), dict(use_graph=True), dict(use_graph=True), dict(mode="fp32_leaf")):
        out = (torch.empty((6_000, 10), dtype=torch.int32, device="cuda"),
               torch.empty((6_000, 10), device="cuda"))
        want = build_graph_batched(X, offs, 3, 10, 5, leaf_size=512, **kw)[:2]
        build_graph_batched(off, offs, 3, 10, 5, leaf_size=512, out=out, **kw)
        assert torch.equal(out[0], want[0]) and torch.equal(out[1], want[1])
    index = build_index(off, 3, 10, 5, leaf_size=512)[0]
    q = build_index(X, 3, 10, 5, leaf_size=512)[0].query(X[:700].contiguous(), 10)
    got = index.query(X[:700].contiguous(), 10)
    assert torch.equal(got[0], q[0]) and torch.equal(got[1], q[1])
