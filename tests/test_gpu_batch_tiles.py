"""A batch takes the leaf kernel's tiles by the mean size of its datasets' leaves,
as their builds alone do, and not by the mean over the batch's leaf slots, most of
which are empty where sizes differ.  Needs a B200."""
import numpy as np
import pytest

from drpt_b200 import build_graph, build_graph_batched, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as _t
    if not _t.cuda.is_available():
        pytest.skip("no CUDA device")
    return _t


def _leaf_kernels(torch, call):
    from torch.profiler import ProfilerActivity, profile
    call()  # (the first call allocates)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    names = {e.name for e in p.events()}
    if not any("k_" in n for n in names):
        pytest.skip("no kernel trace on this machine")
    return {n for n in names if "k_leaf_mma" in n}


@pytest.mark.parametrize("d,big", [(704, 12_000), (704, 6_000), (512, 16_000)])
def test_tiles_of_a_batch(torch, d, big):
    sizes = [big, 1_900, 1_900, 1_900]  # leaves of 1,500 or 2,000 and of 1,900
    X = torch.from_numpy(synth.clustered_f32(sum(sizes), d, n_clusters=9, seed=2)).cuda()
    offs = np.concatenate([[0], np.cumsum(sizes)])
    kw = dict(leaf_size=2048)
    alone = _leaf_kernels(torch, lambda: build_graph(X[:big], 2, 10, 3, mode="mixed", **kw))
    batch = _leaf_kernels(torch, lambda: build_graph_batched(X, offs, 2, 10, 3, **kw))
    assert len(alone) == 1 and batch == alone
