"""The leaf kernel one row before and at the line between its shapes for wide rows
(the K blocks past the fourth x mean leaf size): the lists and, by the kernel that
runs, the side.  Needs a B200."""
import numpy as np
import pytest

from drpt_b200 import build_graph
from tests.test_gpu_leaf_wide import test_one_large_leaf as check_one_large_leaf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n", [(512, 1_750), (576, 1_400), (640, 1_167), (704, 1_000)])
@pytest.mark.parametrize("nn", [10, 20])
def test_both_sides(d, n, nn):
    torch = pytest.importorskip("torch")
    from torch.profiler import ProfilerActivity, profile
    X = torch.from_numpy(np.random.default_rng(d).standard_normal((n, d)).astype(np.float32))
    for m, shape in ((n - 1, 2), (n, 3)):
        check_one_large_leaf(d, "bf16", m, nn)
        rows = X[:m].cuda()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            build_graph(rows, 2, nn, 1, mode="mixed", leaf_size=4096)
            torch.cuda.synchronize()
        names = {e.name for e in p.events()}
        if not any("k_" in e for e in names):
            pytest.skip("no kernel trace on this machine")
        names = {e for e in names if "k_leaf_mma" in e}
        assert len(names) == 1 and f"k_leaf_mma<{16 if nn == 10 else 32}, {shape}, " in names.pop()
