"""Folding a tree's lists into the running ones: the form for many points (a
thread per point, lists turned through shared memory) against the one for few
(a lane per entry).  A batch of small sets folds all of them at once; each set
alone is small.  Ties from repeated rows; point counts off multiples of 32.
Needs a B200."""
import numpy as np
import pytest

from drpt_b200 import build_graph, build_graph_batched

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nn,width,sets,rows", [
    (10, 16, 11, 1_501), (5, 16, 3, 5_463), (16, 32, 9, 931), (20, 32, 5, 1_733)])
def test_many_points_fold_like_few(nn, width, sets, rows):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(nn + rows)
    X = rng.integers(-3, 4, size=(sets * rows, 32)).astype(np.float32)
    X[1::7] = X[::7][: len(X[1::7])]  # every seventh row stands twice
    assert len(X) * width > 1 << 18 and rows * width <= 1 << 18
    offs = rows * np.arange(sets + 1)
    Xd = torch.from_numpy(X).cuda()
    idx, dist, _ = build_graph_batched(Xd, offs, 4, nn, 3, leaf_size=256)
    for s in range(sets):
        part = slice(s * rows, (s + 1) * rows)
        i1, d1, _ = build_graph(Xd[part].contiguous(), 4, nn, 3, mode="mixed", leaf_size=256)
        assert torch.equal(idx[part], i1) and torch.equal(dist[part], d1), s
