"""The tensor-core leaf kernel at the edges of its shapes: K blocks per row
(dimension and precision), keys per row, leaves around its tile sizes.  One
leaf holds every point, so the build is an exact search up to the candidates
the 16-bit (8-bit) scores order wrongly.  Needs a B200."""
import numpy as np
import pytest

from drpt_b200 import build_graph, recall

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as _t
    if not _t.cuda.is_available():
        pytest.skip("no CUDA device")
    return _t


@pytest.mark.parametrize("d,precision", [
    (4, "bf16"), (64, "bf16"), (68, "bf16"), (128, "bf16"), (132, "bf16"), (256, "bf16"),
    (260, "bf16"), (704, "bf16"), (768, "bf16"), (772, "bf16"), (1024, "bf16"),
    (128, "fp8"), (256, "fp8"), (512, "fp8"), (516, "fp8"), (1024, "fp8")])
@pytest.mark.parametrize("n,nn", [(127, 10), (257, 16), (769, 20)])
def test_one_leaf(torch, n, nn, d, precision):
    rng = np.random.default_rng(n + d)
    X = rng.standard_normal((n, d)).astype(np.float32) * 10 + 100
    idx, dist, _ = build_graph(torch.from_numpy(X).cuda(), 2, nn, 1, mode="mixed", leaf_size=1024,
                               precision=precision)
    idx, dist = idx.cpu().numpy(), dist.cpu().numpy()
    assert (idx >= 0).all() and (idx != np.arange(n)[:, None]).all()
    q = np.arange(n)
    ref = np.sqrt(((X[idx].astype(np.float64) - X[q][:, None]) ** 2).sum(-1))
    assert np.allclose(dist, ref, rtol=(d + 3) * 2.0 ** -24, atol=0)
    assert (dist[:, 1:] >= dist[:, :-1]).all()
    # a list holds 1.2 to 2 times nn candidates: with scores off by 2^-9
    # (2^-4 in E4M3) of a coordinate, averaged over d of them, few of the nn
    # fall outside it; at d = 4 the scores' 10-bit keys tie
    ti, _ = recall.exact_knn_fp64(X, q, nn, device="cpu")
    assert recall.recall_at_k(idx, ti) >= (0.97 if precision == "bf16" else 0.80)
