"""The leaf kernel on both sides of the line between its shapes for wide rows
(K blocks x mean leaf size): one leaf, so the lists are the leaf's nearest
neighbours.  Needs a B200."""
import numpy as np
import pytest

from drpt_b200 import build_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,precision,n", [
    (512, "bf16", 1_870), (512, "bf16", 1_880), (640, "bf16", 1_499), (640, "bf16", 1_505),
    (960, "fp8", 1_870), (960, "fp8", 1_880), (448, "bf16", 2_500)])
@pytest.mark.parametrize("nn", [10, 20])
def test_one_large_leaf(d, precision, n, nn):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(n + d)
    X = torch.from_numpy((rng.standard_normal((n, d)) * 10 + 100).astype(np.float32)).cuda()
    idx, dist, _ = build_graph(X, 2, nn, 1, mode="mixed", leaf_size=4096, precision=precision)
    D = torch.cdist(X.double(), X.double(), compute_mode="donot_use_mm_for_euclid_dist")
    D.fill_diagonal_(float("inf"))
    got = D.gather(1, idx.long())
    # FP32 distances: at most d + 3 roundings
    assert torch.allclose(dist.double(), got, rtol=(d + 3) * 2.0 ** -24, atol=0)
    want = D.topk(nn, dim=1, largest=False).values
    # squared distances are 200 d +- 10 sqrt(8 d) 10; scores with relative
    # coordinate errors of 2^-9 (2^-4 in E4M3) move them by about 2^-9 (2^-4) of
    # 200 sqrt(d): lists lie within four such steps of the true ones
    step = 4 * (2.0 ** -4 if precision == "fp8" else 2.0 ** -9) * 200 * d ** 0.5
    assert (got ** 2 <= want[:, -1:] ** 2 + step).all()
