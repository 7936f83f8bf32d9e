"""Learned splits at the edges of their kernels' tiles: training gradients
(128 sample rows, 16 dimensions, rows that are no multiple of 16 bytes) against
the FP64 oracle, and the projections (256 rows a block) through the queries of
a learned index, which must not depend on how a call is cut.  Needs a B200."""
import ctypes

import numpy as np
import pytest

from drpt_b200 import _lib, build_index, synth
from oracle import learned

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as _t
    if not _t.cuda.is_available():
        pytest.skip("no CUDA device")
    return _t


@pytest.mark.parametrize("S,d", [(64, 16), (65, 17), (127, 15), (128, 3), (129, 127), (255, 128),
                                 (1_025, 130), (2_049, 33), (4_100, 252)])
def test_gradient_at_tile_edges(torch, S, d):
    """FP32 sums of at most 4,100 rows with errors of 2^-24 a term stay within
    1e-4 of the largest entry (the bound of the other gradient test)."""
    rng = np.random.default_rng(7 * S + d)
    k, nodes = 6, 2
    X = rng.standard_normal((S, d)).astype(np.float32)
    node = rng.integers(0, nodes, size=S).astype(np.int32)
    nbr = rng.integers(0, S, size=(S, k)).astype(np.int32)
    nbr[:, 0] = 0  # point 0 has a pair with every other one
    W1 = (rng.standard_normal((learned.HIDDEN, d)) / np.sqrt(d)).astype(np.float32)
    b1 = (rng.standard_normal(learned.HIDDEN) * 0.1).astype(np.float32)
    w2 = (rng.standard_normal(learned.HIDDEN) / 8).astype(np.float32)
    b2 = np.float32(0.2)
    params = np.concatenate([W1.ravel(), b1, w2, [b2]]).astype(np.float32)
    grad, loss = np.zeros_like(params), ctypes.c_float()
    _lib.check(_lib.load().drpt_learn_gradient(
        _lib.context(0).handle, X.ctypes.data, S, d, params.ctypes.data, node.ctypes.data,
        nbr.ctypes.data, k, grad.ctypes.data, ctypes.byref(loss)))
    L, dW1, db1, dw2, db2 = learned.loss_and_grad(X, W1, b1, w2, b2, node, nbr)
    want = np.concatenate([dW1.ravel(), db1, dw2, [db2]])
    assert abs(loss.value - L) <= 1e-5 * abs(L)
    assert np.abs(grad - want).max() <= 1e-4 * np.abs(want).max()


@pytest.mark.parametrize("n,d", [(5_000, 256), (4_999, 36), (4_097, 132)])
def test_projections_do_not_depend_on_the_cut(torch, n, d):
    X = torch.from_numpy(synth.latent_manifold_f32(n + 600, d, seed=2)).cuda()
    index = build_index(X[:n].contiguous(), 4, 5, 9, mode="mixed", leaf_size=256,
                        learned_trees=3, learn_sample=1_024, learn_iters=2)[0]
    Q = X[n:].contiguous()
    ids, dist = index.query(Q, 5)[:2]
    for cut in (1, 127, 128, 129, 255, 256, 257):
        a = index.query(Q[:cut].contiguous(), 5)[:2]
        b = index.query(Q[cut:].contiguous(), 5)[:2]
        assert torch.equal(torch.cat([a[0], b[0]]), ids)
        assert torch.equal(torch.cat([a[1], b[1]]), dist)
