"""The global-tree levels at the edges of their units (4,096 positions): one
unit per node, nodes around one and two units, empty nodes, in the exact and
the fast form.  Needs a B200."""
import numpy as np
import pytest

from drpt_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as _t
    if not _t.cuda.is_available():
        pytest.skip("no CUDA device")
    return _t


def _trees(torch, P, T, gd, exact):
    n = P.shape[1]
    nleaf = 1 << (gd - 1)
    Pd = torch.from_numpy(P).cuda()
    order = torch.empty((T, n), dtype=torch.int32, device="cuda")
    offs = torch.empty((T, nleaf + 1), dtype=torch.int32, device="cuda")
    med = torch.empty((T, nleaf - 1), dtype=torch.float32, device="cuda")
    _lib.check(_lib.load().drpt_global_trees(_lib.context(0).handle, Pd.data_ptr(), n, T, gd,
                                             exact, order.data_ptr(), offs.data_ptr(),
                                             med.data_ptr(), 0))
    torch.cuda.synchronize()
    return order.cpu().numpy(), offs.cpu().numpy(), med.cpu().numpy()


@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("n", [2, 31, 4_095, 4_096, 4_097, 8_192, 8_193, 40_001])
@pytest.mark.parametrize("T,gd", [(1, 2), (3, 5), (2, 8)])
def test_levels_follow_their_medians(torch, n, T, gd, exact):
    """Each node splits stably at its stored median: the partition replayed on
    the CPU from the medians gives the same order and offsets."""
    rng = np.random.default_rng(n + gd)
    P = rng.standard_normal((T * (gd - 1), n)).astype(np.float32)
    P[-1, :] = 0.25  # one level of equal values: nodes of its tree stay whole, siblings empty
    order, offs, med = _trees(torch, P, T, gd, exact)
    for t in range(T):
        nodes = [np.arange(n, dtype=np.int32)]
        for lv in range(gd - 1):
            split = []
            for s, ids in enumerate(nodes):
                m = med[t, (1 << lv) - 1 + s]
                v = P[t * (gd - 1) + lv, ids]
                with np.errstate(invalid="ignore"):
                    left = v <= m
                split += [ids[left], ids[~left]]
            nodes = split
        want = np.concatenate(nodes)
        sizes = np.array([len(x) for x in nodes])
        assert np.array_equal(offs[t], np.concatenate([[0], np.cumsum(sizes)]))
        assert np.array_equal(order[t], want)


@pytest.mark.parametrize("n", [4_096, 4_097, 20_011])
def test_values_decide_not_the_form(torch, n):
    """The same values repeated over the trees give the same tree in each."""
    rng = np.random.default_rng(n)
    col = rng.standard_normal((4, n)).astype(np.float32) * 100
    P = np.concatenate([col, col, col])
    for exact in (0, 1):
        order, offs, med = _trees(torch, P, 3, 5, exact)
        for t in (1, 2):
            assert np.array_equal(order[0], order[t]) and np.array_equal(offs[0], offs[t])
            assert med[0].tobytes() == med[t].tobytes()
