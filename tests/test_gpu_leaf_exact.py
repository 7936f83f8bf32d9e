"""The exact leaf brute force (drpt_leaf_knn) at the edges of its kernels' leaf
classes, list widths and row alignments, bit for bit against the same FP32
operation sequence in NumPy.  Needs a B200."""
import numpy as np
import pytest

from drpt_b200 import _lib

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 4, 5, 33, 64, 67, 68, 69, 95, 96, 97, 127, 128, 129, 256, 300)


@pytest.fixture(scope="module")
def torch():
    import torch as _t
    if not _t.cuda.is_available():
        pytest.skip("no CUDA device")
    return _t


def _distances(rows):
    x = rows.astype(np.float32)
    acc = np.zeros((len(x), len(x)), np.float32)
    for i in range(x.shape[1]):  # one rounded subtract, multiply and add per dimension
        df = x[:, i][None, :] - x[:, i][:, None]
        acc += df * df
    return np.sqrt(acc)


@pytest.mark.parametrize("d,dtype,offset,k", [
    (128, "f32", 0, 10), (32, "f32", 0, 32), (33, "f32", 0, 10), (64, "f32", 1, 7),
    (784, "u8", 0, 10), (30, "u8", 0, 1), (48, "u8", 3, 12), (40, "f32", 0, 33)])
def test_leaf_classes(torch, d, dtype, offset, k):
    rng = np.random.default_rng(d + k)
    n = sum(SIZES)
    if dtype == "u8":  # small integers: many equal distances
        X = rng.integers(0, 4, (n, d)).astype(np.uint8)
    else:
        X = (rng.standard_normal((n, d)) * 20).astype(np.float32)
        X[7:12] = X[3]  # repeated rows: zero distances, ties by index
    order = np.stack([rng.permutation(n), np.arange(n)]).astype(np.int32)
    offs = np.concatenate([[0], np.cumsum(SIZES)]).astype(np.int32)
    offs = np.stack([offs, offs])
    # rows from `offset` elements into their buffer (off the 16-byte boundary)
    flat = torch.empty(n * d + offset, dtype=torch.uint8 if dtype == "u8" else torch.float32,
                       device="cuda")
    Xd = flat[offset:]
    Xd.copy_(torch.from_numpy(X).reshape(-1))
    ci = torch.empty((n, 2, k), dtype=torch.int32, device="cuda")
    cd = torch.empty((n, 2, k), dtype=torch.float32, device="cuda")
    od, fd = torch.from_numpy(order).cuda(), torch.from_numpy(offs).cuda()
    _lib.check(_lib.load().drpt_leaf_knn(
        _lib.context(0).handle, Xd.data_ptr(), _lib.DTYPE_U8 if dtype == "u8" else _lib.DTYPE_F32,
        n, d, 2, od.data_ptr(), fd.data_ptr(), len(SIZES), k, ci.data_ptr(), cd.data_ptr(), 0))
    torch.cuda.synchronize()
    ci, cd = ci.cpu().numpy(), cd.cpu().numpy()
    for t in range(2):
        for f, m in enumerate(SIZES):
            ids = order[t, offs[t, f]:offs[t, f] + m]
            D = _distances(X[ids])
            for r in range(m):
                o = np.lexsort((ids, D[r]))
                o = o[o != r][:k]
                want_i = np.full(k, -1, np.int32)
                want_d = np.full(k, np.inf, np.float32)
                want_i[:len(o)], want_d[:len(o)] = ids[o], D[r][o]
                assert np.array_equal(ci[ids[r], t], want_i), (t, m, r)
                assert np.array_equal(cd[ids[r], t], want_d), (t, m, r)
