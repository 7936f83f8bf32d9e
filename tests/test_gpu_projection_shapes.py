"""The projection kernel at the edges of its blocks (points a block by the
dimension, ragged points and dimensions, columns with few or all entries, rows
off 16-byte boundaries): P bit for bit the CPU oracle's ordered sums.  Needs a
B200."""
import numpy as np
import pytest

import oracle
from drpt_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as _t
    if not _t.cuda.is_available():
        pytest.skip("no CUDA device")
    return _t


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dtype", ["f32", "u8"])
@pytest.mark.parametrize("n,d", [
    (1, 1), (31, 3), (128, 4), (130, 36), (4_800, 225), (18_945, 228), (9_475, 452), (9_476, 456),
    (333, 904), (334, 908), (65, 1_816), (66, 1_820), (17, 3_632), (19, 7_263)])
def test_projection_is_the_ordered_sum(torch, n, d, dtype, offset):
    rng = np.random.default_rng(3 * n + d)
    L = 37
    if dtype == "u8":
        X = rng.integers(0, 256, size=(n, d), dtype=np.uint8)
    else:
        X = (rng.standard_normal((n, d)) * 3).astype(np.float32)
    B = rng.standard_normal((d, L)).astype(np.float32)
    B[rng.random((d, L)) > rng.random(L)[None] ** 2] = 0.0  # 0 to all entries a column
    B[:, 5] = 0.0
    cols = np.array([q for q in range(L) if q != 11], np.int32)
    flat = torch.empty(n * d + offset, dtype=torch.uint8 if dtype == "u8" else torch.float32,
                       device="cuda")
    flat[offset:] = torch.from_numpy(X.reshape(-1)).cuda()
    P = torch.full((len(cols), n), float("nan"), dtype=torch.float32, device="cuda")
    _lib.check(_lib.load().drpt_project(
        _lib.context(0).handle, flat[offset:].data_ptr(), n, d, 1 if dtype == "u8" else 0,
        B.ctypes.data, L, cols.ctypes.data, len(cols), P.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    want = np.ascontiguousarray(oracle.project(X, B)[:, cols].T)
    assert np.array_equal(P.cpu().numpy(), want)
