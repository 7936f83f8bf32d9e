"""The size limit of drpt_global_trees_noalloc.  A build may take 64 MiB of the
static scratch, counted by the layout restated here; what a refusal reports is
checked on the CPU, the largest accepted sizes are built on the GPU and compared
bit for bit with drpt_global_trees."""
import ctypes

import pytest

from drpt_b200 import _lib

LIMIT = 64 << 20


def _bytes(n, T, gd):
    """The layout: 256-byte aligned pieces, in order."""
    deep, last = gd >= 3, gd - 2
    G = T << last
    U = T * (-(-n // 4096) + (1 << last))
    pieces = [4 * T * n] * 3 + [4 * T * ((1 << gd - 1) + 1)] if deep else []
    pieces += [4 * (G + 1), 4 * U, 4 * U, 4, 64 * G, 16 * U, 64 * U, 4 * G, 4 * U, 4 * U, 4 * G]
    used = 0
    for p in pieces:
        used = (used + 255) // 256 * 256 + p
    return used


def _largest(T, gd):
    lo, hi = 2, 1 << 24
    while lo < hi:
        m = (lo + hi + 1) // 2
        lo, hi = (m, hi) if _bytes(m, T, gd) <= LIMIT else (lo, m - 1)
    return lo


@pytest.mark.parametrize("T,gd", [(1, 6), (5, 4), (16, 8), (3, 18), (64, 12)])
def test_refusal_names_the_limit(T, gd):
    # (the size check comes before any CUDA call and before the pointers are used)
    n = _largest(T, gd) + 1
    L = _lib.load()
    assert L.drpt_global_trees_noalloc(256, n, T, gd, 0, 256, 256, None, ctypes.c_void_p(0)) == 1
    msg = L.drpt_last_error().decode()
    assert f"needs {_bytes(n, T, gd)} bytes" in msg and f"gets {LIMIT} " in msg


@pytest.mark.gpu
@pytest.mark.parametrize("T,gd", [(1, 6), (5, 4)])
def test_largest_accepted_build(T, gd):
    import torch
    n = _largest(T, gd)
    P = torch.randn(T * (gd - 1), n, generator=torch.Generator(device="cuda").manual_seed(T),
                    device="cuda")
    out = [[torch.full((T, n), -7, dtype=torch.int32, device="cuda"),
            torch.full((T, (1 << gd - 1) + 1), -7, dtype=torch.int32, device="cuda"),
            torch.zeros((T, (1 << gd - 1) - 1), device="cuda")] for _ in range(2)]
    L, s = _lib.load(), torch.cuda.current_stream().cuda_stream
    _lib.check(L.drpt_global_trees_noalloc(P.data_ptr(), n, T, gd, 0,
                                           *[o.data_ptr() for o in out[0]], s))
    _lib.check(L.drpt_global_trees(_lib.context(0).handle, P.data_ptr(), n, T, gd, 0,
                                   *[o.data_ptr() for o in out[1]], s))
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(*out))
