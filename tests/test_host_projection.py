"""The projection matrix's fast generator against the oracle's entry by entry
draws, bit for bit: densities that keep none, few, half and all of the entries,
sizes around its blocks of draws."""
import ctypes

import numpy as np
import pytest

import oracle
from drpt_b200 import _lib


@pytest.mark.parametrize("d,L", [(1, 1), (1, 623), (13, 48), (39, 16), (125, 5), (7, 1000), (784, 84)])
@pytest.mark.parametrize("density", [0.0, 1e-6, 1.0 / 28.0, 0.5, 1.0, 3.0, -1.0])
@pytest.mark.parametrize("seed", [0, 12345, 0xFFFFFFFF])
def test_fast_generator_is_the_oracle_matrix(d, L, density, seed):
    B = np.full((d, L), 7.0, np.float32)
    _lib.check(_lib.load().drpt_host_projection(seed, d, L, ctypes.c_float(density),
                                                B.ctypes.data))
    assert np.array_equal(B, oracle.projection_matrix(seed, d, L, density))
