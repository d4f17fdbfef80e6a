"""The direct solve of stretched cells: where an extent of the cavity in lowest terms is above 512 (a far ratio, or extents
without a common factor), the FP32 form takes its residual in 128-bit integers; up to 512 in 64 bits.

The reference and the bound are those of test_direct_refined.py.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
from test_direct import _dense_sine_solve, _rel
from test_direct_refined import TOL, solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lx,Ly", [(1, 40), (200, 3), (1, 512), (511, 512), (1, 513), (513, 1), (1000, 999), (1, 100000), (65536, 1),
                                   (2147483647, 2147483646)])
@pytest.mark.parametrize("n", [5, 64, 200, 307, 400, 1025])  # N = 4, 63, 199, 306, 399, 1024
def test_every_ratio_matches_the_dense_solve(cnv, n, Lx, Ly):
    f = np.random.default_rng(n).standard_normal((n, n))
    assert _rel(solve(cnv, f, Lx, Ly), _dense_sine_solve(f, Lx / n, Ly / n)) <= TOL
    assert _rel(solve(cnv, np.full((n, n), 0.1), Lx, Ly), _dense_sine_solve(np.full((n, n), 0.1), Lx / n, Ly / n)) <= TOL


def test_stretched_cells_do_not_fall_to_dense_products(cnv):
    """2048^2: the transforms take 1 to 2 ms, dense products 29."""
    f = np.random.default_rng(0).standard_normal((2048, 2048))
    ms = ctypes.c_double()
    with cnv.Cavity(cnv.default_config(nx=2048, ny=2048, Lx=1, Ly=513, poisson_type=cnv.POISSON_DIRECT)) as cav:
        for _ in range(2):
            assert cav.poisson(f)[0] == 0
        cav._lib.cnv_last_stats(cav._h, None, None, ctypes.byref(ms))
    assert ms.value < 12, ms.value
