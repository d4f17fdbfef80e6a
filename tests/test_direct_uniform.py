"""The direct solve of right-hand sides in which many cells hold one value: whatever is rounded off a cell is rounded off
all of them, and the answer is up to 0.07 n^2 times the right-hand side, so it must not be lost.

The reference is the dense FP64 solve, twice corrected by its residual in long double. The bound is 1e-14 of the
largest value: FP64 transforms of these lengths leave 2e-15 .. 4e-14, and a right-hand side held to 2^-58 of the largest psi
alone would leave 1.4e-14 at 400^2 and 2.3e-13 at 2048^2.
"""
from __future__ import annotations

import numpy as np
import pytest
from test_direct import _dense_sine_solve, _rel
from test_direct_refined import solve

pytestmark = pytest.mark.gpu
TOL = 1e-14


def refined_solve(f, dx, dy):
    wide = np.longdouble
    c4, dx2, dy2 = dx * dx * dy * dy, wide(dx * dx), wide(dy * dy)
    psi = _dense_sine_solve(f, dx, dy).astype(wide)
    for _ in range(2):
        a = 2 * (dx2 + dy2) * psi[1:-1, 1:-1] - dy2 * (psi[2:, 1:-1] + psi[:-2, 1:-1]) - dx2 * (psi[1:-1, 2:] + psi[1:-1, :-2])
        r = np.zeros_like(f)
        r[1:-1, 1:-1] = f[1:-1, 1:-1] + a / wide(c4)
        psi += _dense_sine_solve(r, dx, dy)
    return psi


def fields(n):
    y, x = np.mgrid[0:n, 0:n] / n
    yield "constant", np.full((n, n), 0.1)
    yield "disc", np.where((x - 0.4) ** 2 + (y - 0.5) ** 2 < 0.04, -0.3, 0.0)
    f = np.full((n, n), 1e-40)  # far below one unit
    f[n // 3, n // 2] = -2.0
    yield "point", f


@pytest.mark.parametrize("n,Lx", [(64, 1), (200, 1), (400, 1), (400, 3), (1024, 1), (1500, 1), (2048, 1)])
def test_equal_cells_lose_nothing(cnv, n, Lx):
    for name, f in fields(n):
        assert _rel(solve(cnv, f, Lx, 1), refined_solve(f, Lx / n, 1 / n)) <= TOL, name
