"""The direct solve's forms: FP64 at once on small grids, FP32 transforms with exact integer residuals above,
in one launch or a launch per pass, for every kind of FFT radix, stretched cells and extreme scales.

The reference is the dense sine-transform solve in numpy FP64 (products of orthonormal matrices: an error of
about sqrt(n) units of rounding, 1e-14 at 1500^2), so 1e-13 normwise is the bound, as for the dense comparison
of test_direct.py; a form that lost one correction would be off by 1e-11 or more.
"""
from __future__ import annotations

import numpy as np
import pytest
from test_direct import _dense_sine_solve, _rel

pytestmark = pytest.mark.gpu
TOL = 1e-13


def solve(cnv, f, Lx=1, Ly=1):
    n = f.shape[0]
    with cnv.Cavity(cnv.default_config(nx=n, ny=n, Lx=Lx, Ly=Ly, poisson_type=cnv.POISSON_DIRECT)) as cav:
        rc, psi, _, _ = cav.poisson(f)
    assert rc == 0
    return psi


@pytest.mark.parametrize("n,Lx,Ly", [
    (5, 1, 1), (6, 1, 1), (12, 1, 1), (18, 1, 1), (33, 1, 1), (98, 1, 1), (129, 1, 1),  # N = 4, 5, 11, 17, 32, 97, 128
    (132, 1, 1), (138, 1, 1),    # N = 131, 137: the last tabulated radix, the first without a matrix
    (80, 1, 1), (84, 1, 1), (159, 1, 1), (203, 1, 1), (200, 1, 40), (294, 1, 1),  # N = 79, 83, 158, 202, 199, 293: by radix
    (306, 1, 1), (307, 1, 1), (308, 1, 1),  # either side of the FP64 form's last size
    (514, 1, 1), (1026, 1, 1),   # N = 513 = 3^3 19, 1025 = 5^2 41
    (1302, 1, 1), (1303, 1, 1),  # the last size in one launch, the first launch per pass
    (1500, 1, 1),                # N = 1499, prime
    (96, 3, 2), (400, 2, 1), (400, 1, 40),
])
def test_every_form_matches_the_dense_solve(cnv, n, Lx, Ly):
    rng = np.random.default_rng(n)
    f = rng.standard_normal((n, n))
    f[n // 2] *= 1e4  # rows of very different size
    assert _rel(solve(cnv, f, Lx, Ly), _dense_sine_solve(f, Lx / n, Ly / n)) <= TOL


@pytest.mark.parametrize("n", [64, 400])
@pytest.mark.parametrize("scale", [2.0 ** -900, 2.0 ** -200, 2.0 ** 700])
def test_scaling_by_a_power_of_two(cnv, n, scale):
    f = np.random.default_rng(n).standard_normal((n, n))
    assert np.array_equal(solve(cnv, f * scale), solve(cnv, f) * scale)


@pytest.mark.parametrize("n", [64, 400])
def test_zero_point_and_smooth_right_hand_sides(cnv, n):
    assert not solve(cnv, np.zeros((n, n))).any()
    f = np.zeros((n, n))
    f[n // 3, n // 2] = -2.0
    assert _rel(solve(cnv, f), _dense_sine_solve(f, 1 / n, 1 / n)) <= TOL
    x = np.arange(n) / (n - 1)
    f = np.outer(np.sin(np.pi * x), np.sin(2 * np.pi * x))
    assert _rel(solve(cnv, f), _dense_sine_solve(f, 1 / n, 1 / n)) <= TOL


def test_plans_of_two_sizes_alternate(cnv):
    """A small plan made after a large one leaves the large one's launches as they were."""
    f = {n: np.random.default_rng(n).standard_normal((n, n)) for n in (2048, 64)}
    cavs = {n: cnv.Cavity(cnv.default_config(nx=n, ny=n, poisson_type=cnv.POISSON_DIRECT)) for n in (2048, 64)}
    first = {n: cavs[n].poisson(f[n]) for n in (2048, 64)}
    again = {n: cavs[n].poisson(f[n]) for n in (2048, 64)}
    for n in f:
        assert first[n][0] == 0 and again[n][0] == 0 and np.array_equal(first[n][1], again[n][1])
        cavs[n].close()
