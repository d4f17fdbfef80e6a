"""The default FP64 SOR / Gauss-Seidel solve of small and middle grids (a cell of each colour per thread) against the exchange
kernel (sor_blocking = 1), which the other tests hold to the oracle: the same bits of psi, sweep count and stop norm, at
the sizes where its tiles change (one cluster to 90 or, FMA, 112; tiles over all SMs to 530, tiles of many cells above) and one that it leaves (1300).
"""
from __future__ import annotations

import numpy as np
import pytest
from test_gpu_parity import bitwise, make_cfg

pytestmark = pytest.mark.gpu

SIZES = [5, 6, 7, 10, 17, 33, 64, 90, 91, 97, 111, 112, 113, 128, 161, 256, 257, 385, 500, 512, 530, 531, 600, 777, 1024, 1100]


def solve(cnv, n, f, **kw):
    with cnv.Cavity(make_cfg(cnv, n, **kw)) as cav:
        return cav.solver_info(), cav.poisson(f), cav.poisson(f)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kw", [{}, {"poisson_type": 1}, {"Lx": 2}, {"precision": 1}, {"precision": 1, "poisson_type": 1}],
                         ids=["sor", "gs", "rect", "fma", "fma-gs"])
def test_same_bits_as_the_exchange_kernel(cnv, n, kw):
    f = np.random.default_rng(n).standard_normal((n, n))
    for tol, itmax in ((1e-5, 60), (1e-9, 700), (30.0, 60), (1e30, 60), (1e-5, 1), (1e-30, 2), (1e-30, 7)):
        a = dict(poisson_tol=tol, poisson_max_it=itmax, **kw)
        info, (rc, psi, it, err), again = solve(cnv, n, f, **a)
        _, (rc1, psi1, it1, err1), _ = solve(cnv, n, f, sor_blocking=1, **a)
        assert "sor-cells" in info
        assert (rc, it, err) == (rc1, it1, err1), (tol, itmax)
        if rc == 0:
            assert bitwise(psi, psi1)
        assert again[0] == rc and again[2:] == (it, err) and (rc != 0 or bitwise(again[1], psi))


@pytest.mark.parametrize("n", [64, 113, 257, 560])
def test_steps_extreme_values_and_limits(cnv, n):
    """Time steps, values beyond 2^46 (the norm's FP64 part; power-of-two scaling keeps the iterates), tiny values, a solve
    that runs to infinity, and the solve after it."""
    fields = []
    for kw in ({}, {"sor_blocking": 1}):
        with cnv.Cavity(make_cfg(cnv, n, poisson_tol=1e-6, poisson_max_it=20000, **kw)) as cav:
            rc, steps = cav.step(4)
            fields.append((cav.get_fields(), [(s["iters"], s["err"], s["cont_max"]) for s in steps]))
    assert fields[0][1] == fields[1][1] and all(bitwise(a, b) for a, b in zip(fields[0][0], fields[1][0]))
    f = np.random.default_rng(n).standard_normal((n, n))
    for scale in (2.0 ** 70, 2.0 ** 50, 2.0 ** -1000, 1e-320):
        out = [solve(cnv, n, f * scale, poisson_tol=1e-4 * scale, poisson_max_it=300, **kw)[1] for kw in ({}, {"sor_blocking": 1})]
        assert out[0][0] == out[1][0] and out[0][2] == out[1][2]
        assert abs(out[0][3] - out[1][3]) <= 1e-12 * out[1][3]  # the FP64 part of the norm is summed in any order
        assert out[0][0] != 0 or bitwise(out[0][1], out[1][1])
    with cnv.Cavity(make_cfg(cnv, n, poisson_tol=1e-4, poisson_max_it=3000)) as cav:
        # psi peaks near 0.07 |f|; a sweep changes n^2 cells by about psi / n, which overflows in the sum
        assert cav.poisson(np.full((n, n), 1.7e308))[0] == cnv.CNV_NONFINITE
        ok = cav.poisson(f)
    assert ok[0] in (0, cnv.CNV_NOT_CONVERGED) and np.isfinite(ok[3])


def test_sizes_left_to_the_other_kernels(cnv):
    for n, kw in ((1300, {}), (64, {"solver_blocks": 4}), (64, {"sor_blocking": 4}), (64, {"poisson_type": 3})):
        with cnv.Cavity(make_cfg(cnv, n, **kw)) as cav:
            assert "cells" not in cav.solver_info()
