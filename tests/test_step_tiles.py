"""The passes around the solve on grids with cells that take the short sums (all seven taps inside the grid) and cells that do
not, tiles whole and ragged, every order, equal and unequal spacing: the oracle's bits.
"""
from __future__ import annotations

import pytest
from test_gpu_parity import bitwise, make_cfg, run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,Lx,order", [(70, 1, 6), (101, 1, 4), (200, 1, 6), (200, 2, 6), (133, 1, 2), (97, 3, 6)])
def test_steps_with_inner_tiles_equal_the_oracle(cnv, orc, n, Lx, order):
    cfg = make_cfg(cnv, n, Lx=Lx, order=order, poisson_tol=1e-4, poisson_max_it=100000, dt=1e-4)
    g, gs, o, os_ = run_both(cnv, orc, cfg, 3)
    for name, a, b in zip("w u v psi".split(), g, o):
        assert bitwise(a, b), name
    assert [(s["iters"], s["cont_max"], s["cont_min"]) for s in gs] == [(s["iters"], s["cont_max"], s["cont_min"]) for s in os_]
