"""Waits of the default solvers that run out: with the testing-only field test_stall_block one block never publishes
(or never arrives at the grid barrier), so the others' bounded waits end after solver_timeout_ms. The call must return
CNV_TIMEOUT from cnv_step and from cnv_poisson, every time, and a solve on a fresh handle must be right afterwards.
"""
from __future__ import annotations

import time

import numpy as np
import pytest
from test_gpu_parity import make_cfg

pytestmark = pytest.mark.gpu

SOLVERS = [
    (64, dict(poisson_type=4)),   # sine transforms in FP64, one launch
    (400, dict(poisson_type=4)),  # in FP32 with corrections, one launch
    (64, {}),                     # SOR, a cell of each colour per thread: one cluster, mailboxes in shared memory
    (256, {}),                    # mailboxes in global memory
    (500, dict(precision=1)),     # FMA
    (300, dict(poisson_type=1)),  # Gauss-Seidel
    (600, {}),                    # tiles of many cells
    (1024, {}),
    (128, dict(precision=2)),     # mixed: halo cells with their epoch
    (1500, dict(precision=2)),    # flags
]


@pytest.mark.parametrize("n,kw", SOLVERS, ids=[f"{n}-{'-'.join(f'{k}{v}' for k, v in kw.items()) or 'sor'}" for n, kw in SOLVERS])
def test_a_block_that_never_publishes_is_reported(cnv, n, kw):
    f = np.random.default_rng(n).standard_normal((n, n))
    limits = dict(poisson_tol=1e-9, poisson_max_it=200000, **kw)
    with cnv.Cavity(make_cfg(cnv, n, **limits)) as cav:
        rc, want, it, err = cav.poisson(f)
    assert rc == 0
    with cnv.Cavity(make_cfg(cnv, n, solver_timeout_ms=50, test_stall_block=1 + 3, **limits)) as cav:
        t0 = time.perf_counter()
        for _ in range(2):
            assert cav.poisson(f)[0] == cnv.CNV_TIMEOUT
            rc, steps = cav.step(2, raise_on_error=False)
            assert rc == cnv.CNV_TIMEOUT and [s["status"] for s in steps] == [cnv.CNV_TIMEOUT] * 2
        assert time.perf_counter() - t0 < 30
    with cnv.Cavity(make_cfg(cnv, n, **limits)) as cav:
        rc, psi, it2, err2 = cav.poisson(f)
    assert (rc, it2, err2) == (0, it, err) and np.array_equal(psi, want)


@pytest.mark.parametrize("n", [64, 400])
def test_a_forward_run_that_gave_up_cannot_be_differentiated(cnv, n):
    h = 1.0 / n
    cfg = cnv.default_config(nx=n, ny=n, Re=400.0, dt=0.2 * min(h * h * 100.0, h), solver_timeout_ms=50, test_stall_block=1 + 3)
    w0 = cnv.noise_field(n, seed=5, sigma=1.0, passes=4)
    with cnv.Adjoint(cfg, 2) as adj:
        t0 = time.perf_counter()
        for _ in range(2):
            with pytest.raises(cnv.CnvError) as e:
                adj.forward(w0, 1.0, 3)
            assert e.value.status == cnv.CNV_TIMEOUT
            with pytest.raises(cnv.CnvError) as e:
                adj.backward(w0)
            assert e.value.status == cnv.CNV_BAD_ARG
        assert time.perf_counter() - t0 < 1.0  # solver_timeout_ms, not the default of two seconds
