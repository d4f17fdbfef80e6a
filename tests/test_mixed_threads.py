"""Two threads, each with a mixed cavity of its own size on the same kernel: the shared-memory limit belongs to the
kernel, not to a cavity, so one thread's launch must not lower it under the other's."""
from __future__ import annotations

import threading

import numpy as np
import pytest
from test_gpu_parity import make_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1100, 1440), (2300, 33)], ids=["registers", "shared-memory"])
def test_cavities_of_two_sizes_in_two_threads(cnv, sizes):
    done, failed = set(), []

    def run(n):
        f = np.random.default_rng(n).standard_normal((n, n))
        with cnv.Cavity(make_cfg(cnv, n, precision=cnv.PREC_MIXED, mixed_inner_sweeps=8, mixed_max_outer=1)) as cav:
            for k in range(20000):
                if k == 150:
                    done.add(n)
                if failed or len(done) == 2:  # the quicker thread goes on until the other is done
                    return
                rc = cav.poisson(f)[0]
                if rc not in (cnv.CNV_OK, cnv.CNV_NOT_CONVERGED):
                    failed.append((n, rc, cnv.last_error()))

    threads = [threading.Thread(target=run, args=(n,)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
