"""A batch of cavities below 24^2 runs a kernel of its own (scalar sweeps, FP64 multiplications); with a larger one among
them they run the general kernel (vector sweeps, integer multiplications). The same bits either way."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{}, {"order": 2}, {"mixed_warm_start": 1}], ids=["order6", "order2", "warm"])
def test_small_batches_equal_the_general_kernel(cnv, kw):
    small = [dict(n=n, Re=100.0 * n, lid=1.0) for n in (5, 6, 8, 13, 16, 22, 23)]
    runs = []
    for specs in (small, small + [dict(n=24, Re=400.0, lid=1.0)]):
        with cnv.Batch(cnv.default_config(mixed_rtol=1e-10, **kw), specs) as bt:
            rc, last = bt.step(3)
            assert rc == 0
            runs.append(([bt.get_fields(k) for k in range(len(small))], [x["iters"] for x in last[:len(small)]]))
    assert runs[0][1] == runs[1][1]
    for a4, b4 in zip(runs[0][0], runs[1][0]):
        for a, b in zip(a4, b4):
            assert np.array_equal(a.view(np.uint64), b.view(np.uint64))
