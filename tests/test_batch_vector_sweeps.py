"""The batch's vector sweeps at sizes where their vectors, runs of rows and shared-memory placement change: fewer cells
than a vector, odd and even rows, R/den in shared memory (up to 120^2), the largest cavities of one block (239^2,
240^2), strips. Each cavity must equal its single-cavity run, which uses other kernels, as in test_batch.py
(1e-12 normwise, the same number of corrections)."""
from __future__ import annotations

import numpy as np
import pytest
from test_batch import SAME_SCHEME_TOL, _single_mixed

pytestmark = pytest.mark.gpu
SIZES = [5, 7, 8, 9, 17, 41, 65, 119, 121, 130, 193, 239, 240, 241, 257, 385]


@pytest.mark.parametrize("split", [None, 4])
def test_vector_sweeps_equal_single_cavity_runs(cnv, split):
    specs = [dict(n=n, Re=300.0 + n, lid=1.0) for n in SIZES]
    with cnv.Batch(cnv.default_config(mixed_rtol=1e-10), specs) as bt:
        if split:
            bt.split(split, 1)
        rc, last = bt.step(2)
        fields = [bt.get_fields(k) for k in range(len(specs))]
    assert rc == 0
    for k, sp in enumerate(specs):
        steps, single = _single_mixed(cnv, sp, 2)
        assert last[k]["iters"] == steps[-1]["iters"], sp
        for name, a, b in zip("w u v psi".split(), fields[k], single):
            assert np.max(np.abs(a - b)) <= SAME_SCHEME_TOL * np.max(np.abs(b)), (sp, name)
