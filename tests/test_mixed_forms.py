"""The register form of the mixed solve at the sizes where its boxes, patches and walls change: the smallest grids it
takes, odd and even ones (the right wall in an odd or even column of a patch, or between patches: n - 2 a multiple
of 8), each patch height, and the sizes it leaves to the shared-memory form (33, 2500).

Each solve must meet the stop rule by an independent FP64 residual, and agree with the exact solve: a relative residual
of r leaves at most r |g| / lambda_min, about r n times the solution for a right-hand side of noise, so 1e-10 n.
"""
from __future__ import annotations

import numpy as np
import pytest
from test_gpu_parity import MIXED_RTOL, fp64_residual, make_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,Lx", [(33, 1), (50, 1), (51, 1), (66, 1), (97, 2), (128, 1), (131, 1), (200, 1), (257, 1),
                                  (514, 1), (1025, 1), (1101, 1), (1300, 1), (1501, 2), (2050, 1), (2201, 1), (2500, 1)])
def test_every_form_reaches_the_residual_and_the_exact_answer(cnv, n, Lx):
    f = np.random.default_rng(n).standard_normal((n, n))
    with cnv.Cavity(make_cfg(cnv, n, Lx=Lx, precision=cnv.PREC_MIXED, mixed_rtol=MIXED_RTOL)) as cav:
        rc, psi, _, rel = cav.poisson(f)
        assert rc == 0 and rel <= MIXED_RTOL
        rc, again, _, rel2 = cav.poisson(f)  # the exchanged cells of the first solve are not taken for the second's
        assert rc == 0 and rel2 == rel and np.array_equal(again, psi)
    assert fp64_residual(psi, f, Lx=Lx) <= 1.05 * MIXED_RTOL
    assert not (psi[0].any() or psi[-1].any() or psi[:, 0].any() or psi[:, -1].any())
    with cnv.Cavity(make_cfg(cnv, n, Lx=Lx, poisson_type=cnv.POISSON_DIRECT)) as cav:
        _, exact, _, _ = cav.poisson(f)
    assert np.linalg.norm(psi - exact) <= MIXED_RTOL * n * np.linalg.norm(exact)
