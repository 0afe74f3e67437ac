"""GPU test of the FP64 up-leg at the sizes where its blocks change (csrc/kernels.cu,
kProlong64: 4, 8 or 16 fine rows a block), with odd and even node counts, partial last
blocks, rows of an odd length (chunks that span two rows) and voids.

One preconditioner application against the CPU oracle, <= 1e-11 relative as for every
FP64 operator.  Results below 2^-1018 take another way of applying the weights: there
every value is a whole number of 2^-1074, and each of its at most n_coarse + 200 terms
rounds once.
"""
import numpy as np
import pytest

import oracle
from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu


# (z, y, x) elements: 4, 4, 8, 8, 16 and 16 rows
@pytest.mark.parametrize("shape", [(5, 3, 1), (36, 13, 22), (151, 11, 6), (153, 15, 9), (303, 16, 5), (310, 30, 4)])
def test_preconditioner(shape):
    rng = np.random.default_rng(shape[0])
    vox = (rng.random(shape) < 0.85).astype(np.uint8)
    vox[:, 0] = 1
    ids = domains.node_numbering(vox)
    fixed = np.sort(ids[:, 0][ids[:, 0] >= 0])  # a whole side: a well-conditioned coarsest system
    ke = domains.hex8_stiffness()
    levels = 2 if min(shape) < 3 else 3
    o = oracle.Oracle(vox, ke, fixed, levels)
    A = api.assembleSystemMatrix(vox, ke, fixed, levels)
    M = api.MultigridPreconditioner(A)
    r = rng.standard_normal(A.rows())
    z, want = M.solve(r), o.precond(r)
    assert np.linalg.norm(z - want) <= 1e-11 * np.linalg.norm(want)
    tiny = M.solve(np.ldexp(r, -1030))
    bound = (A.coarse_free_dofs + 200) * 2.0 ** -44 * max(1.0, np.abs(want).max())
    assert np.abs(np.ldexp(tiny, 1030) - z).max() <= bound
    free = np.setdiff1d(np.arange(A.rows()), np.repeat(3 * fixed, 3) + np.tile(np.arange(3), fixed.size))
    for bad in (np.nan, np.inf):
        rb = r.copy()
        rb[free[len(free) // 2]] = bad
        assert not np.isfinite(M.solve(rb)[free[len(free) // 2]])
    A.close()
