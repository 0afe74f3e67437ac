"""GPU test of x.(Kx) in the FP32 product: how many plain FP32 additions a sum goes through.

A vector that is not 0 in one node column only, so that one thread sums it: a term
of about 1 at the lowest node, then 45 layers whose single products are just
below half an ulp of 1 and would each be lost if added one at a time.  The grid
(47 node layers, 304 tiles) is marched in one part, the longest march there is.

Tolerance: a thread adds its nodes' sums of three products plainly, 47 layers and 3
operations within a node: 50 roundings of 2^-24 of the sum (all terms are positive).
The reference is the FP64 sum of the same FP32 values x and y = Kx.
"""
import numpy as np
import pytest

from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu


def test_long_march_keeps_small_terms():
    shape = nz, ny, nx = 46, 265, 247
    ke = domains.hex8_stiffness()
    ids = np.arange((nz + 1) * (ny + 1) * (nx + 1)).reshape(nz + 1, ny + 1, nx + 1)
    A = api.assembleSystemMatrix(np.ones(shape, np.uint8), ke, np.sort(ids[:, :, 0].reshape(-1)), 5)
    # per component: a node's own entry, its coupling to the next node of the column
    corners = range(8)
    own = [sum(ke[3 * a + c, 3 * a + c] for a in corners) for c in range(3)]
    up = [sum(ke[3 * a + c, 3 * (a + 4) + c] for a in range(4)) for c in range(3)]
    x = np.zeros((nz + 1, ny + 1, nx + 1, 3), np.float32)
    j, i = 100, 70
    x[0, j, i, 0] = np.sqrt(1.05 / sum(ke[3 * a, 3 * a] for a in range(4)))
    for c in range(3):
        x[2:, j, i, c] = np.sqrt(0.95 * 2.0 ** -24 / (own[c] - 2 * up[c])) * (-1.0) ** np.arange(2, nz + 1)
    y, dot = A.dot_mixed(x.reshape(-1).astype(np.float64))
    terms = x.reshape(-1).astype(np.float64) * y
    small = terms.reshape(x.shape)[3:-1, j, i]
    assert (small > 0.9 * 2.0 ** -24).all() and (small < 2.0 ** -24).all()
    assert abs(dot - terms.sum()) <= 50 * 2.0 ** -24 * np.abs(terms).sum()
    A.close()
