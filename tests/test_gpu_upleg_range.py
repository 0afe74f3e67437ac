"""GPU test: the FP64 V-cycle of values near the top of the FP64 range.

The cycle is linear and every weight of its transfers a power of two, so that a
right-hand side times 2^k gives the result times 2^k bit for bit, as long as nothing
overflows.  k puts the largest result between 2^1021 and 2^1022: the sum of 8 coarse
corners would overflow there, of 2 it doesn't.
"""
import numpy as np
import pytest

from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,levels", [(16, 2), (64, 4), (128, 5)])  # blocks of 4, 8 and 16 rows on the finest level
def test_scaled_cycle_is_exact(n, levels):
    vox = np.ones((n, n, n), np.uint8)
    ids = domains.node_numbering(vox)
    fixed = np.sort(ids[0].reshape(-1))
    A = api.assembleSystemMatrix(vox, domains.hex8_stiffness(), fixed, levels)
    M = api.MultigridPreconditioner(A)
    r = np.zeros((n + 1, n + 1, n + 1, 3))
    r[1:, :, :, 2] = -1.0  # its own weight: displacements of one sign
    z = M.solve(r.reshape(-1))
    assert np.isfinite(z).all()
    k = 1022 - int(np.frexp(np.abs(z).max())[1])
    assert 2.0 ** 1021 <= np.ldexp(np.abs(z).max(), k) < 2.0 ** 1022
    scaled = M.solve(np.ldexp(r, k).reshape(-1))
    np.testing.assert_array_equal(scaled, np.ldexp(z, k))
    A.close()
