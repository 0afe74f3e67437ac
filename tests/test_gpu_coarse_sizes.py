"""GPU test of the coarsest solve around the sizes at which its kernel changes
(csrc/kernels.h, kSmallCoarse: 3000 free DOFs in FP64, 4096 in mixed precision),
with counts that are and are not a multiple of the 8 values a lane loads or of the 8 rows of a block.

A two-level V-cycle against its numpy restatement.  The two inverses are computed
independently, so their products may differ by a few cond(K) roundings: 2^-53 in
FP64; in mixed precision 2^-24, plus 2^-11 for the FP16 inverse and smoother.
"""
import numpy as np
import pytest

from tests import structured_ref as sr
from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,n", [((2, 2, 2), 12), ((3, 5, 8), 120), ((14, 4, 8), 315), ((25, 12, 12), 1911),
                                     ((24, 14, 12), 2016), ((20, 18, 18), 3000), ((22, 24, 12), 3003),
                                     ((34, 18, 14), 4080), ((38, 16, 14), 4104)])
def test_two_level_cycle(shape, n):
    Ke = domains.hex8_stiffness()
    d = domains.cantilever(*shape, 2)
    ref = sr.MultiplicativeMG(d.voxels, Ke, d.fixed, 2)
    A = api.assembleSystemMatrix(d.voxels, Ke, d.fixed, 2)
    assert A.coarse_free_dofs == n == ref.Kinv.shape[0]
    ev = np.linalg.eigvalsh((ref.Kinv + ref.Kinv.T) / 2)
    cond = ev[-1] / ev[0]
    r = np.random.default_rng(n).random(A.rows())
    want = ref.apply(r)
    scale = np.linalg.norm(want)
    for precision, eps in (("fp64", 2.0 ** -53), ("mixed", 2.0 ** -24)):
        z = api.MultigridPreconditioner(A, mode="vcycle", precision=precision).solve(r)
        tol = 8 * cond * eps + (4 * 2.0 ** -11 if precision == "mixed" else 0.0)
        assert np.linalg.norm(z - want) <= tol * scale
    A.close()


def test_even_split_of_the_tiles():
    """6,552 coarse free DOFs: 5,356 tiles of the packed FP16 inverse over 1,824 warps, ranges
    that end within and across row blocks.  Mixed against FP64: 2^-11 of the FP16 inverse and
    smoother and the FP32 inversion, whose condition number here is about 1e4."""
    d = domains.cantilever(28, 24, 22, 2)
    A = api.assembleSystemMatrix(d.voxels, domains.hex8_stiffness(), d.fixed, 2)
    assert A.coarse_free_dofs == 6552
    r = np.random.default_rng(0).random(A.rows())
    z = api.MultigridPreconditioner(A).solve(r)
    zm = api.MultigridPreconditioner(A, precision="mixed").solve(r)
    assert np.linalg.norm(zm - z) <= 8 * 2.0 ** -11 * np.linalg.norm(z)
    A.close()
