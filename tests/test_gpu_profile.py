"""GPU test: vfem_profile_kernels times the fixed-point products (the FP64 product and the
true residual) on operands with work in them, whatever ran before on the problem.
The product on zeros, where every element is skipped, takes half the time; clocks and
runs differ by a few percent (bound: 20%)."""
import pytest

from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu


def test_times_do_not_depend_on_what_ran_before():
    d = domains.cantilever(160, 128, 128, 4)
    A = api.assembleSystemMatrix(d.voxels, domains.hex8_stiffness(), d.fixed, d.num_levels)
    api.profile_kernels(A, 20)  # clocks up
    B = api.assembleSystemMatrix(d.voxels, domains.hex8_stiffness(), d.fixed, d.num_levels)
    fresh = api.profile_kernels(B, 20)
    B.solve(d.load_vector(), precision="fp64", rtol=1e-3)  # dense vectors in their place
    after = api.profile_kernels(B, 20)
    for name in ("matvec_fp64", "true_residual_df"):
        assert abs(fresh[name] - after[name]) <= 0.2 * after[name], name
    A.close()
    B.close()
