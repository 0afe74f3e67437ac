"""GPU test: a solve whose options are refused puts nothing on the GPU.  Its copy of the
warm start would otherwise still read the caller's array after the call has returned."""
import numpy as np
import pytest

from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [{"rtol": -1.0}, {"check_every": -3}, {"mg_mode": "vcycle", "omega": float("nan")}])
def test_refused_options_with_a_warm_start(bad):
    d = domains.cantilever(32, 16, 16, 3)
    A = api.assembleSystemMatrix(d.voxels, domains.hex8_stiffness(), d.fixed, d.num_levels)
    u, _ = A.solve(d.load_vector())
    u0 = 0.9 * u
    before = api.kernel_launch_count()
    with pytest.raises(api.VfemError):
        A.solve(u0=u0, **bad)
    assert api.kernel_launch_count() == before
    v, st = A.solve(u0=u0)  # and the problem stays usable
    assert np.linalg.norm(v - u) <= 1e-5 * np.linalg.norm(u)
    A.close()
