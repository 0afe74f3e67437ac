"""GPU test of the mixed-precision solve with element matrices whose FP64 product is
not in fixed point: its true residual runs in double-float arithmetic (structured and
dense form), in the iteration and, with a warm start, for the first residual.

The reported true residual is compared with f - K u from the FP64 product: double-float
rounds at 2^-44 of the summed magnitudes, here at most 1e4 |f| (tolerance 1e-9, of a
residual of about 1e-7); the displacement with an FP64 solve to 1e-10 (the 1e-5 bar).
"""
import numpy as np
import pytest

from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["scaled", "nu_quarter_reordered"])
@pytest.mark.parametrize("warm", [False, True])
def test_true_residual(kind, warm):
    rng = np.random.default_rng(2)
    shape = (18, 21, 33)
    vox = (rng.random(shape) < 0.85).astype(np.uint8)
    vox[0] = 1
    vox = domains.keep_grounded(vox)
    ids = domains.node_numbering(vox)
    fixed = np.sort(ids[0][ids[0] >= 0])
    top = ids[-1][ids[-1] >= 0]
    if kind == "scaled":
        s = np.tile([1.0, 1.0, 0.5], 8)
        ke = domains.hex8_stiffness() * s[:, None] * s[None, :]
    else:
        dof = [3 * p + c for p in domains.KE0_NODE_PERM for c in range(3)]
        ke = domains.hex8_stiffness(1.0, 0.25)[np.ix_(dof, dof)]
    A = api.assembleSystemMatrix(vox, ke, fixed, 3)
    f = np.zeros(A.rows())
    f.reshape(-1, 3)[top, 2] = -1.0 / top.size
    exact, _ = A.solve(f, precision="fp64", rtol=1e-10)
    u0 = exact * (1 + 0.05 * rng.standard_normal(exact.size)) if warm else None
    u, st = A.solve(f, u0=u0, precision="mixed", rtol=1e-6)
    assert st["residual_replacements"] > 0 and not st["fallback"]
    free = np.ones((f.size // 3, 3))
    free[fixed] = 0
    true = np.linalg.norm((f - A @ u) * free.reshape(-1)) / np.linalg.norm(f)
    assert st["rel_residual"] < 1e-6 and abs(st["rel_residual"] - true) <= 1e-9
    assert np.linalg.norm(u - exact) <= 1e-5 * np.linalg.norm(exact)
    A.close()
