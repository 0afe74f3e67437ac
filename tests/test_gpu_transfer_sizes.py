"""GPU tests of the 2x transfers on both sides of the sizes at which the kernels
change (csrc/kernels.cu, kSmallRestrict and kSmallProlong): one thread per value,
the flat up-leg and the marching restriction, with odd and even element counts.

FP64 against numpy on a solid box (every node used): full weighting sums 27
values with weights adding to 8, interpolation averages at most 8 values; a few
roundings of 2^-53 each, so 1e-14 of the largest value.
"""
import numpy as np
import pytest

from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu


def _axis(n, m):
    """Trilinear weights of m coarse nodes at n fine nodes along one axis."""
    P = np.zeros((n, m))
    for f in range(n):
        P[f, f // 2] += 1.0 if f % 2 == 0 else 0.5
        if f % 2:
            P[f, f // 2 + 1] += 0.5
    return P


# nodes: 4 k and 61 k (both small), 188 k (flat up-leg), 1.09 M and 1.06 M (marching restriction)
@pytest.mark.parametrize("shape", [(17, 16, 13), (40, 38, 37), (60, 61, 49), (104, 102, 100), (101, 103, 99)])
def test_transfers(shape):
    levels = 3 if max(shape) < 64 else 5
    d = domains.cantilever(*shape, levels)
    A = api.assembleSystemMatrix(d.voxels, domains.hex8_stiffness(), d.fixed, levels)
    fine = tuple(s + 1 for s in reversed(shape))
    coarse = tuple((s + 1) // 2 + 1 for s in reversed(shape))
    P = [_axis(n, m) for n, m in zip(fine, coarse)]
    rng = np.random.default_rng(1)
    v, w = rng.standard_normal(fine + (3,)), rng.standard_normal(coarse + (3,))
    up = np.einsum("ai,bj,ck,ijkl->abcl", *P, w, optimize=True)
    down = np.einsum("ai,bj,ck,abcl->ijkl", *P, v, optimize=True)
    assert np.abs(A.interpolate(0, w.reshape(-1)) - up.reshape(-1)).max() <= 1e-14 * np.abs(w).max()
    assert np.abs(A.restrict(0, v.reshape(-1)) - down.reshape(-1)).max() <= 1e-14 * 8 * np.abs(v).max()
    # the whole cycle, mixed against FP64 (FP16 smoothing diagonal and coarsest inverse: 2^-11 each)
    r = v.reshape(-1)
    z = api.MultigridPreconditioner(A).solve(r)
    zm = api.MultigridPreconditioner(A, precision="mixed").solve(r)
    assert np.linalg.norm(zm - z) <= 2e-3 * np.linalg.norm(z)
    A.close()


@pytest.mark.parametrize("n", [24, 60])
def test_fp64_and_mixed_solves_agree(n):
    """Both solvers' iterations on the small-grid kernels (fused residual update, r.z dots)."""
    d = domains.spheres(n, 12, 2.0, 5.0, seed=2, levels=3)
    A = api.assembleSystemMatrix(d.voxels, domains.hex8_stiffness(), d.fixed, 3, E=d.E)
    f = d.load_vector()
    u, st = A.solve(f, precision="fp64", rtol=1e-9)
    um, sm = A.solve(f, precision="mixed", rtol=1e-8)
    assert st["rel_residual"] < 1e-8 and sm["rel_residual"] < 1e-8 and not sm["fallback"]
    assert np.linalg.norm(um - u) <= 1e-6 * np.linalg.norm(u)
    A.close()
