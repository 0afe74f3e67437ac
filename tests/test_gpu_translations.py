"""GPU test of the FP64 product with a large component that FP64 sums exactly (a rigid
translation, or values of few bits) beside small ones: the small components' digits stay.

Entry by entry against extended-precision numpy.  Tolerance for an element: an input is
cut off by less than 2 units of its grid (in its node's and in the element's), a Walsh mode
sums 8, a combination up to three modes: 48 units, but only where the largest
combination has at least 2^43 (smaller ones are multiplied in FP64).  That combination is at
most the sum D of |u - u(corner 0)| over the element's 24 values, so 2^-37 C E D (C the
largest sum of |Khat| over one component's rows), summed over a node's elements; the roundings
of the product itself are 2^-49 of the same and, for the result, 2^-53.
"""
import numpy as np
import pytest

from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu

LD = np.longdouble
H = np.array([[(-1) ** bin(m & a).count("1") for a in range(8)] for m in range(8)], float)

VECTORS = {
    # a component, the same everywhere; the others random
    "x": lambda r, P, s: r.standard_normal(P.shape) * [0, 1, 1] + [s / 3.0, 0, 0],
    "z": lambda r, P, s: r.standard_normal(P.shape) * [1, 1, 0] + [0, 0, -s],
    "two": lambda r, P, s: r.standard_normal(P.shape) * [0, 1, 0] + [s, 0, s / 7.0],
    # few bits: multiples of 1/4 of a size up to 2 s
    "steps": lambda r, P, s: np.stack([np.round(s) + 0.25 * P[:, 0], *r.standard_normal((2, len(P)))], axis=1),
    "smooth": lambda r, P, s: np.stack([np.full(len(P), s), np.sin(0.1 * P[:, 2] + 0.03 * P[:, 0]),
                                        0.02 * P[:, 1] ** 1.5], axis=1),
    "rigid": lambda r, P, s: np.full(P.shape, [s, -s / 3.0, 1e-3]),
}


@pytest.mark.parametrize("size", [1.0, 2.0 ** 9, 1e5, 2.0 ** 19 - 1, 1e6, 1e9, 1e13])
@pytest.mark.parametrize("modulus", [False, True])
def test_small_components_beside_a_translation(size, modulus):
    shape = nz, ny, nx = 9, 8, 33
    rng = np.random.default_rng(3)
    vox = (rng.random(shape) < 0.8).astype(np.uint8)
    vox[0] = 1
    vox = domains.keep_grounded(vox)
    ids = domains.node_numbering(vox)
    fixed = np.sort(ids[0][ids[0] >= 0])
    mask = domains.used_nodes_mask(vox)
    E = rng.lognormal(0, 0.5, shape).astype(np.float32) if modulus else None
    ke = domains.hex8_stiffness()
    A = api.assembleSystemMatrix(vox, ke, fixed, 2, E=E)
    khat = np.zeros((24, 24))
    for c in range(3):
        for d in range(3):
            khat[c::3, d::3] = H @ ke[c::3, d::3] @ H / 64
    C = max(np.abs(khat)[c::3].sum() for c in range(3))
    e = (vox * (1.0 if E is None else E)).astype(LD)[..., None]
    P = np.argwhere(mask)[:, ::-1].astype(float)
    cut = [np.s_[a >> 2:(a >> 2) + nz, (a >> 1 & 1):(a >> 1 & 1) + ny, (a & 1):(a & 1) + nx] for a in range(8)]
    for name, make in VECTORS.items():
        x = np.ascontiguousarray(make(rng, P, size))
        g = np.zeros(mask.shape + (3,), LD)
        g[mask] = x
        # K of a translation is 0: from the (exact) differences to corner 0
        u = np.concatenate([(g[s] - g[cut[0]]) * e for s in cut], axis=-1)
        want, tol = np.zeros_like(g), np.zeros_like(g)
        D = LD(2.0) ** -37 * LD(C) * np.abs(u).sum(axis=-1)
        for a, s in enumerate(cut):
            for c in range(3):
                want[s + (c,)] += sum(LD(ke[3 * a + c, j]) * u[..., j] for j in range(24))
            tol[s] += D[..., None]
        want = want[mask]
        want[fixed] = 0
        off = np.abs((A @ x.reshape(-1)).reshape(-1, 3).astype(LD) - want)
        assert (off <= tol[mask] + LD(2.0) ** -53 * np.abs(want)).all(), name
    A.close()
