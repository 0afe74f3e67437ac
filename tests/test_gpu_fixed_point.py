"""GPU tests of the FP64 product in block fixed point (csrc/matvec_fx.cu).

The product is compared entry by entry with extended-precision numpy (long
double: 64 or 113 bits).  Tolerance, from the number format: an element's output
is off by at most 2^-50 of C E sum|x| (its 24 values; C = the largest sum of
|Khat| over one component's rows): 2^-51 from the inputs (each within 2^-54 of
the largest, doubled three times by the transform), 14 roundings of 2^-56 each;
aligning outputs and the final rounding to FP64 at most double that: 2^-49.
Any other Ke is multiplied as it is; C is then its largest row sum of |Ke| and
the same 2^-49 holds (no transform, one rounding per row and two of its modulus).
"""
import numpy as np
import pytest

from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu

LD = np.longdouble
H = np.array([[(-1) ** bin(m & a).count("1") for a in range(8)] for m in range(8)], float)


def _khat(ke):
    k = np.zeros((24, 24))
    for c in range(3):
        for d in range(3):
            k[c::3, d::3] = H @ ke[c::3, d::3] @ H / 64
    return np.where(np.abs(k) < 1e-13 * np.abs(k).max(), 0.0, k)


def _corners(g, shape):
    nz, ny, nx = shape
    return [g[a >> 2:(a >> 2) + nz, (a >> 1 & 1):(a >> 1 & 1) + ny, (a & 1):(a & 1) + nx] for a in range(8)]


def _reference(vox, E, ke, x, fixed, C=None):
    """K x and the entrywise tolerance."""
    mask = domains.used_nodes_mask(vox)
    g = np.zeros(mask.shape + (3,), LD)
    g[mask] = x.reshape(-1, 3)
    e = vox.astype(LD) * (LD(1) if E is None else E.astype(LD))
    u = np.concatenate(_corners(g, vox.shape), axis=-1)
    w = np.zeros_like(u)
    for i in range(24):
        for j in range(24):
            w[..., i] += LD(ke[i, j]) * u[..., j]
    if C is None:
        C = max(np.abs(_khat(ke))[c::3].sum() for c in range(3))
    t = LD(2.0) ** -49 * LD(C) * (np.abs(u).sum(axis=-1) * e)
    y, tol = np.zeros_like(g), np.zeros(g.shape, LD)
    for a, (v, b) in enumerate(zip(_corners(y, vox.shape), _corners(tol, vox.shape))):
        v += w[..., 3 * a:3 * a + 3] * e[..., None]
        b += t[..., None]
    y, tol = y[mask], tol[mask]
    y[fixed] = 0
    return y.reshape(-1), tol.reshape(-1)


def _domain(shape, seed):
    rng = np.random.default_rng(seed)
    vox = (rng.random(shape) < 0.8).astype(np.uint8)
    vox[0] = 1
    vox = domains.keep_grounded(vox)
    ids = domains.node_numbering(vox)
    return vox, np.sort(ids[0][ids[0] >= 0]), np.argwhere(domains.used_nodes_mask(vox))[:, ::-1].astype(float)


VECTORS = {
    "random": lambda r, P: r.standard_normal(P.shape),
    "smooth": lambda r, P: np.stack([np.sin(P @ [.1, .02, .05]), np.cos(P @ [.05, .1, .01]), P[:, 2] ** 1.5], 1),
    "graded_x": lambda r, P: r.standard_normal(P.shape) * np.exp(0.7 * P[:, :1]),
    "graded_z": lambda r, P: r.standard_normal(P.shape) * np.exp(-2.0 * P[:, 2:]),
    "wide": lambda r, P: r.standard_normal(P.shape) * np.exp(r.uniform(-40, 40, P.shape)),
    "point": lambda r, P: (np.arange(P.size).reshape(P.shape) == P.size // 2) * 1.0,
    "rigid": lambda r, P: np.ones(P.shape) * [1.0, -2.0, 3.0],
    "tiny": lambda r, P: 1e-180 * r.standard_normal(P.shape),       # outside the grid's exponents: FP64 march
    "huge": lambda r, P: 1e250 * r.standard_normal(P.shape),
}


@pytest.mark.parametrize("shape", [(3, 5, 29), (2, 6, 30), (5, 7, 31), (33, 8, 4)])  # [z, y, x]: tile edges
@pytest.mark.parametrize("modulus", ["one", "lognormal", "wide"])
def test_product_against_extended_precision(shape, modulus):
    vox, fixed, P = _domain(shape, 5)
    rng = np.random.default_rng(11)
    E = {"one": None, "lognormal": rng.lognormal(0, 0.5, shape).astype(np.float32),
         "wide": np.exp(rng.uniform(-20, 5, shape)).astype(np.float32)}[modulus]
    ke = domains.hex8_stiffness(1.0, 0.3) if modulus != "wide" else domains.hex8_stiffness(7e10, 0.41)
    A = api.assembleSystemMatrix(vox, ke, fixed, 2, E=E)
    for name, make in VECTORS.items():
        x = make(rng, P).reshape(-1)
        ref, tol = _reference(vox, E, ke, x, fixed)
        off = np.abs((A @ x).astype(LD) - ref)
        assert (off <= tol).all(), (name, float((off / np.where(tol > 0, tol, 1)).max()))
    A.close()


def test_non_finite_values_stay_local():
    shape = (8, 9, 40)
    vox, fixed, P = _domain(shape, 6)
    ke = domains.hex8_stiffness()
    A = api.assembleSystemMatrix(vox, ke, fixed, 2)
    x = np.random.default_rng(1).standard_normal(P.shape)
    ref, tol = _reference(vox, None, ke, x.reshape(-1), fixed)
    bad = P.shape[0] // 2
    x[bad, 1] = np.nan
    x[bad + 200, 0] = np.inf
    y = (A @ x.reshape(-1)).reshape(-1, 3)
    near = (np.abs(P - P[bad]).max(axis=1) <= 1) | (np.abs(P - P[bad + 200]).max(axis=1) <= 1)
    off = np.abs(y.astype(LD).reshape(-1) - ref) <= tol
    assert off.reshape(-1, 3)[~near].all()
    assert not np.isfinite(y[bad]).all() and not np.isfinite(y[bad + 200]).all()
    A.close()


@pytest.mark.parametrize("kind", ["reference_order", "box", "general"])
def test_other_matrices(kind):
    """Ke in the reference's corner order, a box's (components scaled: the cube's
    zero pattern, not its constants) and a symmetric matrix without structure."""
    shape = (5, 8, 32)
    vox, fixed, P = _domain(shape, 7)
    rng = np.random.default_rng(3)
    E = rng.lognormal(0, 0.5, shape).astype(np.float32)
    ke = domains.hex8_stiffness()
    if kind == "reference_order":
        dof = [3 * p + c for p in domains.KE0_NODE_PERM for c in range(3)]
        ke = ke[np.ix_(dof, dof)]
    elif kind == "box":
        s = np.tile([1.0, 2.0, 0.5], 8)
        ke = ke * s[:, None] * s[None, :]
    else:
        B = rng.standard_normal((24, 24))
        ke = 1e-4 * (B @ B.T)
    A = api.assembleSystemMatrix(vox, ke, fixed, 2, E=E)
    C = np.abs(ke).sum(axis=1).max()
    for name in ("random", "smooth", "graded_z", "wide", "huge"):
        x = VECTORS[name](rng, P).reshape(-1)
        ref, tol = _reference(vox, E, ke, x, fixed, C)
        assert (np.abs((A @ x).astype(LD) - ref) <= tol).all(), name
    A.close()
