"""GPU tests of the FP64 product for element matrices whose rows, components or
corners differ in scale or do not couple, where one fixed-point grid for all 24
values would lose the small ones.

Entry by entry against extended-precision numpy.  Tolerances, from the operations:

* no Walsh pattern: 2^-47 of sum |Ke_rc| |E u_c| over a row and the up to 8
  elements of a node: 24 multiply-adds, two factors and 8 additions of 2^-53
  each are 2^-47.9; the integer form stays within 2^-48 and its node sum;
* the cube's pattern (any constants), which is multiplied in the Walsh basis: the
  same 2^-47 (about 14 roundings) of what reaches an output component c, the sum
  over components c' of (sum of |Khat| over the (c, c') entries) (sum of |E u_c'|).
"""
import numpy as np
import pytest

from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu

LD = np.longdouble
H = np.array([[(-1) ** bin(m & a).count("1") for a in range(8)] for m in range(8)], float)


def _reorder(ke):
    dof = [3 * p + c for p in domains.KE0_NODE_PERM for c in range(3)]
    return ke[np.ix_(dof, dof)]


def _scaled(ke, s):
    d = np.tile(s, 8)
    return ke * d[:, None] * d[None, :]


def _brick(hx, hy, hz, nu=0.3):
    """The stiffness of a brick-shaped voxel (2 x 2 x 2 Gauss points)."""
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 0.5 / (1 + nu)
    D = np.diag([2 * mu] * 3 + [mu] * 3)
    D[:3, :3] += lam
    ke = np.zeros((24, 24))
    g = 0.5 + np.array([-1, 1]) / np.sqrt(12.0)
    for z in g:
        for y in g:
            for x in g:
                B = np.zeros((6, 24))
                for a in range(8):
                    dx, dy, dz = a & 1, a >> 1 & 1, a >> 2
                    fx, fy, fz = (x if dx else 1 - x), (y if dy else 1 - y), (z if dz else 1 - z)
                    nx, ny, nz = (2 * dx - 1) * fy * fz / hx, (2 * dy - 1) * fx * fz / hy, (2 * dz - 1) * fx * fy / hz
                    B[:, 3 * a:3 * a + 3] = [[nx, 0, 0], [0, ny, 0], [0, 0, nz], [ny, nx, 0], [0, nz, ny], [nz, 0, nx]]
                ke += B.T @ D @ B * (hx * hy * hz / 8)
    return (ke + ke.T) / 2


def _laplace():
    """Three uncoupled scalar Laplacians."""
    k = np.zeros((8, 8))
    for a in range(8):
        for b in range(8):
            n = [(a >> i ^ b >> i) & 1 for i in range(3)]
            k[a, b] = sum((-1 if n[i] else 1) * np.prod([(1 / 6 if n[j] else 1 / 3) for j in range(3) if j != i])
                          for i in range(3))
    return np.kron(k, np.eye(3))


MATRICES = {
    "component_1e-3": lambda: _scaled(domains.hex8_stiffness(), [1, 1, 1e-3]),
    "component_1e-3_reordered": lambda: _reorder(_scaled(domains.hex8_stiffness(), [1, 1, 1e-3])),
    "component_1e-6_reordered": lambda: _reorder(_scaled(domains.hex8_stiffness(), [1, 1e-6, 1])),
    "brick": lambda: _brick(1.0, 1.5, 20.0),
    "nu_quarter_reordered": lambda: _reorder(domains.hex8_stiffness(1.0, 0.25)),  # a third of the entries is 0
    "laplace": _laplace,
    "lumped": lambda: np.diag(10.0 ** np.random.default_rng(1).uniform(-3, 3, 24)),
    "coupled_reordered": lambda: _reorder(domains.hex8_stiffness()),  # the integer form's own
}
VECTORS = {
    "random": lambda r, n: r.standard_normal((n, 3)),
    "x_only": lambda r, n: r.standard_normal((n, 3)) * [1, 0, 0],
    "z_only": lambda r, n: r.standard_normal((n, 3)) * [0, 0, 1],
    "y_large": lambda r, n: r.standard_normal((n, 3)) * [1, 1e9, 1],
    "spikes": lambda r, n: np.where(r.random((n, 3)) < 0.01, 1e10, 1.0) * r.standard_normal((n, 3)),
}


def _structured(ke):
    """Khat where it has the cube's pattern (each entry's two axis-reflection signs agree), else None."""
    k = np.zeros((24, 24))
    for c in range(3):
        for d in range(3):
            k[c::3, d::3] = H @ ke[c::3, d::3] @ H / 64
    k[np.abs(k) <= 1e-13 * np.abs(k).max()] = 0.0
    for i, j in zip(*np.nonzero(k)):
        (m, c), (n, d) = divmod(i, 3), divmod(j, 3)
        if m == 0 or (m ^ (1 << c)) != (n ^ (1 << d)):
            return None
    return k


@pytest.mark.parametrize("name", MATRICES)
def test_small_rows_and_values_keep_their_digits(name):
    shape = (5, 8, 32)  # [z, y, x]
    rng = np.random.default_rng(5)
    vox = (rng.random(shape) < 0.8).astype(np.uint8)
    vox[0] = 1
    vox = domains.keep_grounded(vox)
    ids = domains.node_numbering(vox)
    fixed = np.sort(ids[0][ids[0] >= 0])
    mask = domains.used_nodes_mask(vox)
    E = rng.lognormal(0, 0.5, shape).astype(np.float32)
    ke = MATRICES[name]()
    ke = np.triu(ke) + np.triu(ke, 1).T
    khat = _structured(ke)
    assert (khat is None) == (name not in ("component_1e-3", "brick", "laplace"))
    if khat is None:
        reach = np.abs(ke)
    else:
        S = np.array([[np.abs(khat[c::3, d::3]).sum() for d in range(3)] for c in range(3)])
        reach = np.tile(S, (8, 8))
    A = api.assembleSystemMatrix(vox, ke, fixed, 2, E=E)
    nz, ny, nx = shape
    at = [np.s_[a >> 2:(a >> 2) + nz, (a >> 1 & 1):(a >> 1 & 1) + ny, (a & 1):(a & 1) + nx] for a in range(8)]
    e = (vox * E).astype(LD)[..., None]
    for vec, make in VECTORS.items():
        x = make(rng, A.rows() // 3)
        g = np.zeros(mask.shape + (3,), LD)
        g[mask] = x
        u = np.concatenate([g[s] for s in at], axis=-1) * e
        w, t = np.zeros_like(u), np.zeros_like(u)
        for r in range(24):
            for c in range(24):
                w[..., r] += LD(ke[r, c]) * u[..., c]
                t[..., r] += LD(reach[r, c]) * np.abs(u[..., c])
        y, tol = np.zeros_like(g), np.zeros_like(g)
        for a, s in enumerate(at):
            y[s] += w[..., 3 * a:3 * a + 3]
            tol[s] += t[..., 3 * a:3 * a + 3]
        y, tol = y[mask], tol[mask] * LD(2.0) ** -47
        y[fixed] = 0
        off = np.abs((A @ x.reshape(-1)).reshape(-1, 3).astype(LD) - y)
        assert (off <= tol).all(), (vec, float((off / np.where(tol > 0, tol, LD(1e-300))).max()))
    A.close()
