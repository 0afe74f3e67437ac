"""GPU test of the fixed-point FP64 product (csrc/matvec_fx.cu) at the largest sums its
grid allows: every node at the top of a binade with alternating signs, so that the
three normal strains of an element add up to 3/4 of 2^63, and the magnitude doubling
once along z, so that the grid chosen below it is kept with no bit to spare.

Tolerance as in the entrywise test of the same product: 2^-49 C E sum|x| over the up
to 8 elements of a node, C the largest sum of |Khat| over one component's rows.
"""
import numpy as np
import pytest

from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu

LD = np.longdouble
H = np.array([[(-1) ** bin(m & a).count("1") for a in range(8)] for m in range(8)], float)


@pytest.mark.parametrize("nu", [0.0, 0.3, 0.49])
@pytest.mark.parametrize("at", [1, 4, 7])  # node layer from which on the magnitude is twice as large
def test_largest_sums(nu, at):
    nz, ny, nx = shape = (9, 8, 33)
    ke = domains.hex8_stiffness(1.0, nu)
    mod = np.float32(2.0) - np.float32(2.0) ** -23
    A = api.assembleSystemMatrix(np.ones(shape, np.uint8), ke, np.arange((nx + 1) * (ny + 1)), 2,
                                 E=np.full(shape, mod, np.float32))
    z, y, x = np.meshgrid(*(np.arange(s + 1) for s in shape), indexing="ij")
    top = 2.0 - 2.0 ** -52
    g = np.stack([(-1.0) ** x, (-1.0) ** y, (-1.0) ** z], axis=-1) * top * np.where(z >= at, 2.0, 1.0)[..., None]
    cut = [np.s_[a >> 2:(a >> 2) + nz, (a >> 1 & 1):(a >> 1 & 1) + ny, (a & 1):(a & 1) + nx] for a in range(8)]
    u = np.concatenate([g[s] for s in cut], axis=-1).astype(LD) * LD(mod)
    khat = np.zeros((24, 24))
    for c in range(3):
        for d in range(3):
            khat[c::3, d::3] = H @ ke[c::3, d::3] @ H / 64
    C = max(np.abs(khat)[c::3].sum() for c in range(3))
    want, tol = np.zeros(g.shape, LD), np.zeros(g.shape, LD)
    for a, s in enumerate(cut):
        for c in range(3):
            want[s + (c,)] += sum(LD(ke[3 * a + c, j]) * u[..., j] for j in range(24))
        tol[s] += (LD(2.0) ** -49 * LD(C) * np.abs(u).sum(axis=-1))[..., None]
    want[0] = 0
    assert (np.abs((A @ g.reshape(-1)).astype(LD).reshape(g.shape) - want) <= tol).all()
    A.close()
