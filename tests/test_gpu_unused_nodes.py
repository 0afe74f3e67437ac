"""GPU test: values of x at unused nodes stay out of the device product's y and
x.(Kx) also where the product leaves its fixed-point range (csrc/matvec_fx.cu)
and a block repeats its march in FP64.

x is a plain vector times a power of two, and its product the plain one times that
power; a modulus of 2^-130 (subnormal in FP32) on one voxel beside others of 1 gives
the product of a modulus of 2^-100 there.  Both sides are rounded FP64 results of
the same operator (tolerance 1e-11 relative, the operator's parity bar).
"""
import ctypes

import numpy as np
import pytest

from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu

TOL = 1e-11


def _product(A, mask, x, at_unused):
    torch = pytest.importorskip("torch")
    xd = np.full(mask.shape + (3,), at_unused)
    xd[mask] = x.reshape(-1, 3)
    tx = torch.from_numpy(xd.reshape(-1)).cuda()
    ty = torch.full_like(tx, float("nan"))
    dot = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")
    args = [ctypes.c_void_p(t.data_ptr()) for t in (tx, ty, dot)]
    status = api.load_library().vfem_apply_operator_device_noalloc(
        A._h, *args, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert status == api.OK, api.STATUS_NAMES.get(status, status)
    torch.cuda.synchronize()
    return ty.cpu().numpy().reshape(mask.shape + (3,))[mask].reshape(-1), float(dot.item())


# power of two of x (2^-600 is outside of the integer grid's range), power of two of one voxel's modulus
@pytest.mark.parametrize("xpow,epow", [(0, 0), (-600, 0), (0, -130)])
@pytest.mark.parametrize("order", ["cube", "reordered"])
@pytest.mark.parametrize("at_unused", [float("nan"), float("inf")])
def test_unused_nodes_do_not_reach_the_dot(xpow, epow, order, at_unused):
    rng = np.random.default_rng(21)
    vox = (rng.random((9, 11, 37)) < 0.4).astype(np.uint8)
    vox[0] = 1
    vox = domains.keep_grounded(vox)
    ids = domains.node_numbering(vox)
    fixed = np.sort(ids[0][ids[0] >= 0])
    mask = domains.used_nodes_mask(vox)
    # a voxel whose nodes have other voxels too, with unused nodes around in its own layers
    n = np.zeros(mask.shape, int)
    for a in range(8):
        n[a >> 2:(a >> 2) + 9, (a >> 1 & 1):(a >> 1 & 1) + 11, (a & 1):(a & 1) + 37] += vox
    at = next((z, y, x) for z, y, x in np.argwhere(vox) if z > 2 and y < 6 and x < 30
              and n[z:z + 2, y:y + 2, x:x + 2].min() > 1 and not mask[z, :6, :30].all())
    ke = domains.hex8_stiffness()
    if order == "reordered":
        dof = [3 * p + c for p in domains.KE0_NODE_PERM for c in range(3)]
        ke = ke[np.ix_(dof, dof)]

    def problem(power):
        E = np.ones(vox.shape, np.float32)
        E[at] = 2.0 ** power
        return api.assembleSystemMatrix(vox, ke, fixed, 2, E=E)

    plain, A = problem(max(epow, -100)), problem(epow)
    x = rng.standard_normal(A.rows())
    y0, dot0 = _product(plain, mask, x, 0.0)
    y, dot = _product(A, mask, np.ldexp(x, xpow), at_unused)
    assert np.isfinite(y).all()
    assert np.linalg.norm(np.ldexp(y, -xpow) - y0) <= TOL * np.linalg.norm(y0)
    want = np.ldexp(dot0, 2 * xpow)  # 2^-1200 of a number: 0 in FP64
    assert np.isfinite(dot) and abs(dot - want) <= TOL * abs(want)
    plain.close()
    A.close()
