"""GPU tests of the copies between the caller's arrays and the device
(csrc/host_copy.h): directly below 192 MB, through the pinned ring above; fresh
and unaligned result arrays; the bytes around a result stay as they were.  The
values are compared exactly with the same product on device arrays.
"""
import ctypes

import numpy as np
import pytest

from vulkanfem_gb300 import api, domains

pytestmark = pytest.mark.gpu


def _device_product(A, mask, x):
    torch = pytest.importorskip("torch")
    g = np.zeros(mask.shape + (3,))
    g[mask] = x.reshape(-1, 3)
    tx = torch.from_numpy(g).cuda()
    ty, td = torch.empty_like(tx), torch.empty(1, dtype=torch.float64, device="cuda")
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (tx, ty, td)]
    s = api.load_library().vfem_apply_operator_device_noalloc(
        A._h, *ptr, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert s == 0
    torch.cuda.synchronize()
    return ty.cpu().numpy()[mask].reshape(-1)


# the second shape has 8.6 M nodes: 207 MB, 24 full chunks of the ring and a part
@pytest.mark.parametrize("shape,levels", [((9, 7, 5), 2), ((211, 203, 199), 6)])
def test_host_product_equals_device_product(shape, levels):
    d = domains.cantilever(*shape, levels)
    A = api.assembleSystemMatrix(d.voxels, domains.hex8_stiffness(), d.fixed, levels)
    mask = domains.used_nodes_mask(d.voxels)
    n = A.rows()
    buf = np.random.default_rng(0).standard_normal(n + 2)
    x = buf[1:-1]                                    # not page-aligned
    ref = _device_product(A, mask, x)
    y = np.full(n + 2, 7.0)
    lib = api.load_library()
    for _ in range(2):
        y[1:-1] = 0.0
        assert lib.vfem_apply_operator(A._h, x, y[1:-1]) == 0
        assert np.array_equal(y[1:-1], ref) and y[0] == 7.0 and y[-1] == 7.0
    assert np.array_equal(A @ x, ref)                # a fresh result array
    A.close()
