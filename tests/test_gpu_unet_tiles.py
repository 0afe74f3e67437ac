"""GPU tests of the U-Net's convolution tiles (csrc/unet.cu) where they can go
wrong: grids smaller than a tile, with remainders on every level (n = 24: 24,
12, 6, 3 voxels an edge; 40: 40, 20, 10, 5) and the first grid with tall tiles on
the finest level.

Against the numpy restatement (tests/unet_ref.py: the same BF16 rounding points,
64-bit sums), tolerance 2e-2 relative L2 per layer as in test_gpu_learned.py:
a BF16 rounding is 2^-9 and each of eight layers adds one.
"""
import numpy as np
import pytest

from tests import unet_ref as U
from vulkanfem_gb300 import learned

pytestmark = pytest.mark.gpu

TOL = 2e-2


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _problem(n):
    rng = np.random.default_rng(n)
    x = np.zeros((n, n, n, 16), np.float32)
    x[..., :9] = rng.standard_normal((n, n, n, 9)) * 0.5
    t = (rng.standard_normal((n, n, n, 3)) * 0.1).astype(np.float32)
    return x, t, (rng.random((n, n, n)) < 0.8).astype(np.float32)


@pytest.mark.parametrize("n", [8, 24, 40])
def test_forward_and_gradients(n):
    U.ROUND = True
    p = U.init_params(n)
    x, t, m = _problem(n)
    net = learned.UNet(n, p)
    y = net.forward(x)
    loss, g = net.train_batch(x[None], t[None], m[None], 0.0, want_grads=True)
    _, g2 = net.train_batch(x[None], t[None], m[None], 0.0, want_grads=True)
    net.close()
    loss_ref, g_ref, y_ref = U.loss_and_grads(p.astype(np.float64), x.astype(np.float64), t.astype(np.float64),
                                              m.astype(np.float64))
    assert _rel(y, y_ref[..., :3]) < TOL
    assert loss == pytest.approx(loss_ref, rel=TOL)
    for l, ((w0, w1), (b0, b1)) in enumerate(U.param_layout()[0]):
        assert _rel(g[w0:w1], g_ref[w0:w1]) < TOL, ("weights", l)
        assert _rel(g[b0:b1], g_ref[b0:b1]) < TOL, ("bias", l)
    assert np.array_equal(g, g2)


def test_weights_follow_set_params_and_training():
    """The BF16 working weights are those of the last set_params or Adam step."""
    n = 16
    x, t, m = _problem(n)
    net = learned.UNet(n, U.init_params(1))
    a = net.forward(x)
    net.train_batch(x[None], t[None], m[None], 1e-2)
    b = net.forward(x)
    trained = net.get_params()
    net.set_params(U.init_params(1))
    assert np.array_equal(net.forward(x), a) and not np.array_equal(a, b)
    net.set_params(trained)
    assert np.array_equal(net.forward(x), b)
    net.close()
