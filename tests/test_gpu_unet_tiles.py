"""The U-Net's tile variants against the CPU oracle: crops whose convolutions
fill the chip with 16x8x4 tiles (at full resolution, and down to half of it),
crops that run 16x4x2 tiles throughout, and remainders of both in every
direction.  The tolerances are those of the gradient against the same oracle
elsewhere (BF16 rounding of the gradients before each ReLU).  Two gradients of
the same inputs are the same bits."""
import numpy as np
import pytest

import unet_oracle as UO
from test_gpu_unet import GRAD_TOL, _data, _net, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(4, 4, 4), (36, 28, 20), (68, 60, 64), (52, 100, 44)])
def test_gradient_tiles(cuda_lib, dims):
    import vfs_poisson as V
    net, p = _net()
    (f, t, w), (fd, td, wd) = _data(dims, seed=2)
    g = [np.zeros(net.num_params, np.float32) for _ in range(2)]
    losses = [net.gradient(V.UNet.batch(fd, td, wd), a) for a in g]
    assert losses[0] == losses[1]
    np.testing.assert_array_equal(g[0], g[1])
    lref, gref = UO.loss_and_grad(p, f, t, w)
    assert abs(losses[0] - lref) <= 1e-2 * abs(lref)
    off = 0
    for li, (ci, co) in enumerate(UO.LAYERS):
        nw = 27 * ci * co
        gw, rw = g[0][off:off + nw].reshape(27, ci, co), gref[off:off + nw].reshape(27, ci, co)
        fed = 4 if li == 0 else ci
        assert _rel(gw[:, :fed].ravel(), rw[:, :fed].ravel()) < GRAD_TOL, f"layer {li} weights"
        off += nw
        assert _rel(g[0][off:off + co], gref[off:off + co]) < GRAD_TOL, f"layer {li} bias"
        off += co
    assert _rel(g[0][off:], gref[off:]) < GRAD_TOL, "head"
    net.close()
