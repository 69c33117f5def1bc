"""The U-Net's weight-gradient sums.

A weight gradient is a sum over all voxels of a crop in FP32, in chains of tensor-core
accumulations whose order is part of the result (the last bits of a gradient decide
BF16 roundings of the next step).  One test holds the chains to those of a recorded
gradient; the other holds every sum to the oracle's exactly, with operands for which
no order and no rounding matters, so that one voxel left out or counted twice shows."""
import os

import numpy as np
import pytest

import unet_oracle as UO
from test_gpu_unet import _data, _net, _rel

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "unet", "wgrad_64.npz")
# The recorded gradient's 33 chains were added by atomics, in any order: 33 additions
# of relative error 2^-24 each, at random sqrt(33) 2^-24 = 3.4e-7; two such orders
# differ by at most twice that.  Chains over other tiles are 5.7e-6 off.
CHAIN_TOL = 7e-7


def test_weight_gradient_chains(cuda_lib):
    """Layer 8 (48 to 16 channels, 512 voxel tiles) at 64^3 against the gradient
    recorded from the kernel that dealt the tiles to 33 chains for each channel group
    and dz plane."""
    import vfs_poisson as V
    net, p = _net(12)
    (f, t, w), (fd, td, wd) = _data((64, 64, 64), seed=2)
    g = np.zeros(net.num_params, np.float32)
    net.gradient(V.UNet.batch(fd, td, wd), g)
    net.close()
    off = sum(27 * a * b + b for a, b in UO.LAYERS[:8])
    want = np.load(GOLDEN)["layer8"]
    assert _rel(g[off:off + want.size].astype(np.float64), want.astype(np.float64)) <= CHAIN_TOL


def _exact_case(dims, seed):
    """Weights of 0 and +-1 (one or two inputs a channel; a channel goes to the coarser
    level or to a skip, not to both), features of 0 and 64 (multiples of 8 and of 1 after
    a pool each), errors of 0 and +-1 and a power of two of loss weights: every
    activation and every gradient has at most 8 significant bits, every sum at most 24."""
    rng = np.random.default_rng(seed)
    coarser = {2: (8, 16), 4: (16, 32)}
    parts = []
    for li, (ci, co) in enumerate(UO.LAYERS):
        w = np.zeros((27, ci, co), np.float32)
        if li == 6:
            src = np.concatenate([rng.permutation(64)[:16], 64 + np.arange(16)])
        elif li == 8:
            src = np.concatenate([rng.permutation(32)[:8], 32 + np.arange(8)])
        else:
            lo, hi = coarser.get(li, (0, 4 if li == 0 else ci))
            src = lo + np.arange(co) % (hi - lo)
        w[rng.integers(0, 27, co), rng.permutation(src), np.arange(co)] = 1.0
        if li % 2:
            w[rng.integers(0, 27, co), rng.permutation(src), np.arange(co)] -= 1.0
        parts += [w.ravel(), np.zeros(co, np.float32)]
    head = np.zeros(17, np.float32)
    head[:16] = rng.choice([-1.0, 1.0], 16)
    p = np.concatenate(parts + [head])
    shape = dims[::-1]
    f = np.where(rng.random((4,) + shape) < 0.5, np.float32(64), np.float32(0))
    out, _ = UO.forward(p, f, bf16=False)
    w = np.zeros(f[0].size, np.float32)
    w[rng.permutation(w.size)[:1 << int(np.log2(w.size))]] = 1.0
    e = rng.choice(np.array([-1, 0, 0, 0, 0, 0, 0, 1], np.float32), shape)
    return p, f, out.detach().numpy() - e, w.reshape(shape)


@pytest.mark.parametrize("dims", [(20, 12, 8), (36, 28, 20), (64, 64, 64), (100, 52, 44)])
def test_gradient_sums_are_exact(cuda_lib, dims):
    import torch
    import vfs_poisson as V
    p, f, t, w = _exact_case(dims, seed=3)
    want_loss, want = UO.loss_and_grad(p, f, t, w, bf16=False)
    net = V.UNet(0)
    net.set_params(p)
    g = np.zeros(net.num_params, np.float32)
    fd, td, wd = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (f, t, w))
    loss = net.gradient(V.UNet.batch(fd, td, wd), g)
    net.close()
    assert loss == want_loss
    off = 0
    for li, (ci, co) in enumerate(UO.LAYERS):
        n = 27 * ci * co
        fed = 4 if li == 0 else ci  # (the oracle's other inputs of layer 0 are zeros, too)
        np.testing.assert_array_equal(g[off:off + n].reshape(27, ci, co)[:, :fed],
                                      want[off:off + n].reshape(27, ci, co)[:, :fed], err_msg=f"layer {li} weights")
        off += n
        np.testing.assert_array_equal(g[off:off + co], want[off:off + co], err_msg=f"layer {li} bias")
        off += co
    np.testing.assert_array_equal(g[off:], want[off:], err_msg="head")
