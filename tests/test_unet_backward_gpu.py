"""Tensor-core backward pass of the U-Net (unet_bwd.cu) at the sizes where its
bricks and row tiles have remainders: the smallest grid, x-rows split into
several bricks, odd extents, and one sample's gradient reproduced bit for bit.

Tolerance: both sides start from the device's stored forward tensors.  The
device's data gradient goes through at most 10 layers and its weight gradient
through one more sum, each FP32 sum within 2 units in the last place of its
norm (2 x 2^-23), so 11 x 2^-22 = 2.6e-6 per layer's gradient; 3e-6 is asserted.
"""
import os
import sys

import numpy as np
import pytest

from conftest import rel_l2

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import unet_oracle as U  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(5, 5, 5), (9, 5, 17), (33, 13, 9), (69, 9, 5), (5, 37, 21), (133, 5, 9)])
def test_gradient_per_layer(dims):
    import cfdfs
    net = cfdfs.UNet(device=0, seed=0)
    theta = U.init_params(11)
    net.set_params(theta)
    rng = np.random.default_rng(12)
    x = rng.standard_normal(dims[::-1]).astype(np.float32)
    t = rng.standard_normal(dims[::-1]).astype(np.float32)
    _, g = net.gradient(x, t, dims)
    T = [net.tensor(k, dims).astype(np.float64) for k in range(len(U.TENSORS))]
    _, ref = U.backward(theta, T, t.astype(np.float64))
    offs = np.cumsum([0] + [a + b for (a, b, _, _) in U.layer_shapes()])
    for layer in range(len(U.CONVS)):
        sl = slice(offs[layer], offs[layer + 1])
        assert rel_l2(g[sl], ref[sl]) < 3e-6, layer
    _, again = net.gradient(x, t, dims)
    assert np.array_equal(g, again)
    net.close()
