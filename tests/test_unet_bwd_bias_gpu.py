"""The backward pass carries no error that adds up in one direction over the layers:
weight gradients of every layer against the oracle's, from the device's own stored
forward tensors, with the trained network and a residual-like field.

Tolerance: a layer d layers from the output gets its gradient through d - 1 data
gradients and the loss's and sums it once; each of these d + 1 results within half a
unit in the last place of its norm (2^-25), as sums of rounded-to-nearest additions
are on grids of this many voxels, gives (d + 1) 2^-25.  Truncated sums lose up to a
whole unit each, always towards zero.
"""
import os
import sys

import numpy as np
import pytest

from conftest import PKG, ROOT, rel_l2

sys.path.insert(0, os.path.join(ROOT, "oracle"))
import unet_oracle as U  # noqa: E402

pytestmark = pytest.mark.gpu


def _field(dims, seed):
    rng = np.random.default_rng(seed)
    z, y, x = np.meshgrid(*[np.linspace(0.0, np.pi, n) for n in dims[::-1]], indexing="ij")
    f = 0.3 * rng.standard_normal(dims[::-1])
    for _ in range(6):
        k = rng.integers(0, 5, size=3)
        f += rng.standard_normal() * np.cos(k[0] * x + 0.3) * np.cos(k[1] * y) * np.cos(k[2] * z)
    return (f / np.sqrt((f ** 2).mean())).astype(np.float32)


@pytest.mark.parametrize("dims", [(33, 33, 33), (37, 21, 61)])
def test_layer_gradients_are_unbiased(dims):
    import cfdfs
    net = cfdfs.UNet(device=0, path=os.path.join(PKG, "weights", "unet_cavity.bin"))
    theta = net.params()
    x, t = _field(dims, 3), 0.3 * _field(dims, 4)
    _, g = net.gradient(x, t, dims)
    T = [net.tensor(k, dims).astype(np.float64) for k in range(len(U.TENSORS))]
    net.close()
    _, ref = U.backward(theta, T, t.astype(np.float64))
    offs = np.cumsum([0] + [a + b for (a, b, _, _) in U.layer_shapes()])
    n = len(U.CONVS)
    for layer in range(n):
        sl = slice(offs[layer], offs[layer + 1])
        assert rel_l2(g[sl], ref[sl]) <= (n - layer + 1) * 2.0 ** -25, layer
