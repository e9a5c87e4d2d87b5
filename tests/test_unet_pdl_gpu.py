"""The network's forward pass with its layers started early (programmatic
dependent launch) and in turn: the same kernels in the same order, so every
output and every activation is equal bit for bit, also when passes of different
inputs follow one another and when new weights are packed in between."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _outputs(pdl, dims):
    import cfdfs
    os.environ["CFD_PDL"] = "1" if pdl else "0"
    try:
        net = cfdfs.UNet(device=0, seed=5)
    finally:
        del os.environ["CFD_PDL"]
    rng = np.random.default_rng(2)
    n = int(np.prod(dims))
    out = []
    for k in range(4):
        x = rng.standard_normal(n).astype(np.float32)
        out.append(np.array(net.forward(x, dims)))
        if k == 1:
            w = net.params()
            net.set_params(w + 0.01 * rng.standard_normal(w.shape).astype(w.dtype))
    net.close()
    return out


@pytest.mark.parametrize("dims", [(5, 5, 5), (17, 9, 33), (25, 25, 161), (65, 65, 65)])
def test_early_start_is_bit_identical(dims):
    for a, b in zip(_outputs(True, dims), _outputs(False, dims)):
        assert np.isfinite(a).all() and np.linalg.norm(b) > 0
        assert np.array_equal(a, b)
