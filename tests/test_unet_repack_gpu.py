"""Forward passes that pack new weights themselves (after set_params and after a
training step): with the layers started early and in turn every output is equal bit
for bit, and equal to a fresh network's with the same weights."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _net(pdl):
    import cfdfs
    os.environ["CFD_PDL"] = "1" if pdl else "0"
    try:
        return cfdfs.UNet(device=0, seed=5)
    finally:
        del os.environ["CFD_PDL"]


@pytest.mark.parametrize("dims", [(5, 5, 5), (33, 17, 9), (65, 65, 65)])
def test_repacked_weights_are_the_ones_used(dims):
    rng = np.random.default_rng(3)
    n = int(np.prod(dims))
    x, t = rng.standard_normal(n).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    early, turn = _net(True), _net(False)
    w = early.params()
    for k in range(12):
        w = (w * np.float32(1.0 + 0.3 * (-1) ** k)).astype(np.float32)
        early.set_params(w)
        turn.set_params(w)
        a, b = early.forward(x, dims), turn.forward(x, dims)
        assert np.isfinite(a).all() and np.array_equal(a, b), k
        if k % 4 == 3:
            for net in (early, turn):
                net.train_batch(x.reshape(1, *dims[::-1]), t.reshape(1, *dims[::-1]), dims, 1e-3)
            assert np.array_equal(early.forward(x, dims), turn.forward(x, dims)), k
            assert np.array_equal(early.params(), turn.params())
            w = early.params()
    fresh = _net(True)
    fresh.set_params(early.params())
    assert np.array_equal(fresh.forward(x, dims), early.forward(x, dims))
    for net in (early, turn, fresh):
        net.close()
