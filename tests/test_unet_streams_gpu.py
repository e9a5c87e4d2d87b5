"""The backward pass with its weight gradients on a second stream.  Every sum has a
fixed order, so a pass that read or overwrote something too early would show as
other bits: gradients of alternating inputs are equal to those of the first time,
and a step on a batch equals a step on the same batch by another network."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(5, 5, 5), (33, 17, 9), (25, 25, 161), (65, 65, 65)])
def test_gradients_repeat_bit_for_bit(dims):
    import cfdfs
    rng = np.random.default_rng(4)
    n = int(np.prod(dims))
    x = rng.standard_normal((3, n)).astype(np.float32)
    t = rng.standard_normal((3, n)).astype(np.float32)
    net = cfdfs.UNet(device=0, seed=6)
    first = [np.array(net.gradient(x[k], t[k], dims)[1]) for k in range(3)]
    for _ in range(4):
        for k in (2, 0, 1):
            assert np.array_equal(np.array(net.gradient(x[k], t[k], dims)[1]), first[k])
    other = cfdfs.UNet(device=0, seed=6)
    for _ in range(3):
        for m in (net, other):
            m.train_batch(x, t, dims, lr=1e-3)
    assert np.array_equal(net.params(), other.params())
    net.close()
    other.close()
