"""One context that loads a small, a larger and a small deck again gives each time the
numbers of a fresh context, to the last bit (deterministic mode), and holds the device
memory of the deck it has.

Memory: what a context keeps from the driver is within a block of its pool (16 MiB at
these sizes, more where a larger block is only partly used) and the driver's own
granularity of the fresh context's: 64 MiB.
"""
import os

import numpy as np
import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

OPTIONS = {
    "fp64_jacobi": dict(precond=0),
    "fp64_twolevel": dict(precond=2),
    "mixed_jacobi": dict(precision=1, precond=0),
    "mixed_twolevel": dict(precision=1, precond=2, cg_warm=1, inner_rtol=1e-5),
    "mixed_learned": dict(precision=1, precond=1, cg_warm=1, inner_rtol=1e-5, fcg_net_iters=1),
}


def _step(s, deck, method, n):
    s.load(deck)
    s.step0()
    if method == "mixed_learned":
        s.load_unet(os.path.join(PKG, "weights", "unet_cavity.bin"), (n + 1,) * 3)
    s.run(2)
    return s.state()


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


@pytest.mark.parametrize("method", list(OPTIONS))
def test_small_larger_small(method, tmp_path):
    import cfdfs
    from cfdfs import meshgen
    sizes = [8, 28, 12, 8]
    decks = {n: meshgen.write_cavity(str(tmp_path / f"c{n}.inp"), meshgen.CavitySpec(
        n, re=200, dt=0.002, steps=5, grading=1.0)) for n in set(sizes)}
    new = lambda: cfdfs.Solver(device=0, deterministic=1, **OPTIONS[method])  # noqa: E731
    s = new()
    _step(s, decks[8], method, 8)  # modules loaded, contexts set up
    s.close()
    want, held = {}, {}
    for n in decks:
        before = _free()
        s = new()
        want[n] = _step(s, decks[n], method, n)
        held[n] = before - _free()
        s.close()
    before = _free()
    s = new()
    for n in sizes:
        got = _step(s, decks[n], method, n)
        for a, b in zip(got, want[n]):
            assert np.isfinite(a).all() and np.array_equal(a, b), n
        assert abs(before - _free() - held[n]) <= 64 << 20, n
    # a failed load leaves nothing loaded, and the context usable
    with pytest.raises(cfdfs.CfdError):
        s.load(str(tmp_path / "missing.inp"))
    with pytest.raises(cfdfs.CfdError):
        s.run(1)
    with pytest.raises(cfdfs.CfdError):
        s.checkConvergenceGPU(1e-3)
    got = _step(s, decks[12], method, 12)
    assert all(np.array_equal(a, b) for a, b in zip(got, want[12]))
    s.close()


def test_network_and_grid_of_another_size_are_dropped(tmp_path):
    import cfdfs
    from cfdfs import meshgen
    small = meshgen.write_cavity(str(tmp_path / "a.inp"), meshgen.CavitySpec(8, re=200, dt=0.002, steps=5))
    duct = meshgen.write_duct(str(tmp_path / "d.inp"), n_cross=4, n_axial=20)
    s = cfdfs.Solver(device=0, deterministic=1, **OPTIONS["mixed_learned"])
    _step(s, small, "mixed_learned", 8)
    s.load(duct)  # no grid, no network: Jacobi
    s.step0()
    s.run(1)
    p = s.state()[1]
    s.close()
    s = cfdfs.Solver(device=0, deterministic=1, **OPTIONS["mixed_learned"])
    s.load(duct)
    s.step0()
    s.run(1)
    assert np.array_equal(p, s.state()[1])
    s.close()
    # the same number of nodes: the declared grid stays
    s = cfdfs.Solver(device=0, deterministic=1, **OPTIONS["mixed_twolevel"])
    out = []
    for again in (0, 1):
        s.load(duct)
        s.step0()
        if not again:
            s.set_pressure_grid(meshgen.duct_grid_dims(4, 20))
        s.run(1)
        out.append(s.state()[1])
    assert np.array_equal(out[0], out[1])
    s.close()
