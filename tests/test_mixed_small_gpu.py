"""Mixed-precision runs on small meshes give the pressures they gave before the
convection kernel had a finer split for few elements: golden/mixed_small.npz,
recorded with 32 elements per block (two steps from a vortex at rest walls, named
Gauss points, grading, elements per axis, steps).

The convection term is added up in FP32 in the order in which blocks arrive, so a
pass may land one inner iteration away (1e-7) from the others; on these meshes
twelve of twelve recorded passes were equal to the last bit, and most of the passes
here have to be.  Tolerance: everything but that order is FP64 or keeps its order,
so an equal pass differs by FP64 rounding through the refinement only: 1e-9.
"""
import os

import numpy as np
import pytest

from conftest import GOLDEN, rel_l2

pytestmark = pytest.mark.gpu


def _vortex(xyz):
    x, y, z = xyz.T
    s = lambda a: np.sin(np.pi * a) ** 2  # noqa: E731
    d = lambda a: np.pi * np.sin(2 * np.pi * a)  # noqa: E731
    return np.concatenate([0.05 * s(x) * d(y) * s(z), -0.05 * d(x) * s(y) * s(z), np.zeros_like(x)])


@pytest.mark.parametrize("key", ["8_0_7_2", "8_0_8_2", "8_1.5_9_2", "27_0_9_2", "27_1.5_11_2"])
def test_small_mixed_pressure(key, tmp_path):
    import cfdfs
    from cfdfs import meshgen
    ngp, grading, n, steps = int(key.split("_")[0]), float(key.split("_")[1]), *map(int, key.split("_")[2:])
    deck = meshgen.write_cavity(str(tmp_path / "c.inp"), meshgen.CavitySpec(
        n, re=300, dt=0.001, steps=5, ngp=ngp, grading=grading))
    m = cfdfs.HostMesh(deck)
    flow = _vortex(m.coord())
    m.close()
    p_ref = np.load(os.path.join(GOLDEN, "mixed_small.npz"))[key]
    off = []
    for _ in range(3):
        s = cfdfs.Solver(device=0, precision=cfdfs.MIXED)
        s.load(deck)
        s.step0()
        u0, p0 = s.state()
        for _ in range(3):
            s.set_state(u0 + flow, p0)
            s.run(steps)
            off.append(rel_l2(s.state()[1], p_ref))
        s.close()
    assert sorted(off)[len(off) // 2] <= 1e-9, off
