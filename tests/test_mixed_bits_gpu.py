"""Deterministic mixed-precision runs repeat recorded pressures: golden/mixed_bits.npz,
from kernels that add every FP64 sum in the order of its entries.  An FP64 sum in
another order differs in its last bit, which is seldom, but in some run, the bit that
decides how a value rounds to FP32; from there the pressure moves by 1e-9 to 3e-8,
through as many inner solves as follow.

Tolerance: sums in the recorded order give the recorded bits; 1e-13 leaves room for
the last bits of the host's arithmetic and none for a value rounded the other way.
"""
import os

import numpy as np
import pytest

from conftest import GOLDEN, PKG, rel_l2

pytestmark = pytest.mark.gpu

OPTIONS = {
    "two": dict(precond=2, cg_warm=1, inner_rtol=1e-5),
    "lrn": dict(precond=1, cg_warm=1, inner_rtol=1e-5, fcg_net_iters=1),
    "jac": dict(precond=0),
}
CASES = [
    # the FP64 residual between inner solves
    "duct_4_40_174.2_two_3", "cav_16_1_27_jac",
    # the lumped mass
    "duct_4_60_174.2_jac_3", "cav_12_1.5_8_jac",
    # the coarse right-hand side of a line cut into ranges
    "duct_6_70_250_two_3",
]


@pytest.mark.parametrize("key", CASES)
def test_recorded_pressure(key, tmp_path):
    import cfdfs
    from cfdfs import meshgen
    part = key.split("_")
    if part[0] == "duct":
        (c, a), re, method, steps = map(int, part[1:3]), float(part[3]), part[4], int(part[5])
        dims = (a + 1, c + 1, c + 1)
        deck = meshgen.write_duct(str(tmp_path / "d.inp"), n_cross=c, n_axial=a, re=re, dt=0.002, steps=100)
    else:
        n, grading, ngp, method, steps = int(part[1]), float(part[2]), int(part[3]), part[4], 2
        dims = (n + 1,) * 3
        deck = meshgen.write_cavity(str(tmp_path / "c.inp"), meshgen.CavitySpec(
            n, re=300, dt=0.001, steps=5, ngp=ngp, grading=grading))
    s = cfdfs.Solver(device=0, precision=cfdfs.MIXED, deterministic=1, **OPTIONS[method])
    s.load(deck)
    s.step0()
    if part[0] == "duct":
        s.set_pressure_grid(meshgen.duct_grid_dims(c, a))
    if method == "lrn":
        s.load_unet(os.path.join(PKG, "weights", "unet_cavity.bin"), dims)
    s.run(steps)
    p = s.state()[1]
    s.close()
    assert rel_l2(p, np.load(os.path.join(GOLDEN, "mixed_bits.npz"))[key]) <= 1e-13
