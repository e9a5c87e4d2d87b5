"""FP64 pressure solves of right-hand sides of very small and very large norm: scaling
by a power of two scales every number of the iteration exactly, until r^T D^-1 r leaves
the normal range, and the solve still ends at its tolerance there.

Tolerance: inside the normal range the solution is the scaled one to the last bit.
Below it a dot product keeps 12 digits and more down to 1e-312; the solve stops at
||r|| <= 1e-8 ||b|| with a condition number below 2e3: 2e-5, and 1e-4 is asserted.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 8, 11, 14])
def test_solution_scales_with_the_right_hand_side(n, tmp_path):
    import cfdfs
    from cfdfs import meshgen
    deck = meshgen.write_cavity(str(tmp_path / "c.inp"), meshgen.CavitySpec(n, grading=1.0))
    s = cfdfs.Solver(device=0, cg_rtol=1e-8, cg_maxit=2000)
    i = s.load(deck)
    s.step0()
    rp, col, val = s.matrix("Z")
    diag = val[[rp[r] + int(np.searchsorted(col[rp[r]:rp[r + 1]], r)) for r in range(i.NNp)]]
    b = np.random.default_rng(1).standard_normal(i.NNp)
    x, st = s.pressure_solve(b)
    assert st.status == 0
    for k in (-300, -40, 40, 300):
        y, sy = s.pressure_solve(np.ldexp(b, k))
        assert sy.iterations == st.iterations and np.array_equal(np.ldexp(y, -k), x), k
    # r^T D^-1 r falls from 1e-298 to about 1e-314 in the course of the solve
    g = float((b * b / diag).sum())
    k = int(np.floor(0.5 * np.log2(1e-298 / g)))
    y, sy = s.pressure_solve(np.ldexp(b, k))
    assert sy.status == 0
    assert np.linalg.norm(np.ldexp(y, -k) - x) <= 1e-4 * np.linalg.norm(x)
    s.close()
