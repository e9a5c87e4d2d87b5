"""The pressure solve of small structured grids in one cluster of blocks
(pcg_dia.cu): the fewest rows, one and several slices and tap groups per block and
warp, the last grid that fits and the first that does not, unequal axes.  Against a
direct solve of the downloaded matrix.

Tolerance: the solve stops at ||r|| <= 1e-10 ||b||; the Jacobi-scaled Z has a
condition number below 2e3 at these sizes, and its diagonal varies by less than 2e3
but for the pinned row, so the solution is within 2e3 x 1e-10 x sqrt(2e3) = 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 5, 9, 10, 11, 12, (2, 50), (4, 37)])
def test_small_solves(n, tmp_path):
    import scipy.sparse as sp
    import scipy.sparse.linalg as sl
    import cfdfs
    from cfdfs import meshgen
    if isinstance(n, tuple):
        deck = meshgen.write_duct(str(tmp_path / "d.inp"), n_cross=n[0], n_axial=n[1])
    else:
        deck = meshgen.write_cavity(str(tmp_path / "c.inp"), meshgen.CavitySpec(n, grading=1.0))
    rng = np.random.default_rng(8)
    for warm in (0, 1):
        s = cfdfs.Solver(device=0, cg_rtol=1e-10, cg_maxit=5000, cg_warm=warm)
        i = s.load(deck)
        s.step0()
        rp, col, val = s.matrix("Z")
        Z = sp.csr_matrix((val, col, rp), shape=(i.NNp, i.NNp)).tocsc()
        for _ in range(3):
            b, g = rng.standard_normal(i.NNp), rng.standard_normal(i.NNp)
            x, st = s.pressure_solve(b, g if warm else None)
            assert st.status == 0 and st.relres <= 1e-10
            assert s.pressure_residual(b, x)[1] <= 1.1e-10 * np.linalg.norm(b)
            y = sl.spsolve(Z, b)
            assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y)
        x, st = s.pressure_solve(np.zeros(i.NNp), g if warm else None)
        assert st.status == 0 and st.iterations == 0 and not x.any()
        s.set_options(cg_maxit=2)
        x, st = s.pressure_solve(b, np.zeros(i.NNp) if warm else None)
        assert st.iterations <= 2 and (st.status == 1) == (st.relres > 1e-10)
        bad = b.copy()
        bad[i.NNp // 2] = np.nan
        with pytest.raises(cfdfs.CfdError, match="non-finite"):
            s.pressure_solve(bad, np.zeros(i.NNp) if warm else None)
        s.close()
