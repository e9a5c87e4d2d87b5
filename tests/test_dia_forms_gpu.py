"""The pressure operator by offsets and in the SELL-32 form (CFD_DIA=0; also what a
context falls back to where device memory is short): the FP64 residual of mixed runs is
equal to the last bit, so deterministic mixed runs are; FP64 solves add in other orders.

Tolerance of the FP64 solves: both stop at ||r|| <= 1e-10 ||b|| of the same operator,
whose condition number is below 2e3 at these sizes (scaled by the diagonal, which
varies by less than 2e3): 2e3 x 1e-10 x sqrt(2e3) = 1e-5.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(dia, **kw):
    import cfdfs
    os.environ["CFD_DIA"] = "1" if dia else "0"
    try:
        return cfdfs.Solver(device=0, **kw)
    finally:
        del os.environ["CFD_DIA"]


def _deck(shape, path):
    from cfdfs import meshgen
    if len(shape) == 2:
        return meshgen.write_duct(path, n_cross=shape[0], n_axial=shape[1], dt=0.002), meshgen.duct_grid_dims(*shape)
    return meshgen.write_cavity(path, meshgen.CavitySpec(shape[0], re=200, dt=0.002, grading=1.2)), None


@pytest.mark.parametrize("shape", [(1,), (5,), (12,), (18,), (3, 40), (6, 31)])
@pytest.mark.parametrize("precond", [0, 2])
def test_mixed_runs_are_equal(shape, precond, tmp_path):
    import cfdfs
    if precond == 2 and shape == (1,):
        pytest.skip("no coarse space on eight nodes")
    deck, dims = _deck(shape, str(tmp_path / "d.inp"))
    out = []
    for dia in (1, 0):
        s = _solver(dia, precision=cfdfs.MIXED, precond=precond, deterministic=1, cg_warm=1)
        s.load(deck)
        s.step0()
        if dims:
            s.set_pressure_grid(dims)
        s.run(2)
        out.append(s.state())
        s.close()
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)


@pytest.mark.parametrize("shape", [(5,), (13,), (4, 37)])
@pytest.mark.parametrize("precond", [0, 2])
def test_fp64_solves_agree(shape, precond, tmp_path):
    deck, dims = _deck(shape, str(tmp_path / "d.inp"))
    out = []
    for dia in (1, 0):
        s = _solver(dia, precond=precond, cg_rtol=1e-10, cg_maxit=5000)
        i = s.load(deck)
        for _ in range(2):  # Z assembled again: the forms are filled again
            s.step0()
            if dims:
                s.set_pressure_grid(dims)
            b, g = (np.random.default_rng(k).standard_normal(i.NNp) for k in (1, 2))
            s.set_options(cg_warm=0)
            cold = s.pressure_solve(b)[0]
            s.set_options(cg_warm=1)
            warm = s.pressure_solve(b, g)[0]
            s.set_options(precond=0)
            jac = s.pressure_solve(b, g)[0]
            s.set_options(precond=precond)
        out.append((cold, warm, jac))
        s.close()
    for x in out[0] + out[1]:
        assert np.linalg.norm(x - out[0][0]) <= 1e-5 * np.linalg.norm(out[0][0])
