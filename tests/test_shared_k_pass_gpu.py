"""cfd_run computes K Acc_prev in step 1's pass over K; the stage calls compute it
in a pass of its own (calculate_KtimesAcc_prev).  Both loops, on cavities that
reach every way to share a slice, with steps that converge and steps that run
out of sub-iterations.

Mixed precision adds a row's products in the order of the entries in both, so in
deterministic mode every number is equal.  FP64 may share a slice between other
numbers of warps, which reorders at most 125 products (1e-13 of K Acc); that can
move the CG across its 1e-8 stopping test by one iteration: 1e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,max_iter,tol", [(2, 3, 1e-30), (3, 10, 1e-3), (9, 2, 1e-30), (16, 4, 1e-3), (25, 3, 1e-30)])
@pytest.mark.parametrize("mixed", [0, 1])
def test_run_equals_stage_calls(n, max_iter, tol, mixed, tmp_path):
    import cfdfs
    from cfdfs import meshgen
    deck = meshgen.write_cavity(str(tmp_path / "c.inp"), meshgen.CavitySpec(
        n, re=200, dt=0.002, steps=4, max_iter=max_iter, tol=tol, converge=1e-30))
    out = []
    for staged in (0, 1):
        s = cfdfs.Solver(device=0, precision=cfdfs.MIXED if mixed else cfdfs.FP64, deterministic=1)
        s.load(deck)
        s.step0()
        if staged:
            for _ in range(2):
                s.time_step()
        else:
            s.run(2)
        out.append(list(s.state()) + [s.vector("KtimesAcc_prev")])
        s.close()
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.linalg.norm(b) > 0
        if mixed:
            assert np.array_equal(a, b)
        else:
            assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(b)
