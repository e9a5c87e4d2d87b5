"""The persistent solves when a wait runs out: cfd_selftest_wait_timeout lets the
neighbours' phase and the arrivals of a reduction never come, in both forms of the
by-offsets CG (reductions beside the products and after them) and in the
allocation-free CG, and checks status 3, then a normal solve.  Afterwards the context
and the allocation-free solve work as before."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_waits_give_up_and_solves_go_on(tmp_path):
    import torch
    import cfdfs
    from cfdfs import meshgen
    deck = meshgen.write_cavity(str(tmp_path / "c.inp"), meshgen.CavitySpec(13, grading=1.0))
    s = cfdfs.Solver(device=0, cg_rtol=1e-10, cg_maxit=5000)
    i = s.load(deck)
    s.step0()
    b = np.random.default_rng(0).standard_normal(i.NNp)
    before = s.pressure_solve(b)[0]
    for ms in (20, 60):
        t = time.perf_counter()
        assert s.selftest_wait_timeout(ms) == cfdfs.CFD_E_TIMEOUT
        # nine waits of ms each (a block that starts late ends late), and small solves
        assert 9e-3 * ms <= time.perf_counter() - t <= 30e-3 * ms + 5.0
    x, st = s.pressure_solve(b)
    assert st.status == 0 and np.array_equal(x, before)
    rp, col, val = s.matrix("Z")
    diag = val[np.repeat(np.arange(i.NNp), np.diff(rp)) == col]
    dev = [torch.from_numpy(a).cuda() for a in (rp, col, val, 1.0 / diag, b)]
    y = torch.zeros(i.NNp, dtype=torch.float64, device="cuda")
    rc, info, msg = cfdfs.pcg_solve_noalloc(*[t.data_ptr() for t in dev], y.data_ptr(), i.NNp, 1e-10, 5000,
                                            torch.cuda.current_stream().cuda_stream)
    assert rc == cfdfs.CFD_OK, msg
    assert np.linalg.norm(y.cpu().numpy() - x) <= 1e-5 * np.linalg.norm(x)
    s.close()
