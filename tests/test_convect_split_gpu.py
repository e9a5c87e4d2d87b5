"""The convection term with few elements per launch (16 or 32 threads per element)
and with many (4): a deterministic context launches one colour at a time, so its
launches are small where the other context's single launch is not.

Tolerance: every element's sums run in the same order in both; a node adds the
terms of at most 8 elements in another order, 8 x 2^-53 (FP32: 2^-24) of their
magnitudes: 1e-12 and 1e-5 of the vector's norm leave room for cancellation.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5, 13, 14, 17, 18])
@pytest.mark.parametrize("ngp", [1, 8, 27])
@pytest.mark.parametrize("mixed", [0, 1])
def test_small_and_large_launches_agree(n, ngp, mixed, tmp_path):
    import cfdfs
    from cfdfs import meshgen
    deck = meshgen.write_cavity(str(tmp_path / "c.inp"), meshgen.CavitySpec(n, re=200, dt=0.002, ngp=ngp, grading=1.2))
    out = []
    for det in (0, 1):
        s = cfdfs.Solver(device=0, precision=cfdfs.MIXED if mixed else cfdfs.FP64, deterministic=det)
        i = s.load(deck)
        s.step0()
        rng = np.random.default_rng(n)
        s.set_state(rng.standard_normal(3 * i.NN), np.zeros(i.NNp))
        s.begin_step()
        s.calculateMatrixAGPU()
        s.step1GPUpart(1)
        out.append(s.vector("R1"))
        s.close()
    assert np.isfinite(out[1]).all()
    assert np.linalg.norm(out[0] - out[1]) <= (1e-5 if mixed else 1e-12) * np.linalg.norm(out[1])
