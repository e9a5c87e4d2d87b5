"""The convection term of few elements per launch (16 or 32 threads per element in
FP64) against the CPU oracle's: fewer elements than a block, than a launch of
several blocks, and the sizes on either side of the line to the coarser split
(2368 elements on 148 SMs).

Tolerance: a node adds at most 8 elements' terms, each a sum over 27 nodes and 27
Gauss points; 1e-12 of the vector's norm is some thousand units of FP64, 1e-4 as
many of FP32.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 5, 13, 14])
@pytest.mark.parametrize("ngp", [1, 8, 27])
@pytest.mark.parametrize("mixed", [0, 1])
def test_convection_matches_oracle(n, ngp, mixed, tmp_path, oracle_mod):
    import cfdfs
    from cfdfs import meshgen
    deck = meshgen.write_cavity(str(tmp_path / "c.inp"), meshgen.CavitySpec(n, re=200, dt=0.002, ngp=ngp, grading=1.2))
    o = oracle_mod.Oracle(deck)
    o.step0()
    s = cfdfs.Solver(device=0, precision=cfdfs.MIXED if mixed else cfdfs.FP64)
    s.load(deck)
    s.step0()
    u = np.random.default_rng(n).standard_normal(3 * o.NN)
    s.set_state(u, np.zeros(o.NNp))
    o.set_vec("Un", u)
    o.begin_step()
    s.begin_step()
    o.convect()
    o.step1(1)
    s.calculateMatrixAGPU()
    s.step1GPUpart(1)
    assert rel_l2(s.vector("R1"), o.vec("R1")) <= (1e-4 if mixed else 1e-12)
    s.close()
    o.close()
