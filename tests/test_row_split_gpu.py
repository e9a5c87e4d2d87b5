"""The stage kernels that share a matrix slice between 1, 2, 4 or 8 warps
(steps.cu), against the downloaded CSR operators, at sizes that reach every
split, a last block with idle slices and a last slice with idle rows.

Tolerances: FP64 rows have at most 125 products, so a reordered sum differs by
at most 125 x 2^-53 of the sum of magnitudes; 1e-12 relative to the vector's norm
leaves room for cancellation.  Mixed precision rounds operators, gathered vectors
and sums to FP32 (2^-24 per operation, 128 operations at most): 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mul(csr, x, n):
    rp, col, val = csr
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    y = np.zeros(n)
    np.add.at(y, rows, val * x[col])
    return y


@pytest.mark.parametrize("n", [2, 3, 8, 16, 31, 40])
@pytest.mark.parametrize("mixed", [0, 1])
def test_stage_products(n, mixed, tmp_path):
    import cfdfs
    from cfdfs import meshgen
    deck = meshgen.write_cavity(str(tmp_path / "c.inp"), meshgen.CavitySpec(n, re=200, dt=0.002, steps=4))
    s = cfdfs.Solver(device=0, precision=cfdfs.MIXED if mixed else cfdfs.FP64)
    info = s.load(deck)
    s.step0()
    NN, NNp, dt = info.NN, info.NNp, info.dt
    rng = np.random.default_rng(n)
    U, P = s.state()
    free = s.vector("MdInv").reshape(3, NN)[0] != 1.0
    U = (U.reshape(3, NN) + 0.1 * rng.standard_normal((3, NN)) * free).reshape(-1)
    s.set_state(U, rng.standard_normal(NNp))
    K, G, GT = s.matrix("K"), s.matrix("G"), s.matrix("GT")
    tol = 1e-5 if mixed else 1e-12

    def close(a, b):
        return np.linalg.norm(a - b) <= tol * max(np.linalg.norm(b), 1e-300)

    s.begin_step()
    Un, Pn = s.vector("Un").reshape(3, NN), s.vector("Pn")
    s.calculateMatrixAGPU()
    s.step1GPUpart(1)
    R1a = s.vector("R1").reshape(3, NN)
    # without pressure, and with the velocity doubled in K only through linearity:
    # R1(P) - R1(0) = -G P, both from the same convection term
    s.set_state(U, np.zeros(NNp))
    s.begin_step()
    s.calculateMatrixAGPU()
    s.step1GPUpart(1)
    R1b = s.vector("R1").reshape(3, NN)
    for d in range(3):
        gp = _mul((G[0], G[1], G[2][:, d]), Pn, NN)
        scale = np.linalg.norm(R1b[d]) + np.linalg.norm(gp)
        assert np.linalg.norm((R1a[d] - R1b[d] + gp) * free) <= tol * scale, d
    h = s.vector("UnpHalf").reshape(3, NN)
    s.step2GPU(1)
    r2 = sum(_mul((GT[0], GT[1], GT[2][:, d]), h[d] / dt**2, NNp) for d in range(3))
    r2[info.zeroPressureNode] = 0.0 if info.zeroPressureNode > 0 else r2[info.zeroPressureNode]
    big = sum(_mul((GT[0], GT[1], np.abs(GT[2][:, d])), np.abs(h[d]) / dt**2, NNp) for d in range(3))
    assert np.linalg.norm(s.vector("R2") - r2) <= tol * np.linalg.norm(big)
    pd = s.vector("Pdot")
    s.step3GPU(1)
    acc, minv = s.vector("Acc").reshape(3, NN), s.vector("MdInv").reshape(3, NN)[0]
    for d in range(3):
        gp = _mul((G[0], G[1], G[2][:, d]), pd, NN)
        assert close(acc[d], -dt * gp * minv * free), d
    assert close(s.vector("Unp1"), s.vector("UnpHalf") + dt * acc.reshape(-1))
    s.rotate()
    s.calculate_KtimesAcc_prevGPU()
    ka, ap = s.vector("KtimesAcc_prev").reshape(3, NN), s.vector("Acc_prev").reshape(3, NN)
    for d in range(3):
        ref = _mul(K, ap[d], NN)
        scale = np.linalg.norm(_mul((K[0], K[1], np.abs(K[2])), np.abs(ap[d]), NN))
        assert np.linalg.norm(ka[d] - ref) <= tol * scale, d
    s.close()
