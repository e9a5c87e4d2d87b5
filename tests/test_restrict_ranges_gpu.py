"""The linear two-level preconditioner z = D^-1 r + P Zc^-1 P^T r on grids whose
restriction splits the coarse x-nodes into ranges (long axis, few y-z pairs) and on
grids where it does not, against the dense product built on the host.

Tolerance: the device rounds the coarse inverse to FP16 (2^-11 of its largest entry
per entry) and the coarse vectors to FP32; relative to the correction's norm that
stays below 5e-3, while a lost or doubled coarse node changes it by O(1) in its
neighbourhood.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hats(n, ncd):
    """(n, ncd) trilinear weights of one axis, as the solver's lattice."""
    w = np.zeros((n, ncd))
    if ncd == 1:
        w[:, 0] = 1.0
        return w
    h = (n - 1) / (ncd - 1)
    for x in range(n):
        i = min(max(int(np.floor(x / h)), 0), ncd - 2)
        f = min(max(x / h - i, 0.0), 1.0)
        w[x, i] += 1.0 - f
        w[x, i + 1] += f
    return w


@pytest.mark.parametrize("n_cross,n_axial", [(4, 16), (4, 61), (6, 97), (9, 40), (5, 130)])
def test_two_level_apply(n_cross, n_axial, tmp_path):
    import cfdfs
    from cfdfs import meshgen
    deck = meshgen.write_duct(str(tmp_path / "d.inp"), n_cross=n_cross, n_axial=n_axial, steps=2)
    dims = meshgen.duct_grid_dims(n_cross, n_axial)
    s = cfdfs.Solver(device=0, precond=cfdfs.PC_TWOLEVEL)
    s.load(deck)
    s.step0()
    s.set_pressure_grid(dims)
    rp, col, val = s.matrix("Z")
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    diag = val[rows == col]
    cd, inv = cfdfs.coarse_inverse(dims, rp, col, val)
    wx, wy, wz = (_hats(n, c) for n, c in zip(dims, cd))
    rng = np.random.default_rng(8)
    for r in (rng.standard_normal(len(diag)), np.ones(len(diag))):
        g = r.reshape(dims[::-1])
        c = np.einsum("zyx,xi,yj,zk->kji", g, wx, wy, wz, optimize=True).reshape(-1)
        e = (inv @ c).reshape(cd[::-1])
        corr = np.einsum("kji,xi,yj,zk->zyx", e, wx, wy, wz, optimize=True).reshape(-1)
        got = s.precond_apply(r) - r / diag
        assert np.linalg.norm(got - corr) <= 5e-3 * np.linalg.norm(corr)
        assert np.max(np.abs(got - corr)) <= 2e-2 * np.max(np.abs(corr))
    s.close()
