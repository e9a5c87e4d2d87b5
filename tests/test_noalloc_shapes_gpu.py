"""cfd_pcg_solve_noalloc over the row lengths and sizes its kernel switches on:
lanes per row from the mean length (2, 4, 8, 16, 32), rows longer than one
pass of a group's loads, one block against several, block ranges that do not
divide n.

Tolerance: the matrices are symmetric and strictly diagonally dominant with
unit-scaled condition number at most 4, so ||r|| <= 1e-11 ||b|| bounds the
relative error by 4e-11; 1e-10 is asserted.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n, per_row, seed):
    """Symmetric CSR matrix with about per_row entries per row (one row in 50
    five times as long), off-diagonal row sums at most 0.6 of the diagonal."""
    rng = np.random.default_rng(seed)
    half = max(0, (per_row - 1) // 2)
    i = np.repeat(np.arange(n), half)
    j = (i + rng.integers(1, max(2, n // 2), size=i.size)) % n
    for r in range(0, n, 50):
        k = rng.integers(0, n, size=2 * per_row)
        i, j = np.concatenate([i, np.full(k.size, r)]), np.concatenate([j, k])
    a = {}
    for r, c in zip(i.tolist(), j.tolist()):
        if r != c:
            v = float(rng.uniform(-1.0, 1.0))
            a[(r, c)] = v
            a[(c, r)] = v
    rows = [[] for _ in range(n)]
    for (r, c), v in a.items():
        rows[r].append((c, v))
    rp, col, val = [0], [], []
    for r in range(n):
        d = max(1.0, sum(abs(v) for _, v in rows[r]) / 0.6)
        ent = sorted(rows[r] + [(r, d)])
        col += [c for c, _ in ent]
        val += [v for _, v in ent]
        rp.append(len(col))
    return np.array(rp, np.int32), np.array(col, np.int32), np.array(val)


@pytest.mark.parametrize("n,per_row", [(1, 1), (7, 3), (511, 7), (512, 13), (513, 27), (1025, 41), (2000, 101),
                                       (40001, 9)])
def test_noalloc_row_lengths(n, per_row):
    import torch
    import cfdfs
    rp, col, val = _system(n, per_row, n + per_row)
    rows = np.repeat(np.arange(n), np.diff(rp))
    x_true = np.random.default_rng(5).standard_normal(n)
    b = np.zeros(n)
    np.add.at(b, rows, val * x_true[col])
    diag = val[rows == col]
    dev = [torch.from_numpy(a).cuda() for a in (rp, col, val, 1.0 / diag, b)]
    x = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
    rc, info, msg = cfdfs.pcg_solve_noalloc(*[t.data_ptr() for t in dev], x.data_ptr(), n, 1e-11, 500,
                                            torch.cuda.current_stream().cuda_stream)
    assert rc == cfdfs.CFD_OK, msg
    assert info[1] <= 1e-11
    assert np.linalg.norm(x.cpu().numpy() - x_true) <= 1e-10 * np.linalg.norm(x_true)
    # too few iterations: reported, with the iterate of the last one
    if info[0] > 1:
        rc, part, _ = cfdfs.pcg_solve_noalloc(*[t.data_ptr() for t in dev], x.data_ptr(), n, 1e-11, 1,
                                              torch.cuda.current_stream().cuda_stream)
        assert rc == cfdfs.CFD_E_NOCONV and part[0] == 1
