"""cfd_pcg_solve_noalloc as on a device or partition of few SMs (CFD_NOALLOC_SMS), whose
shared memory does not hold the vectors: one block, several, row ranges that do not
divide n, the last size that fits a block (5120 rows) and the first that does not.

Tolerance: as in test_noalloc_shapes_gpu.py, 1e-10 of the solution's norm.
"""
import numpy as np
import pytest

from test_noalloc_shapes_gpu import _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sms,n,per_row", [(1, 5120, 7), (1, 5121, 7), (2, 10241, 13), (7, 40001, 9), (3, 17000, 27)])
def test_few_sms(sms, n, per_row, monkeypatch):
    import torch
    import cfdfs
    rp, col, val = _system(n, per_row, n + per_row)
    rows = np.repeat(np.arange(n), np.diff(rp))
    x_true = np.random.default_rng(5).standard_normal(n)
    b = np.zeros(n)
    np.add.at(b, rows, val * x_true[col])
    diag = val[rows == col]
    dev = [torch.from_numpy(a).cuda() for a in (rp, col, val, 1.0 / diag, b)]
    out = {}
    for limit in (sms, 148, sms):
        monkeypatch.setenv("CFD_NOALLOC_SMS", str(limit))
        x = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
        free = torch.cuda.mem_get_info(0)[0]
        rc, info, msg = cfdfs.pcg_solve_noalloc(*[t.data_ptr() for t in dev], x.data_ptr(), n, 1e-11, 500,
                                                torch.cuda.current_stream().cuda_stream)
        assert rc == cfdfs.CFD_OK, msg
        assert info[1] <= 1e-11
        assert np.linalg.norm(x.cpu().numpy() - x_true) <= 1e-10 * np.linalg.norm(x_true)
        if limit in out:  # a second call allocates nothing and repeats the first
            assert torch.cuda.mem_get_info(0)[0] == free
            assert torch.equal(out[limit], x)
        out[limit] = x.clone()
    rc, part, _ = cfdfs.pcg_solve_noalloc(*[t.data_ptr() for t in dev], x.data_ptr(), n, 1e-11, 1,
                                          torch.cuda.current_stream().cuda_stream)
    assert rc == cfdfs.CFD_E_NOCONV and part[0] == 1


def test_limits_are_unchanged(monkeypatch):
    import torch
    import cfdfs
    monkeypatch.setenv("CFD_NOALLOC_SMS", "1")
    p = torch.zeros(4, dtype=torch.float64, device="cuda").data_ptr()
    rc, _, msg = cfdfs.pcg_solve_noalloc(p, p, p, p, p, p, cfdfs.NOALLOC_MAX_N + 1, 1e-8, 10, 0)
    assert rc == cfdfs.CFD_E_BADARG and "524288" in msg
