"""The FP64 solves on the pressure matrix stored by offsets (pcg_dia.cu: the
Jacobi-PCG, the two-level flexible CG's SpMV, the residual) against the general
kernels: the same mesh with its corner nodes renumbered at
random has the same Z up to a permutation, but no few-diagonal form, so it takes
the SELL-32 kernel.

Sizes: matrices of one slice, of fewer groups than warps, one to three slices per
block, every SM busy, a duct (unequal axes), a graded mesh.  Tolerance: both stop
at ||r|| <= 1e-10 ||b||, and the condition number of the Jacobi-scaled Z is below
about 2e3 at these sizes, so the solutions agree to 2 x 2e3 x 1e-10 = 4e-7.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _decks(tmp_path, kind, n):
    from cfdfs import meshgen
    if kind == "duct":
        xyz, conn, inlet, walls, _ = meshgen.duct_arrays(*n)
        faces = np.array([(e, f, 1) for e, f in inlet] + [(e, f, 2) for e, f in walls])
        bcs = [(1.0, 0.0, 0.0), (0.0, 0.0, 0.0)]
    else:
        xyz, conn, faces = meshgen.cavity_arrays(n, 1.5 if kind == "graded" else 0.0)
        bcs = [(0.0, 0.0, 0.0), (1.0, 0.0, 0.0)]
    perm = np.random.default_rng(7).permutation(len(xyz))  # old node -> new node
    inv = np.argsort(perm)
    zp = len(xyz) // 2 + 1  # 1-based pinned node, old numbering
    a = meshgen.deck_from_arrays(xyz, conn, faces, bcs, zero_p_node1=zp)
    b = meshgen.deck_from_arrays(xyz[inv], perm[conn], faces, bcs, zero_p_node1=int(perm[zp - 1]) + 1)
    pa, pb = str(tmp_path / "a.inp"), str(tmp_path / "b.inp")
    meshgen.write_text(pa, a)
    meshgen.write_text(pb, b)
    return pa, pb, perm


@pytest.mark.parametrize("kind,n", [("cavity", 2), ("cavity", 3), ("cavity", 8), ("graded", 11), ("cavity", 15),
                                    ("duct", (4, 37)), ("graded", 18), ("cavity", 27), ("duct", (9, 60))])
@pytest.mark.parametrize("warm", [0, 1])
def test_offsets_form_matches_general(kind, n, warm, tmp_path):
    import cfdfs
    pa, pb, perm = _decks(tmp_path, kind, n)
    xs, its = [], []
    rng = np.random.default_rng(3)
    rhs = x0 = None
    for path in (pa, pb):
        s = cfdfs.Solver(device=0, cg_rtol=1e-10, cg_maxit=5000, cg_warm=warm)
        i = s.load(path)
        s.step0()
        if rhs is None:
            rhs, x0 = rng.standard_normal(i.NNp), rng.standard_normal(i.NNp)
            b, g = rhs, x0
        else:
            b, g = np.empty_like(rhs), np.empty_like(x0)
            b[perm], g[perm] = rhs, x0
        x, st = s.pressure_solve(b, g if warm else None)
        assert st.status == 0 and st.relres <= 1e-10
        r, nr = s.pressure_residual(b, x)
        assert nr <= 1.1e-10 * np.linalg.norm(b)
        xs.append(x if path == pa else x[perm])
        its.append(st.iterations)
        # a zero right-hand side, and an iteration limit
        if not warm:
            z, st0 = s.pressure_solve(np.zeros(i.NNp))
            assert st0.iterations == 0 and not z.any()
            s.set_options(cg_maxit=3)
            _, st3 = s.pressure_solve(b)
            assert st3.status == 1 and st3.iterations == 3
        s.close()
    assert abs(its[0] - its[1]) <= 2
    assert np.linalg.norm(xs[0] - xs[1]) <= 4e-7 * np.linalg.norm(xs[1])


@pytest.mark.parametrize("kind,n", [("cavity", 4), ("graded", 12), ("duct", (8, 40)), ("cavity", 21)])
def test_offsets_form_two_level(kind, n, tmp_path):
    """FP64 two-level solves and a mixed solve's FP64 refinement on both forms."""
    import cfdfs
    from cfdfs import meshgen
    pa, pb, perm = _decks(tmp_path, kind, n)
    dims = meshgen.duct_grid_dims(*n) if kind == "duct" else (n + 1,) * 3
    rhs = np.random.default_rng(4).standard_normal(len(perm))
    b = np.empty_like(rhs)
    b[perm] = rhs
    for precision in (cfdfs.FP64, cfdfs.MIXED):
        got = []
        for path, f, pmap in ((pa, rhs, None), (pb, b, perm)):
            s = cfdfs.Solver(device=0, precision=precision, precond=cfdfs.PC_TWOLEVEL, cg_rtol=1e-10)
            s.load(path)
            s.step0()
            s.set_pressure_grid(dims, pmap)
            x, st = s.pressure_solve(f)
            assert st.status == 0 and st.fallback == 0 and st.relres <= 1e-10
            got.append((x if pmap is None else x[perm], st.iterations))
            s.close()
        assert abs(got[0][1] - got[1][1]) <= 2 + (precision == cfdfs.MIXED) * 8
        assert np.linalg.norm(got[0][0] - got[1][0]) <= 4e-7 * np.linalg.norm(got[1][0])
