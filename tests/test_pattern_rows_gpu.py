"""Operator patterns built on the device where a row's candidates stop fitting a
warp (512) and then a block (2048): hexahedra fanned around a common axis, so
that an axis node has 2 m elements.  m = 3 and 9 stay in the warps (18 x 27 =
486 candidates in K), m = 10 puts K's and Z's axis rows on the list of the
blocks, m = 24 gives Z rows that neither holds (the build on the host takes
over).  Integers: equal to the host build."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fan_deck(m, layers):
    from cfdfs import meshgen
    th = 2 * np.pi * np.arange(m) / m
    ring = np.stack([np.cos(th), np.sin(th)], axis=1)
    tip = 1.2 * np.stack([np.cos(th + np.pi / m), np.sin(th + np.pi / m)], axis=1)
    plane = np.concatenate([np.zeros((1, 2)), ring, tip])
    xyz = np.concatenate([np.column_stack([plane, np.full(len(plane), float(k))]) for k in range(layers + 1)])
    conn = []
    for k in range(layers):
        for i in range(m):
            q = np.array([0, 1 + i, 1 + m + i, 1 + (i + 1) % m])
            conn.append(np.concatenate([q + k * len(plane), q + (k + 1) * len(plane)]))
    faces = [(e + 1, 1, 1) for e in range(m)]
    return meshgen.deck_from_arrays(xyz, conn, faces, [(0.0, 0.0, 0.0)], monitor=(0.0, 0.0, 0.0))


@pytest.mark.parametrize("m,layers", [(3, 2), (9, 4), (10, 4), (24, 3)])
def test_rows_of_every_size_equal_the_host_build(m, layers, tmp_path):
    import ctypes as C
    import cfdfs
    from cfdfs import meshgen
    deck = meshgen.write_text(str(tmp_path / "fan.inp"), fan_deck(m, layers))
    h = cfdfs.HostMesh(deck)
    s = cfdfs.Solver(device=0)
    s.load(deck)
    for which in ("K", "G", "GT", "Z"):
        rp_h, col_h = h.pattern(which)
        nnz = C.c_longlong(0)
        w = cfdfs.MAT[which]
        assert s.L.cfd_download_matrix(s.h, w, C.byref(nnz), None, None, None) == 0
        rp = np.zeros(len(rp_h), dtype=np.int32)
        col = np.zeros(nnz.value, dtype=np.int32)
        assert s.L.cfd_download_matrix(s.h, w, C.byref(nnz), cfdfs._p(rp, C.c_int), cfdfs._p(col, C.c_int), None) == 0
        assert np.array_equal(rp, rp_h), which
        assert np.array_equal(col, col_h), which
    s.close()
    h.close()
