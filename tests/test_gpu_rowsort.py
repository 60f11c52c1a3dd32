"""VT rows at the edges of the row sort's tiers (16 / 24 / 32 entries in a
thread's registers, up to 64 by a warp, longer ones by a heap sort) and of its
shared-memory staging (128 rows that fit, and that do not), against a stable
sort of the cells by vertex on the host.  Whole numbers: equality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _vt(tv, n_verts):
    flat = tv.reshape(-1)
    order = np.argsort(flat, kind="stable")
    off = np.zeros(n_verts + 1, np.int64)
    np.cumsum(np.bincount(flat, minlength=n_verts), out=off[1:])
    return off, (order // 4).astype(np.int32)


# a hub of D cells per entry of the list (its other vertices its own)
@pytest.mark.parametrize("sizes", [[1, 15, 16], [17, 23, 24, 25], [31, 32, 33], [63, 64, 65, 66],
                                   [32] * 64 + [33] * 64, [16, 40, 200, 24, 8] * 30])
def test_rows_of_given_lengths(gpu_lib, sizes):
    rng = np.random.default_rng(len(sizes))
    cells, nv = [], len(sizes)
    for hub, d in enumerate(sizes):
        for _ in range(d):
            cells.append([hub, nv, nv + 1, nv + 2])
            nv += 3
    tv = np.array(cells, dtype=np.int32)[rng.permutation(len(cells))]
    with gpu_lib.Mesh(tv, nv) as g:
        off, ent = g.relation("VT")
    want = _vt(tv, nv)
    assert np.array_equal(off, want[0]) and np.array_equal(ent, want[1])


# random cells over 128 k + r vertices: means of 8 to 94 cells a vertex, past
# what a block stages from 32 on
@pytest.mark.parametrize("n_verts,n_cells", [(128, 256), (129, 1030), (300, 3600), (128, 3000)])
def test_random_rows(gpu_lib, n_verts, n_cells):
    rng = np.random.default_rng(n_cells)
    tv = np.argsort(rng.random((n_cells, n_verts)), axis=1)[:, :4].astype(np.int32)
    with gpu_lib.Mesh(tv, n_verts) as g:
        off, ent = g.relation("VT")
    want = _vt(tv, n_verts)
    assert np.array_equal(off, want[0]) and np.array_equal(ent, want[1])
