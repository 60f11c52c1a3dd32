"""Offsets where the scan's rows of 64 and tiles of 2048 elements end, by the
number of vertices (most of them in no cell) and of cells.  Against the CPU
oracle; whole numbers: equality."""
import numpy as np
import pytest

from helpers import RELS, assert_relations_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("verts", [63, 64, 65, 66, 2047, 2048, 2049, 4095, 4096, 4097])
def test_vertices(gpu_lib, oracle, verts):
    rng = np.random.default_rng(verts)
    tv = rng.permutation(verts)[: 4 * 15].reshape(15, 4).astype(np.int32)
    tv[0] = [verts - 1, verts - 2, 0, 1]
    ref = oracle.extract(oracle.canonicalize(tv, verts), verts)
    with gpu_lib.Mesh(tv, verts) as g:
        g.extract(gpu_lib.ALL_RELATIONS, options=gpu_lib.OPT_LINK_ADJACENCY)
        assert g.counts() == ref["counts"]
        assert_relations_equal({r: g.relation(r) for r in RELS}, ref)


# occurrence bits: 6 a cell for edges (a tile is 2048 words of 32), 4 for faces
@pytest.mark.parametrize("cells", [341, 342, 10922, 10923, 16384, 16385])
def test_cells(gpu_lib, oracle, cells):
    rng = np.random.default_rng(cells)
    tv = rng.permuted(np.arange(4 * cells).reshape(cells, 4), axis=1).astype(np.int32)
    ref = oracle.extract(oracle.canonicalize(tv, 4 * cells), 4 * cells)
    with gpu_lib.Mesh(tv, 4 * cells) as g:
        g.extract(gpu_lib.ALL_RELATIONS)
        assert g.counts() == ref["counts"]
        assert_relations_equal({r: g.relation(r) for r in RELS}, ref)
