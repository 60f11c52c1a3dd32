"""Meshes of more than 2^20 cells with few and with many edges a cell: room for
two edges a cell at first, for six when that is not enough; just
below and just above, with stars of 32 to 64 and of more than 64 cells among
the rest.  Every relation against the CPU oracle; whole numbers: equality."""
import numpy as np
import pytest

from helpers import RELS, assert_relations_equal
from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu

CELLS = 1 << 20


def _ring(k):
    return np.array([[0, 1, 2 + i, 2 + (i + 1) % k] for i in range(k)]), k + 2


def _mesh(more):
    """CELLS cells: a grid, rings, and cells that share nothing, as many that
    2 CELLS edges are just reached (more = 0) or passed by two (more = 2)."""
    grid = meshgen.kuhn_mesh((52, 53, 51), 0.0, seed=3)
    tvs, n = [grid.tv], grid.n_verts
    for k in (40, 64, 65, 90):
        tv, m = _ring(k)
        tvs.append(tv + n)
        n += m
    rest = CELLS - sum(len(t) for t in tvs)
    # edges: of the grid and the rings (3 k + 1 each), 6 a cell that shares
    # nothing, 3 more for a cell glued to the one before
    pairs = np.sort(np.concatenate([grid.tv[:, [a, b]] for a in range(4) for b in range(a + 1, 4)]), 1)
    have = len(np.unique(pairs[:, 0].astype(np.int64) * n + pairs[:, 1])) + sum(3 * k + 1 for k in (40, 64, 65, 90))
    want = 2 * CELLS + more
    glued = 6 * rest - (want - have)          # each of the 3 lost per glued cell, then 1 per shared edge
    by_face, by_edge = glued // 3, glued % 3
    assert 0 < by_face + by_edge <= rest // 2
    tv = np.arange(4 * rest).reshape(rest, 4)
    a = tv[0:2 * by_face:2]
    tv[1:2 * by_face:2, :3] = a[:, :3]        # a face in common
    a = tv[2 * by_face:2 * (by_face + by_edge):2]
    tv[2 * by_face + 1:2 * (by_face + by_edge):2, :2] = a[:, :2]
    tvs.append(tv + n)
    n += 4 * rest
    tv = np.concatenate(tvs)
    assert len(tv) == CELLS
    return np.random.default_rng(4).permutation(n)[tv].astype(np.int32), n, want


@pytest.mark.parametrize("more", [0, 2])
def test_room(gpu_lib, oracle, more):
    tv, n, edges = _mesh(more)
    tvs = oracle.canonicalize(tv, n)
    ref = oracle.extract(tvs, n)
    with gpu_lib.Mesh(tv, n) as g:
        g.extract(gpu_lib.ALL_RELATIONS)
        assert g.counts() == ref["counts"] and g.counts()[1] == edges
        assert_relations_equal({r: g.relation(r) for r in RELS}, ref)
    with gpu_lib.Mesh(tv, n) as g:           # a pass that needs no ids
        g.extract(["VV"])
        assert_relations_equal({"VV": g.relation("VV")}, ref, ["VV"])
