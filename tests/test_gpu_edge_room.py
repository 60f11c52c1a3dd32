"""Meshes of more than 2^20 cells whose edges just fit the room that their cells
and vertices suggest, and just do not (the star pass runs again), with stars of
32 to 64 and of more than 64 cells among the rest.  Every relation against the
CPU oracle; whole numbers: equality."""
import numpy as np
import pytest

from helpers import RELS, assert_relations_equal

pytestmark = pytest.mark.gpu

CELLS = (1 << 20) + 5


def _ring(k):
    return np.array([[0, 1, 2 + i, 2 + (i + 1) % k] for i in range(k)]), k + 2


def _mesh(more):
    """Cells of random vertices (nearly six edges each) and rings, with as many
    vertices besides that CELLS + 2 n_verts is the number of edges (more = 0) or
    two below it (more = 2)."""
    rng = np.random.default_rng(3)
    tvs, n = [], 0
    for k in (40, 64, 65, 90):
        tv, m = _ring(k)
        tvs.append(tv + n)
        n += m
    rest = CELLS - sum(len(t) for t in tvs)
    cells = np.sort(rng.integers(0, CELLS // 2, (rest, 4)), 1)
    cells = cells + np.arange(4)                 # distinct
    tv = np.concatenate([cells + n] + tvs)
    n += CELLS // 2 + 3
    while True:
        pairs = np.concatenate([np.sort(tv[:, [a, b]], 1) for a in range(4) for b in range(a + 1, 4)])
        edges = len(np.unique(pairs[:, 0] * n + pairs[:, 1]))
        if (edges - CELLS) % 2 == 0:
            break
        tv[0] = [n, n + 1, tv[0, 2], tv[0, 3]]   # one edge of cell 0 kept, whatever it was
        n += 2
    verts = (edges - CELLS - more) // 2
    assert verts >= n and len(tv) == CELLS
    return rng.permutation(verts)[tv].astype(np.int32), verts, edges


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
