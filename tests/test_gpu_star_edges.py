"""The star pass and the per-edge passes at the sizes where their tiles end:
stars of 31 cells (one lane a cell) to 64 (two), edges of 16 cells (what an
edge lists at a time) and more, blocks whose vertices own more edges than
their shared memory keeps, cell counts around the blocks' 256.  Every relation
and the classes against the CPU oracle; whole numbers: equality."""
import numpy as np
import pytest

from helpers import RELS, assert_relations_equal
from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _check(tg, oracle, tv, n):
    tvs = oracle.canonicalize(tv, n)
    ref = oracle.extract(tvs, n)
    field = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    with tg.Mesh(tv, n) as g:
        g.extract(tg.ALL_RELATIONS, options=tg.OPT_LINK_ADJACENCY)
        assert g.counts() == ref["counts"]
        assert_relations_equal({r: g.relation(r) for r in RELS}, ref)
        assert np.array_equal(g.critical_points(field), oracle.critical_points(tvs, n, field))


@pytest.mark.parametrize("k", [15, 16, 17, 31, 32, 33, 48, 49, 63, 64])
def test_ring(gpu_lib, oracle, k):
    # k cells around the axis (0, 1), closed; an open one beside it (a cell
    # left out: the axis is on the boundary)
    rng = np.random.default_rng(k)
    ring = np.array([[0, 1, 2 + i, 2 + (i + 1) % k] for i in range(k)])
    tv = np.concatenate([ring, ring[:-1] + k + 2])
    n = 2 * (k + 2)
    tv = rng.permuted(rng.permutation(n)[tv], axis=1).astype(np.int32)
    _check(gpu_lib, oracle, tv, n)


@pytest.mark.parametrize("hubs,cells", [(4, 7), (16, 10), (40, 31), (20, 60), (1, 64)])
def test_hubs_owning_many_edges(gpu_lib, oracle, hubs, cells):
    # hubs with the lowest ids, 3 * cells neighbours each, one after another
    # in the processing order
    tv, n = [], hubs
    for _ in range(cells):
        for h in range(hubs):
            tv.append([h, n, n + 1, n + 2])
            n += 3
    _check(gpu_lib, oracle, np.array(tv, dtype=np.int32), n)


@pytest.mark.parametrize("dims,coned", [((1, 1, 1), 0.0), ((42, 1, 1), 0.0), ((43, 1, 1), 0.0),
                                        ((7, 6, 1), 0.0), ((11, 5, 3), 0.4)])
def test_grids_around_a_block(gpu_lib, oracle, dims, coned):
    m = meshgen.kuhn_mesh(dims, coned, seed=5)
    _check(gpu_lib, oracle, m.tv, m.n_verts)


def test_cells_given_twice(gpu_lib, oracle):
    # every face in two cells, no boundary, each edge in the same two cells
    m = meshgen.kuhn_mesh((2, 1, 1), seed=6)
    one = m.tv[::4]
    _check(gpu_lib, oracle, np.concatenate([one, one[:, ::-1]]), m.n_verts)


@pytest.mark.parametrize("k", [13, 14, 15, 16, 21, 22, 23, 24, 30, 31, 61, 62, 63, 64])
def test_edge_rows_of_given_lengths(gpu_lib, oracle, k):
    # EE at the edges of its tiers (rows of fewer than 16, 24, at most 32, 64):
    # the axis vertices of the rings have k + 1 edges, some edges only in the
    # last warp of a block, the totals not multiples of four
    rng = np.random.default_rng(100 + k)
    ring = np.array([[0, 1, 2 + i, 2 + (i + 1) % k] for i in range(k)])
    tv = np.concatenate([ring + j * (k + 2) for j in range(5)])
    n = 5 * (k + 2)
    _check(gpu_lib, oracle, rng.permutation(n)[tv].astype(np.int32), n)


@pytest.mark.parametrize("names", [["EV", "TE"], ["EV", "ET"], ["EV", "EF"], ["EV", "TE", "FV"],
                                   ["EV", "EF", "EE"], ["EF", "VV"]])
def test_ev_beside_rows(gpu_lib, oracle, names):
    # EV by the pass that writes rows, or before it where EE reads it; EF
    # without TF; a last warp of one edge to thirty-one
    for dims, coned, hub in (((1, 1, 1), 0.0, 0), ((3, 2, 1), 0.0, 0), ((5, 4, 3), 0.5, 70)):
        m = meshgen.kuhn_mesh(dims, coned, seed=7)
        n = m.n_verts
        fan = [[n, n + 1 + i, n + 2 + i, n + hub + 2] for i in range(hub)]
        tv = np.concatenate([m.tv, np.array(fan, np.int32).reshape(-1, 4)]).astype(np.int32)
        n += hub + 3 if hub else 0
        ref = oracle.extract(oracle.canonicalize(tv, n), n)
        with gpu_lib.Mesh(tv, n) as g:
            g.extract(names)
            assert_relations_equal({r: g.relation(r) for r in names}, ref, names)
