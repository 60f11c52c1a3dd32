"""Stars of one and two cells, alone and among larger ones: cells that share
nothing, a vertex, an edge, a face or everything, in numbers around a warp's
vertices, chains, and a grid between them.  Every relation and the classes
against the CPU oracle; whole numbers: equality."""
import numpy as np
import pytest

from helpers import RELS, assert_relations_equal
from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _pairs(n, shared, base):
    """n pairs of cells with `shared` vertices in common."""
    k = 8 - shared
    i = base + k * np.arange(n)[:, None]
    a = i + np.arange(4)
    b = np.concatenate([a[:, :shared], i + np.arange(4, k)], 1)
    return np.stack([a, b], 1).reshape(-1, 4), base + k * n


def _check(tg, oracle, tv, n, seed):
    rng = np.random.default_rng(seed)
    tv = rng.permuted(rng.permutation(n)[tv], axis=1).astype(np.int32)
    tvs = oracle.canonicalize(tv, n)
    ref = oracle.extract(tvs, n)
    f = rng.standard_normal(n).astype(np.float32)
    with tg.Mesh(tv, n) as g:
        g.extract(tg.ALL_RELATIONS, options=tg.OPT_LINK_ADJACENCY)
        assert g.counts() == ref["counts"]
        assert_relations_equal({r: g.relation(r) for r in RELS}, ref)
        assert np.array_equal(g.critical_points(f), oracle.critical_points(tvs, n, f))
    with tg.Mesh(tv, n) as g:           # without the faces' second cells
        g.extract(["EF", "VV"])
        assert_relations_equal({r: g.relation(r) for r in ("EF", "VV")}, ref, ["EF", "VV"])


@pytest.mark.parametrize("shared", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 2, 5, 64, 5000])
def test_pairs(gpu_lib, oracle, shared, n):
    tv, verts = _pairs(n, shared, 0)
    _check(gpu_lib, oracle, tv, verts, n + shared)


@pytest.mark.parametrize("n", [2, 7, 300])
def test_chain(gpu_lib, oracle, n):
    tv = np.arange(n)[:, None] * np.array([[1]]) + np.arange(4)    # cell i: i .. i + 3
    _check(gpu_lib, oracle, tv, n + 3, n)


def test_among_others(gpu_lib, oracle):
    grid = meshgen.kuhn_mesh((12, 11, 10), 0.3, seed=2)
    tvs, n = [grid.tv], grid.n_verts
    for shared in range(5):
        tv, n = _pairs(700, shared, n)
        tvs.append(tv)
    for k in (5, 40, 70):       # rings: two cells at each vertex but the axis'
        i = np.arange(k)
        tvs.append(np.stack([0 * i + n, 0 * i + n + 1, n + 2 + i, n + 2 + (i + 1) % k], 1))
        n += k + 2
    tv = np.concatenate(tvs)
    _check(gpu_lib, oracle, tv, n, 1)
    _check(gpu_lib, oracle, tv[np.random.default_rng(3).permutation(len(tv))], n, 2)


def test_with_heavy_vertices(gpu_lib, oracle):
    """Short rows on average, but vertices of more than 64 neighbours too (and of
    33 to 64), some of them in the same windows of the link masks."""
    tvs, n = [], 0
    for k in (80, 70, 40, 25, 66):     # fans around a vertex, rings around an edge
        tvs.append(n + np.stack([0 * np.arange(k), *(3 * np.arange(k) + j for j in (1, 2, 3))], 1))
        n += 3 * k + 1
        i = np.arange(k)
        tvs.append(np.stack([0 * i + n, 0 * i + n + 1, n + 2 + i, n + 2 + (i + 1) % k], 1))
        n += k + 2
    tv, n = _pairs(3000, 0, n)
    tvs.append(tv)
    _check(gpu_lib, oracle, np.concatenate(tvs), n, 3)


def test_in_a_batch(gpu_lib, oracle):
    rng = np.random.default_rng(4)
    meshes = [_pairs(40 * i, shared, 0) for i, shared in ((1, 0), (30, 2), (3, 1), (50, 0))]
    meshes = [(rng.permutation(n)[tv].astype(np.int32), n) for tv, n in meshes]
    fields = [[rng.standard_normal(n).astype(d) for d in (np.float32, np.float64)] for _, n in meshes]
    with gpu_lib.Server(n_slots=1) as srv:
        sent = [srv.submit_mesh(tv, n, f[0]) for (tv, n), f in zip(meshes, fields)]
        got = [[srv.wait(rid)[0], srv.wait(srv.submit_field(mid, f[1]))[0]] for (rid, mid), f in zip(sent, fields)]
    for (tv, n), f, g in zip(meshes, fields, got):
        tvs = oracle.canonicalize(tv, n)
        for k in range(2):
            assert np.array_equal(g[k], oracle.critical_points(tvs, n, f[k]))
