"""Classification rows of every length up to 64 in one mesh, several heavy stars
(64 cells and more, at most 64 neighbours) among them, with ties, infinities,
NaN and zeros of both signs in the field, against the oracle."""
import numpy as np
import pytest

from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _bipyramid(k):
    # k cells around the edge (0, 1): rows of k + 1 and of 4 entries (2 at the ring: 0, 1 and two neighbours)
    return np.array([[0, 1, 2 + i, 2 + (i + 1) % k] for i in range(k)]), k + 2


def _ball(k):
    # a vertex joined to the triangles between two poles and a ring of k: 2k cells, k + 2 neighbours
    c, a, b = 0, 1, 2
    return np.array([[c, p, 3 + i, 3 + (i + 1) % k] for i in range(k) for p in (a, b)]), k + 3


def _mesh(seed):
    grid = meshgen.kuhn_mesh((9, 8, 7), 0.2, seed=seed)
    parts = [(grid.tv, grid.n_verts)] + [_bipyramid(k) for k in range(3, 64, 5)]
    parts += [_ball(k) for k in list(range(3, 32, 4)) + list(range(33, 62, 2)) * 3]
    tvs, n = [], 0
    for tv, m in parts:
        tvs.append(tv + n)
        n += m
    rng = np.random.default_rng(seed)
    return rng.permutation(n)[np.concatenate(tvs)].astype(np.int32), n


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("values", ["distinct", "ties", "special"])
def test_rows(gpu_lib, oracle, values, dtype):
    tv, n = _mesh(3)
    rng = np.random.default_rng(4)
    f = rng.standard_normal(n).astype(dtype)
    if values == "ties":
        f = np.round(f)
    elif values == "special":
        f = rng.choice(np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, -1.0, np.finfo(dtype).tiny,
                                 -np.finfo(dtype).tiny, np.finfo(dtype).max], dtype), n)
    want = oracle.critical_points(oracle.canonicalize(tv, n), n, f)
    with gpu_lib.Mesh(tv, n) as g:
        assert np.array_equal(g.critical_points(f), want)
        off, _ = g.relation("VV")
        cells, _ = g.relation("VT")
        long, star = np.diff(off), np.diff(cells)
        assert long.max() == 64 and ((star > 64) & (long <= 64)).sum() > 32
