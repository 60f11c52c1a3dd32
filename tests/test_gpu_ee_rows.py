"""EE rows whose ends have every number of edges from 3 to 75, so that a warp's
edges fall on both sides of each limit (16, 24, 32, 64 edges of an end), in
several orders of ids and cells.  Against the CPU oracle; whole numbers:
equality."""
import numpy as np
import pytest

from helpers import assert_relations_equal
from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _ball(k):
    # a vertex joined to the triangles between two poles and a ring of k
    return np.array([[0, p, 3 + i, 3 + (i + 1) % k] for i in range(k) for p in (1, 2)]), k + 3


@pytest.mark.parametrize("longest", [13, 14, 21, 22, 29, 30, 31, 61, 62, 63, 70])
@pytest.mark.parametrize("order", ["sorted", "permuted"])
def test_rows(gpu_lib, oracle, longest, order):
    grid = meshgen.kuhn_mesh((5, 4, 3), 0.0, seed=1)
    tvs, n = [grid.tv], grid.n_verts
    for k in list(range(3, longest + 1)) + [longest] * 3:
        tv, m = _ball(k)
        tvs.append(tv + n)
        n += m
    tv = np.concatenate(tvs)
    rng = np.random.default_rng(longest)
    if order == "permuted":
        tv = rng.permutation(n)[tv][rng.permutation(len(tv))]
    tv = tv.astype(np.int32)
    ref = oracle.extract(oracle.canonicalize(tv, n), n)
    with gpu_lib.Mesh(tv, n) as g:
        g.extract(["EE"])
        off, _ = g.relation("VV")
        assert np.diff(off).max() == longest + 2
        assert_relations_equal({"EE": g.relation("EE")}, ref, ["EE"])
