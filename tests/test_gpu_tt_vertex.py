"""TT by shared vertex where its tiles end: cell counts around a warp and a
block, warps whose rows and whose results just fit in shared memory and just
do not, a row larger than all of it, the same cell given twice.  Against the
CPU oracle; whole numbers: equality."""
import numpy as np
import pytest

from helpers import assert_relations_equal
from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _check(tg, oracle, tv, n):
    tvs = oracle.canonicalize(tv, n)
    ref = oracle.extract(tvs, n, mask=1 << 10, options=1)
    with tg.Mesh(tv, n) as g:
        g.extract(["TT"], options=tg.OPT_TT_VERTEX_SHARING)
        assert_relations_equal({"TT": g.relation("TT")}, ref)


# a hub of k cells that share nothing else.  A warp's rows take k + 1 words and
# two for each of 96 vertices of one cell (1536 at k = 1343); its results 32
# (k - 1) entries (2556 between k = 80 and 81)
@pytest.mark.parametrize("k", [1, 31, 32, 33, 63, 64, 65, 80, 81, 1342, 1343, 1344, 1600])
def test_hub(gpu_lib, oracle, k):
    tv = np.array([[0, 1 + 3 * i, 2 + 3 * i, 3 + 3 * i] for i in range(k)], dtype=np.int32)
    rng = np.random.default_rng(k)
    n = 3 * k + 1
    _check(gpu_lib, oracle, rng.permutation(n)[tv].astype(np.int32), n)


@pytest.mark.parametrize("dims,coned", [((1, 1, 1), 0.0), ((3, 2, 1), 0.5), ((7, 6, 5), 0.3)])
def test_grid_and_cells_given_twice(gpu_lib, oracle, dims, coned):
    m = meshgen.kuhn_mesh(dims, coned, seed=3)
    _check(gpu_lib, oracle, m.tv, m.n_verts)
    _check(gpu_lib, oracle, np.concatenate([m.tv, m.tv[::3]]).astype(np.int32), m.n_verts)
