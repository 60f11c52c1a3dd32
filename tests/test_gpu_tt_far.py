"""TT by shared vertex of meshes large enough for a list of the warps whose rows
do not fit in shared memory: none of them, some, all of them, rows that fit but
whose results do not, the cell counts where the list begins.  Against the CPU
oracle; whole numbers: equality."""
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


@pytest.mark.parametrize("cells", ["in order", "scattered", "half scattered"])
def test_order_of_cells(gpu_lib, oracle, cells):
    m = meshgen.kuhn_mesh((24, 23, 22), 0.2, seed=2)
    rng = np.random.default_rng(3)
    order = np.arange(len(m.tv))
    if cells != "in order":
        part = len(order) if cells == "scattered" else len(order) // 2 + 7
        order[:part] = rng.permutation(part)
    _check(gpu_lib, oracle, m.tv[order], m.n_verts)


@pytest.mark.parametrize("n_cells", [(1 << 16) - 1, 1 << 16, (1 << 16) + 1, (1 << 16) + 33])
def test_where_the_list_begins(gpu_lib, oracle, n_cells):
    m = meshgen.kuhn_mesh((24, 23, 22), 0.0, seed=4)
    _check(gpu_lib, oracle, m.tv[np.random.default_rng(5).permutation(len(m.tv))[:n_cells]], m.n_verts)


def test_results_that_are_not_collected(gpu_lib, oracle):
    """Hubs of 90 cells that share nothing else: 32 x 89 results to a warp,
    1,500 words of rows; one hub of 3,000."""
    tvs, n = [], 0
    for k in [90] * 800 + [3000]:
        tvs.append(np.array([[0, 1 + 3 * i, 2 + 3 * i, 3 + 3 * i] for i in range(k)]) + n)
        n += 3 * k + 1
    tv = np.concatenate(tvs)
    assert len(tv) >= 1 << 16
    _check(gpu_lib, oracle, np.random.default_rng(6).permutation(n)[tv].astype(np.int32), n)
