"""Counting and filling VT where its tiles end: cell counts around a warp's 32
and a block's 256, warps whose cells share all, some and none of their vertices
(1 to 128 of them), vertex ids that hash alike, and rejected cells among them.
Against the CPU oracle; whole numbers: equality."""
import numpy as np
import pytest

from helpers import assert_relations_equal

pytestmark = pytest.mark.gpu


def _check(tg, oracle, tv, n):
    ref = oracle.extract(oracle.canonicalize(tv, n), n, mask=1 << 9)
    with tg.Mesh(tv, n) as g:
        g.extract(["VT"])
        assert_relations_equal({"VT": g.relation("VT")}, ref)


@pytest.mark.parametrize("cells", [1, 31, 32, 33, 255, 256, 257, 1000])
@pytest.mark.parametrize("verts", [4, 5, 40, 5000])
def test_counts(gpu_lib, oracle, cells, verts):
    rng = np.random.default_rng(cells * verts)
    tv = np.array([rng.choice(verts, 4, replace=False) for _ in range(cells)], dtype=np.int32)
    _check(gpu_lib, oracle, tv, verts)


@pytest.mark.parametrize("verts", [4, 20, 128, 2000])
def test_ids_that_hash_alike(gpu_lib, oracle, verts):
    ids = np.arange(1 << 20, dtype=np.uint32)
    same = ids[(ids * np.uint32(0x9E3779B1)) >> 23 == 0][:verts]   # one slot of 512 for all of them
    rng = np.random.default_rng(verts)
    tv = np.array([rng.choice(same, 4, replace=False) for _ in range(300)], dtype=np.int32)
    tv[:32] = rng.permutation(same)[:128].reshape(-1, 4) if verts >= 128 else tv[:32]
    _check(gpu_lib, oracle, tv, 1 << 20)


@pytest.mark.parametrize("at", [0, 31, 32, 299])
def test_a_rejected_cell(gpu_lib, at):
    tv = np.arange(1200, dtype=np.int32).reshape(300, 4)
    tv[at, 2] = 1200
    with pytest.raises(gpu_lib.TetraGPUError) as ei:
        gpu_lib.Mesh(tv, 1200)
    assert f"cell {at} " in str(ei.value)
