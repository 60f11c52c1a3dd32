"""Critical points at the sizes where the link graph's rows and hash tables
change: rows of 7 to 65 neighbours (padding to eights, 32-bit and 64-bit masks,
several rows per window and one that fills it), vertices without cells, fields
large enough to be put in processing order, and a member of a batch.  Classes
against the CPU oracle, or against the mesh alone; whole numbers: equality."""
import numpy as np
import pytest

from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _check(tg, oracle, tv, n, seed):
    rng = np.random.default_rng(seed)
    tvs = oracle.canonicalize(tv, n)
    for field in (rng.standard_normal(n).astype(np.float32),
                  rng.integers(0, 3, n).astype(np.float64)):      # ties by id
        want = oracle.critical_points(tvs, n, field)
        with tg.Mesh(tv, n) as g:
            assert np.array_equal(g.critical_points(field), want)
            assert np.array_equal(g.critical_points(field), want)


@pytest.mark.parametrize("k", [7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 40, 62, 63, 64])
def test_rings(gpu_lib, oracle, k):
    # both axis vertices have k + 1 neighbours; vertices without cells between
    rng = np.random.default_rng(k)
    ring = np.array([[0, 1, 2 + i, 2 + (i + 1) % k] for i in range(k)])
    tv = np.concatenate([ring, ring + k + 5, ring + 2 * (k + 5)])
    n = 3 * (k + 5)
    _check(gpu_lib, oracle, rng.permutation(n)[tv].astype(np.int32), n, k)


@pytest.mark.parametrize("n_verts,n_cells", [(12, 6), (40, 60), (64, 200), (66, 300)])
def test_dense_neighbourhoods(gpu_lib, oracle, n_verts, n_cells):
    # cells over few vertices: nearly everything is adjacent; cells that would
    # put a face in a third cell are left out
    rng = np.random.default_rng(n_cells)
    seen, cells = {}, []
    while len(cells) < n_cells and len(seen) < 3 * n_cells:
        c = tuple(sorted(rng.choice(n_verts, 4, replace=False)))
        faces = [c[:k] + c[k + 1:] for k in range(4)]
        if all(seen.get(f, 0) < 2 for f in faces):
            cells.append(c)
            for f in faces:
                seen[f] = seen.get(f, 0) + 1
    _check(gpu_lib, oracle, np.array(cells, dtype=np.int32), n_verts, n_cells)


def test_field_put_in_order(gpu_lib, oracle):
    m = meshgen.kuhn_mesh((60, 50, 46), 0.02, seed=3)
    assert m.n_verts > 1 << 17
    field = meshgen.sine_field(m.coords, seed=4)
    tvs = oracle.canonicalize(m.tv, m.n_verts)
    want = oracle.critical_points(tvs, m.n_verts, field)
    with gpu_lib.Mesh(m.tv, m.n_verts) as g:
        assert np.array_equal(g.critical_points(field), want)
        assert np.array_equal(g.critical_points(field.astype(np.float64)), want)
    # a large and a small member of a server's batch, fields one by one
    small = meshgen.kuhn_mesh(5, 0.3, seed=5)
    f2 = meshgen.sine_field(small.coords, seed=6)
    with gpu_lib.Server() as s:
        sent = [s.submit_mesh(x.tv, x.n_verts, f) for x, f in ((small, f2), (m, field), (small, f2))]
        for rid, _ in sent:
            s.wait(rid)
        assert np.array_equal(s.wait(s.submit_field(sent[1][1], field))[0], want)
        got = s.wait(s.submit_field(sent[2][1], f2))[0]
    with gpu_lib.Mesh(small.tv, small.n_verts) as g:
        assert np.array_equal(got, g.critical_points(f2))
