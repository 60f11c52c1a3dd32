"""Classification and smoothing of meshes above 2^17 vertices whose ids keep
neighbours together or do not, with cells in order or scattered: the link graph
is in the order of ids or of the star pass, with a vertex of more than 64
neighbours and one of more than 32 (64-bit masks) among the rest or without."""
import numpy as np
import pytest

from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _natural(dims, coned, seed):
    """The generator's mesh with ids along the grid's lines again."""
    m = meshgen.kuhn_mesh(dims, coned, seed=seed)
    by = np.lexsort((m.coords[:, 0], m.coords[:, 1], m.coords[:, 2]))
    back = np.empty(m.n_verts, np.int64)
    back[by] = np.arange(m.n_verts)
    return back[m.tv], m.n_verts


def _mesh(ids, cells, extra):
    tv, n = _natural((54, 51, 47), 0.1, 1)
    if extra:
        fan = np.array([[0, 3 * i + 1, 3 * i + 2, 3 * i + 3] for i in range(80)])
        ring = np.array([[0, 1, 2 + i, 2 + (i + 1) % 40] for i in range(40)])
        tv, n = np.concatenate([tv, fan + n, ring + n + 241]), n + 241 + 42
    rng = np.random.default_rng(2)
    if ids == "permuted":
        tv = rng.permutation(n)[tv]
    if cells == "scattered":
        tv = tv[rng.permutation(len(tv))]
    return tv.astype(np.int32), n


@pytest.mark.parametrize("extra", [False, True])
@pytest.mark.parametrize("cells", ["in order", "scattered"])
@pytest.mark.parametrize("ids", ["in order", "permuted"])
def test_classes_and_smoothing(gpu_lib, oracle, ids, cells, extra):
    import torch
    tv, n = _mesh(ids, cells, extra)
    tvs = oracle.canonicalize(tv, n)
    f = np.round(np.random.default_rng(3).standard_normal(n), 1)     # with ties
    x = torch.from_numpy(f.astype(np.float32)).cuda()
    out, tmp = torch.empty_like(x), torch.empty_like(x)
    steps = 6
    for smooth_first in (False, True):
        with gpu_lib.Mesh(tv, n) as g:
            if smooth_first:
                g.smooth_field(x.data_ptr(), out.data_ptr(), steps, tmp.data_ptr())
            for dtype in (np.float32, np.float64):
                assert np.array_equal(g.critical_points(f.astype(dtype)),
                                      oracle.critical_points(tvs, n, f.astype(dtype)))
            g.smooth_field(x.data_ptr(), out.data_ptr(), steps, tmp.data_ptr())
            off, ent = g.relation("VV")
    d = np.diff(off)
    want = f.astype(np.float32).astype(np.float64)
    bound = steps * (int(d.max()) + 2) * 2.0**-24 * np.abs(want).max()
    rows = np.repeat(np.arange(n), d)
    for _ in range(steps):
        want = (want + np.bincount(rows, want[ent], n)) / (d + 1)
    assert np.abs(out.cpu().numpy() - want).max() <= bound


def test_members_of_a_batch(gpu_lib):
    """New fields on the meshes of a batch whose union has ids in order."""
    meshes = [_natural((40, 38, 36 + i), 0.0, i) for i in range(4)]
    rng = np.random.default_rng(6)
    fields = [[rng.standard_normal(n).astype(np.float32) for _ in range(2)] for _, n in meshes]
    with gpu_lib.Server(n_slots=1) as srv:
        sent = [srv.submit_mesh(tv.astype(np.int32), n, f[0]) for (tv, n), f in zip(meshes, fields)]
        got = [srv.wait(rid)[0] for rid, _ in sent]
        again = [srv.wait(srv.submit_field(mid, f[1]))[0] for (_, mid), f in zip(sent, fields)]
    for (tv, n), f, a, b in zip(meshes, fields, got, again):
        with gpu_lib.Mesh(tv.astype(np.int32), n) as g:
            assert np.array_equal(a, g.critical_points(f[0])) and np.array_equal(b, g.critical_points(f[1]))
