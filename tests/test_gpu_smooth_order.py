"""Smoothing over VV by position against the sums in float64: vertex counts
below and above where it begins, step counts around those that make its rows,
rows that are there already, a second stream, a recorded graph, a vertex with
many neighbours.  Bound: n + 2 roundings of values up to max |f| a step."""
import numpy as np
import pytest

from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _grid(dims, coned, seed):
    m = meshgen.kuhn_mesh(dims, coned, seed=seed)
    rng = np.random.default_rng(seed)
    return rng.permutation(m.n_verts)[m.tv].astype(np.int32), m.n_verts


def _want(off, ent, f, steps):
    x = f.astype(np.float64)
    n = np.diff(off)
    rows = np.repeat(np.arange(n.size), n)
    for _ in range(steps):
        x = (x + np.bincount(rows, x[ent], n.size)) / (n + 1)
    return x


def _bound(off, f, steps):
    return steps * (int(np.diff(off).max()) + 2) * 2.0**-24 * np.abs(f).max()


@pytest.fixture(scope="module")
def meshes():
    big, nb = _grid((54, 51, 47), 0.1, 1)          # above 2^17 vertices
    small, ns = _grid((48, 51, 50), 0.0, 2)        # just below
    hub = np.array([[nb, 4 * i, 4 * i + 1, 4 * i + 2] for i in range(60)], dtype=np.int32)
    return {"big": (big, nb), "small": (small, ns), "hub": (np.concatenate([big, hub]), nb + 1)}


@pytest.mark.parametrize("which", ["big", "small", "hub"])
@pytest.mark.parametrize("rows_first", [False, True])
@pytest.mark.parametrize("steps", [1, 2, 4, 5, 6])
def test_steps(gpu_lib, meshes, which, rows_first, steps):
    import torch
    tv, n = meshes[which]
    f = np.random.default_rng(steps).standard_normal(n).astype(np.float32)
    with gpu_lib.Mesh(tv, n) as g:
        g.extract(["VV"])
        off, ent = g.relation("VV")
        if rows_first:
            classes = g.critical_points(f)
        x = torch.from_numpy(f).cuda()
        out, tmp = torch.full_like(x, 9.0), torch.full_like(x, 9.0)
        for _ in range(2):
            g.smooth_field(x.data_ptr(), out.data_ptr(), steps, tmp.data_ptr())
            got = out.cpu().numpy()
            assert np.abs(got - _want(off, ent, f, steps)).max() <= _bound(off, f, steps)
        if rows_first:   # the masks' rows are as they were
            assert np.array_equal(g.critical_points(f), classes)


def test_another_stream_and_a_recorded_graph(gpu_lib, meshes):
    import torch
    tv, n = meshes["big"]
    f = np.random.default_rng(9).standard_normal(n).astype(np.float32)
    x = torch.from_numpy(f).cuda()
    with gpu_lib.Mesh(tv, n) as g:
        g.extract(["VV"])
        off, ent = g.relation("VV")
        want, bound = _want(off, ent, f, 6), _bound(off, f, 6)
        streams = [torch.cuda.Stream() for _ in range(3)]
        outs = [torch.empty_like(x) for _ in streams]
        tmps = [torch.empty_like(x) for _ in streams]
        torch.cuda.synchronize()
        for s, o, t in zip(streams, outs, tmps):   # the first makes the rows
            g.smooth_field(x.data_ptr(), o.data_ptr(), 6, t.data_ptr(), stream=s.cuda_stream)
        torch.cuda.synchronize()
        for o in outs:
            assert np.abs(o.cpu().numpy() - want).max() <= bound
    with gpu_lib.Mesh(tv, n) as g:
        g.extract(["VV"])
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=streams[0]):
            g.smooth_field(x.data_ptr(), outs[0].data_ptr(), 6, tmps[0].data_ptr(),
                           stream=streams[0].cuda_stream)
        outs[0].fill_(9.0)
        graph.replay()
        torch.cuda.synchronize()
        assert np.abs(outs[0].cpu().numpy() - want).max() <= bound
