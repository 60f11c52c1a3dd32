"""Classification recorded into a graph: with the link masks on the mesh and
without them (what it makes then belongs to the graph, not to the mesh), run
several times with other fields and with other calls in between, on meshes
below and above the size from which a field is put in processing order, one
with vertices of more than 64 neighbours."""
import numpy as np
import pytest

from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _mesh(dims, heavy, seed):
    m = meshgen.kuhn_mesh(dims, 0.1, seed=seed)
    tv, n = m.tv, m.n_verts
    if heavy:     # a fan of 80 cells that share one vertex
        fan = np.array([[0, 3 * i + 1, 3 * i + 2, 3 * i + 3] for i in range(80)], dtype=np.int32)
        tv, n = np.concatenate([tv, fan + n]), n + 241
    return np.random.default_rng(seed).permutation(n)[tv].astype(np.int32), n


@pytest.mark.parametrize("masks", [True, False])
@pytest.mark.parametrize("dims, heavy", [((9, 8, 7), False), ((9, 8, 7), True), ((54, 51, 47), False),
                                         ((54, 51, 47), True)])
def test_recorded(gpu_lib, dims, heavy, masks):
    import torch
    tv, n = _mesh(dims, heavy, 4)
    rng = np.random.default_rng(5)
    fields = [rng.standard_normal(n).astype(np.float32) for _ in range(4)]
    with gpu_lib.Mesh(tv, n) as g:
        want = [g.critical_points(f) for f in fields]
    s = torch.cuda.Stream()
    x, out = torch.empty(n, device="cuda"), torch.empty((n, 3), dtype=torch.int32, device="cuda")
    a, b = torch.empty_like(x), torch.empty_like(x)

    def recorded(f):
        x.copy_(torch.from_numpy(f))
        out.fill_(9)
        graph.replay()
        torch.cuda.synchronize()
        return out.cpu().numpy().astype(np.uint32)

    with gpu_lib.Mesh(tv, n) as g:
        g.extract(["VV"], gpu_lib.OPT_LINK_ADJACENCY if masks else 0)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            g.critical_points(x.data_ptr(), on_device=True, out_ptr=out.data_ptr(), stream=s)
        # the mesh by itself, before the graph has run at all
        g.smooth_field(x.data_ptr(), a.data_ptr(), 6, b.data_ptr())
        assert np.array_equal(g.critical_points(fields[3]), want[3])
        for k in range(3):
            assert np.array_equal(recorded(fields[k]), want[k])
            assert np.array_equal(g.critical_points(fields[k]), want[k])
        g.smooth_field(x.data_ptr(), a.data_ptr(), 6, b.data_ptr())
        assert np.array_equal(recorded(fields[0]), want[0])
        del graph
        torch.cuda.synchronize()
        assert np.array_equal(g.critical_points(fields[1]), want[1])
