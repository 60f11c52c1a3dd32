"""A mesh smoothed on one stream and destroyed or extracted again from another, or
smoothed while copies of it are on their way, with nothing waited for in between: the smoothed values are those of a mesh
left alone.  The smoothing stream is kept busy first, so that its steps come
after the other stream's frees and reuse of memory would have."""
import numpy as np
import pytest

from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu

STEPS = 6


@pytest.fixture(scope="module")
def mesh():
    m = meshgen.kuhn_mesh((54, 51, 47), 0.1, seed=1)     # above 2^17 vertices
    return np.random.default_rng(1).permutation(m.n_verts)[m.tv].astype(np.int32), m.n_verts


@pytest.mark.parametrize("then", ["destroy", "extract", "destroy after a field elsewhere"])
@pytest.mark.parametrize("rows_first", [False, True])
def test_smoothed_on_another_stream(gpu_lib, mesh, then, rows_first):
    import torch
    tv, n = mesh
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    f = np.random.default_rng(3).standard_normal(n).astype(np.float32)
    x = torch.from_numpy(f).cuda()
    out, tmp, want = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    classes = torch.empty((n, 3), dtype=torch.int32, device="cuda")
    with gpu_lib.Mesh(tv, n) as g:
        g.smooth_field(x.data_ptr(), want.data_ptr(), STEPS, tmp.data_ptr())
        torch.cuda.synchronize()
    for _ in range(3):
        out.fill_(9.0)
        g = gpu_lib.Mesh(tv, n, stream=a)
        g.extract(["VV"], stream=a)
        torch.cuda.synchronize()
        if rows_first:
            g.smooth_field(x.data_ptr(), out.data_ptr(), STEPS, tmp.data_ptr(), stream=b)
            torch.cuda.synchronize()
            out.fill_(9.0)
            torch.cuda.synchronize()
        with torch.cuda.stream(b):
            torch.cuda._sleep(20_000_000)      # about 10 ms
        g.smooth_field(x.data_ptr(), out.data_ptr(), STEPS, tmp.data_ptr(), stream=b)
        if then == "extract":
            g.extract(["EE"], stream=a)
        elif then.startswith("destroy after"):
            g.critical_points(x.data_ptr(), on_device=True, out_ptr=classes.data_ptr(), stream=a)
        else:
            g.close()
        # meshes that take the memory given back
        others = [gpu_lib.Mesh(tv, n, stream=a) for _ in range(2)]
        for o in others:
            o.extract(["VV"], gpu_lib.OPT_LINK_ADJACENCY, stream=a)
        if then.startswith("destroy after"):
            g.close()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
        for o in others:
            o.close()
        g.close()


@pytest.mark.parametrize("steps", [1, STEPS])
def test_smoothed_while_copies_are_on_their_way(gpu_lib, mesh, steps):
    """Destroying the mesh waits for the copies' stream and for the smoothing."""
    import torch
    tv, n = mesh
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.from_numpy(np.random.default_rng(4).standard_normal(n).astype(np.float32)).cuda()
    out, tmp, want = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    with gpu_lib.Mesh(tv, n) as g:
        g.extract(["VV"])
        g.smooth_field(x.data_ptr(), want.data_ptr(), steps, tmp.data_ptr())
        off, ent = g.relation("VV")
        torch.cuda.synchronize()
    h_off = torch.zeros(off.size, dtype=torch.int64).pin_memory()
    h_ent = torch.zeros(ent.size, dtype=torch.int32).pin_memory()
    for first, second in ((a, b), (b, a)):
        h_off.zero_()
        h_ent.zero_()
        out.fill_(9.0)
        g = gpu_lib.Mesh(tv, n, stream=first)
        g.extract(["VV"], stream=first)
        torch.cuda.synchronize()
        for s in (a, b):
            with torch.cuda.stream(s):
                torch.cuda._sleep(20_000_000)
        gpu_lib._lib.check(g._lib.tg_copy_relation_async(g._h, gpu_lib.REL["VV"], h_off.data_ptr(),
                                                         h_ent.data_ptr(), first.cuda_stream))
        g.smooth_field(x.data_ptr(), out.data_ptr(), steps, tmp.data_ptr(), stream=second)
        g.close()
        assert np.array_equal(h_off.numpy(), off) and np.array_equal(h_ent.numpy(), ent)
        with gpu_lib.Mesh(tv, n, stream=first) as other:     # takes the memory given back
            other.extract(["VV"], gpu_lib.OPT_LINK_ADJACENCY, stream=first)
        torch.cuda.synchronize()
        assert torch.equal(out, want)
