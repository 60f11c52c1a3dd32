"""Smoothed values repeat bit for bit: whatever was called on the mesh before,
and for two meshes made from one TV, also with several vertices of more than 64
cells next to each other (their order must not depend on timing)."""
import numpy as np
import pytest

from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh():
    m = meshgen.kuhn_mesh((54, 51, 47), 0.1, seed=1)     # above 2^17 vertices
    parts, n = [m.tv], m.n_verts
    for _ in range(40):      # rings of 70 cells around an edge of two heavy vertices
        parts.append(np.array([[n, n + 1, n + 2 + i, n + 2 + (i + 1) % 70] for i in range(70)], np.int32))
        n += 72
    rng = np.random.default_rng(2)
    tv = rng.permutation(n)[np.concatenate(parts)].astype(np.int32)
    return tv, n, rng.standard_normal(n).astype(np.float32)


@pytest.mark.parametrize("steps", [2, 4, 5, 7])
def test_same_bits(gpu_lib, mesh, steps):
    import torch
    tv, n, f = mesh
    x = torch.from_numpy(f).cuda()
    out, tmp = torch.empty_like(x), torch.empty_like(x)
    seen = []

    def smooth(g, k):
        g.smooth_field(x.data_ptr(), out.data_ptr(), k, tmp.data_ptr())
        return out.cpu().numpy().view(np.uint32)

    for first in ("nothing", "classes", "five steps", "masks in the extraction"):
        with gpu_lib.Mesh(tv, n) as g:
            g.extract(["VV"], gpu_lib.OPT_LINK_ADJACENCY if first.startswith("masks") else 0)
            if first == "classes":
                g.critical_points(f)
            elif first == "five steps":
                smooth(g, 5)
            seen += [smooth(g, steps), smooth(g, steps)]
    assert all(np.array_equal(s, seen[0]) for s in seen)
