"""Meshes of a server released after their batch was evicted, before and after
it was built again, and while other members of the batch are still asked for."""
import numpy as np
import pytest

from tetragpu_gb300 import meshgen

pytestmark = pytest.mark.gpu


def test_release_after_eviction(gpu_lib):
    rng = np.random.default_rng(1)
    meshes = [meshgen.kuhn_mesh((3 + i % 3, 4, 2 + i % 2), 0.2, seed=i) for i in range(8)]
    with gpu_lib.Server(n_slots=2, hbm_budget_bytes=1) as srv:    # every batch goes once it is idle

        def ask(k):
            m = meshes[k]
            f = rng.standard_normal(m.n_verts).astype(np.float32)
            got, _ = srv.wait(srv.submit_field(ids[k], f))
            with gpu_lib.Mesh(m.tv, m.n_verts) as g:
                assert np.array_equal(got, g.critical_points(f))

        sent = [srv.submit_mesh(m.tv, m.n_verts, rng.standard_normal(m.n_verts).astype(np.float32)) for m in meshes]
        ids = [mid for _, mid in sent]
        for rid, _ in sent:
            srv.wait(rid)
        srv.release(ids[0])                  # its batch evicted or still there
        for k in (1, 2, 3):                  # built again alone, evicting each other
            ask(k)
        assert srv.stats()["evictions"] > 0
        srv.release(ids[1])                  # evicted after it was built again
        srv.release(ids[4])                  # evicted and never built again
        for k in (3, 2, 5, 6, 7):
            ask(k)
        for k in (0, 1, 4):
            with pytest.raises(gpu_lib.TetraGPUError):
                srv.submit_field(ids[k], np.zeros(meshes[k].n_verts, np.float32))
        for k in (2, 3, 5, 6, 7):
            srv.release(ids[k])
        st = srv.stats()
        assert st["resident_meshes"] == 0 and st["resident_bytes"] == 0 and st["failed"] == 0
