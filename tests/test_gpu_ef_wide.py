"""EF past 2^31 entries: cells that share nothing (EF of an edge: its cell's two
faces at it, in closed form) and after them a ring around an edge whose ends
lie in more than 64 cells (the rows of heavy stars), compared with the oracle's
EF of the ring alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CELLS = 178_960_000     # 12 a cell: 2^31 + 36,352 entries
RING = 70


class _Array:
    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 2}


def test_rows_past_two_to_the_31(gpu_lib, oracle):
    import torch
    if torch.cuda.mem_get_info()[0] < 140 * 10**9:
        pytest.skip("needs 140 GB of device memory")
    ring = np.array([[0, 1, 2 + i, 2 + (i + 1) % RING] for i in range(RING)], np.int32)
    n_ring = RING + 2
    want_off, want_ent = oracle.extract(oracle.canonicalize(ring, n_ring), n_ring)["EF"]
    n = 4 * CELLS + n_ring
    tv = torch.empty((CELLS + RING, 4), dtype=torch.int32, device="cuda")
    tv[:CELLS] = torch.arange(4 * CELLS, dtype=torch.int32, device="cuda").view(-1, 4)
    tv[CELLS:] = torch.from_numpy(ring + 4 * CELLS).cuda()
    torch.cuda.synchronize()
    with gpu_lib.Mesh(tv.data_ptr(), n, CELLS + RING, on_device=True) as g:
        del tv
        g.extract(["EF"])
        d = g.device_relation("EF")
        assert d["rows"] == 6 * CELLS + want_off.size - 1 and d["n_entries"] == 12 * CELLS + want_ent.size
        off = torch.as_tensor(_Array(d["offsets"], d["rows"] + 1, "<i8"), device="cuda")
        ent = torch.as_tensor(_Array(d["entries"], d["n_entries"], "<i4"), device="cuda")
        torch.cuda.synchronize()
        assert np.array_equal(off[6 * CELLS:].cpu().numpy(), want_off + 12 * CELLS)
        assert np.array_equal(ent[12 * CELLS:].cpu().numpy(), want_ent + 4 * CELLS)
        # face column k leaves out slot 3 - k; edge (s, t) lies in the columns of the other two slots
        pairs = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]
        cell = torch.tensor([[3 - x for x in (3, 2, 1, 0) if x not in p] for p in pairs], device="cuda").view(-1)
        step = 1 << 22
        for c0 in range(0, CELLS, step):
            c = torch.arange(c0, min(c0 + step, CELLS), device="cuda")
            assert torch.equal(ent[12 * c0:12 * (c0 + c.numel())], (4 * c[:, None] + cell).view(-1).int())
            e = torch.arange(6 * c0, 6 * (c0 + c.numel()), device="cuda")
            assert torch.equal(off[6 * c0:6 * (c0 + c.numel())], 2 * e)
