"""MPI_Neighbor_alltoallw over self-edges, beyond the exchanges whose table
travels with the launch: more edges than that, or more than two strided
dimensions.  The table is copied to the device when it changes, and only
then."""
import numpy as np
import pytest

from tempi_b200 import _lib, mpi

from . import helpers as H
from .test_canon import desc_pack
from .test_exchange_gpu import desc_unpack

pytestmark = pytest.mark.gpu


def hvectors(block, dims):
    """A committed type of `block` bytes in nested hvectors of (count, gap)."""
    t, inner = mpi.Type_contiguous(block, mpi.BYTE), block
    for n, gap in dims:
        t = mpi.Type_create_hvector(n, 1, inner + gap, t)
        inner = n * (inner + gap)
    t = mpi.Type_create_resized(t, 0, inner)
    assert mpi.Type_commit(t) == 0
    return t, inner


class Exchange:
    """`edges` objects of one type, edge k from slot k to slot edges - 1 - k,
    `shift` bytes into the slots of the source."""

    def __init__(self, t, extent, edges, counts=None, room=1):
        import torch

        self.t, self.edges, self.d = t, edges, mpi.describe(t)[1]
        self.counts = counts or [1] * edges
        self.slot = extent * room + 64
        self.src_np = H.splitmix_bytes(self.slot * edges, edges)
        self.src = torch.from_numpy(self.src_np).cuda()
        self.dst = torch.empty_like(self.src)
        err, self.comm = mpi.Dist_graph_create_adjacent([0] * edges, [0] * edges)
        assert err == 0

    def run(self, shift=0):
        import torch

        n, slot, types = self.edges, self.slot, [self.t] * self.edges
        sd = [k * slot + shift for k in range(n)]
        rd = [(n - 1 - k) * slot for k in range(n)]
        self.dst.fill_(0xAA)
        torch.cuda.synchronize()
        before = _lib.counter("neighbor_fused")
        assert mpi.Neighbor_alltoallw(self.src.data_ptr(), self.counts, sd, types,
                                      self.dst.data_ptr(), self.counts, rd, types,
                                      self.comm) == 0, _lib.last_error()
        assert _lib.counter("neighbor_fused") == before + 1
        want = np.full(slot * n, 0xAA, np.uint8)
        for k in range(n):
            if self.counts[k]:
                desc_unpack(self.d, desc_pack(self.d, self.src_np[sd[k]:], self.counts[k]),
                            want[rd[k]:], self.counts[k])
        assert self.dst.cpu().numpy().tobytes() == want.tobytes()


@pytest.mark.parametrize("edges,dims", [
    (33, [(6, 16)]), (100, [(3, 8), (2, 40)]), (12, [(3, 8), (2, 8), (2, 8)]),
])
def test_unchanged_tables_are_copied_once(cuda, mpi_init, edges, dims):
    t, extent = hvectors(24, dims)
    x, other = Exchange(t, extent, edges), Exchange(t, extent, edges)
    n = _lib.counter("neighbor_uploads")
    assert n >= 0
    for _ in range(3):
        x.run()
    assert _lib.counter("neighbor_uploads") == n + 1
    x.run(8)  # other displacements
    x.run(8)
    assert _lib.counter("neighbor_uploads") == n + 2
    other.run()  # other buffers
    x.run()
    assert _lib.counter("neighbor_uploads") == n + 4
    mpi.Comm_free(x.comm)
    mpi.Comm_free(other.comm)


def test_growing_exchanges_share_an_allocation(cuda, mpi_init):
    """From 33 edges to 64, one more at a time: at most one allocation (none if
    an earlier exchange of the process had as many)."""
    t, extent = hvectors(8, [(3, 8)])
    n = _lib.counter("neighbor_tables")
    assert n >= 0
    for edges in range(33, 65):
        x = Exchange(t, extent, edges)
        x.run()
        mpi.Comm_free(x.comm)
    assert _lib.counter("neighbor_tables") <= n + 1


def test_single_objects_whatever_else_was_tuned(cuda, mpi_init, tmp_path, monkeypatch):
    """Exchanges of up to 32 single objects take their entries from what the
    types' commit settled, also after an unrelated batch was tuned; after a
    batch of the same signature was tuned they take its choices."""
    import torch

    from tempi_b200 import halo

    monkeypatch.setenv("TEMPI_CACHE_DIR", str(tmp_path))
    _lib.tempi().tempi_reload_env()
    other = halo.Grid((18, 11, 9), 1)
    data = torch.from_numpy(H.splitmix_bytes(other.nbytes, 1)).cuda()
    b = halo.HaloExchange([other], [data.data_ptr()])
    b.tune(None, 1)
    b.close()
    t, extent = hvectors(24, [(3, 8), (2, 40)])
    for edges in (1, 26, 32):
        x = Exchange(t, extent, edges)
        n = _lib.counter("neighbor_unit")
        assert n >= 0
        x.run()
        x.run(8)
        assert _lib.counter("neighbor_unit") == n + 2
        mpi.Comm_free(x.comm)
    # the signature of an exchange itself
    g = halo.Grid((24, 16, 12), 2)
    start = H.splitmix_bytes(g.nbytes, 2)
    a, c = torch.from_numpy(start).cuda(), torch.from_numpy(start).cuda()
    b = halo.HaloExchange([g], [a.data_ptr()])
    b.tune(None, 2)
    threads = b.config()[0]
    b.launch()
    n = _lib.counter("neighbor_unit")
    torch.cuda.synchronize()
    halo.exchange_alltoallw(halo.SelfGraph(g), c.data_ptr())
    torch.cuda.synchronize()
    assert _lib.counter("neighbor_unit") == n + (1 if threads == 256 else 0)
    assert torch.equal(a, c)
    b.close()
    monkeypatch.undo()
    _lib.tempi().tempi_reload_env()


@pytest.mark.parametrize("counts,single", [
    ([1] * 25 + [0], True), ([0] * 5, True), ([0, 1] * 32, True), ([0] + [1] * 33, False),
    ([1, 0, 2], False),
])
def test_edges_without_objects(cuda, mpi_init, counts, single):
    """Neighbours that get nothing do not lengthen the others' way: only the
    edges that exchange something count against the 32."""
    t, extent = hvectors(24, [(3, 8), (2, 40)])
    x = Exchange(t, extent, len(counts), counts, room=max(counts + [1]))
    n = _lib.counter("neighbor_unit")
    x.run()
    x.run(8)
    assert _lib.counter("neighbor_unit") == n + (2 if single else 0)
    mpi.Comm_free(x.comm)
