"""Batch launches start before the kernel ahead of them has ended and read their
table then; what they may not overlap is work of other kinds ahead of them (a
copy, a memset, another stream's event), nor each other's buffers, and a table
made while earlier launches run has to be whole.  Each case keeps the work
ahead running while the launches are issued."""
import numpy as np
import pytest

from tempi_b200 import halo

from . import helpers as H
from .test_batch_gpu import oracle_pack, oracle_unpack

pytestmark = pytest.mark.gpu

BUSY = 20_000_000  # cycles: 10 ms


def grid(shape=(60, 37, 29), radius=2, seed=1):
    import torch

    g = halo.Grid(shape, radius)
    start = H.splitmix_bytes(g.nbytes, seed)
    return g, start, torch.from_numpy(start).cuda()


def packer(g, data):
    import torch

    packed = torch.zeros(g.packed_bytes, dtype=torch.uint8, device="cuda")
    return packed, halo.HaloBatch([g], [data.data_ptr()], [packed.data_ptr()])


@pytest.mark.parametrize("ahead", ["copy", "memset", "event", "kernel"])
def test_behind_other_work(cuda, mpi_init, ahead):
    import torch

    g, start, data = grid()
    packed, b = packer(g, data)
    fresh = H.splitmix_bytes(g.nbytes, 99)
    if ahead == "memset":
        fresh = np.full(g.nbytes, 7, np.uint8)
    pinned, on_gpu = torch.from_numpy(fresh).pin_memory(), torch.from_numpy(fresh).cuda()
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(5):
        first = torch.empty_like(packed)
        with torch.cuda.stream(s):
            data.copy_(torch.from_numpy(start).pin_memory(), non_blocking=True)
            b.launch(s.cuda_stream)
            first.copy_(packed)
            b.launch(s.cuda_stream)  # a batch launch directly before the other work
            if ahead == "copy":
                data.copy_(pinned, non_blocking=True)
            elif ahead == "memset":
                data.fill_(7)
            elif ahead == "kernel":
                torch.cuda._sleep(BUSY)
                data.copy_(on_gpu)
            else:
                other.wait_stream(s)
                with torch.cuda.stream(other):
                    torch.cuda._sleep(BUSY)
                    data.copy_(on_gpu)
                s.wait_stream(other)
            b.launch(s.cuda_stream)
        torch.cuda.synchronize()
        assert first.cpu().numpy().tobytes() == oracle_pack(g, start).tobytes()
        assert packed.cpu().numpy().tobytes() == oracle_pack(g, fresh).tobytes()
    b.close()


def test_tables_made_while_launches_run(cuda, mpi_init):
    """Batches created, launched and closed while earlier ones of the stream
    are still queued, so that tables take the place of closed batches'."""
    import torch

    s = torch.cuda.Stream()
    grids = [grid((30 + 3 * k, 41 - 2 * k, 17 + k), 1 + k % 3, k) for k in range(8)]
    torch.cuda.synchronize()
    kept, outs = [], []
    for k in range(40):
        g, start, data = grids[k % 8]
        with torch.cuda.stream(s):
            torch.cuda._sleep(BUSY // 10)
            packed, b = packer(g, data)
            b.launch(s.cuda_stream)
        kept.append(b)
        outs.append((packed, g, start))
        if k % 3 == 2:
            kept.pop(0).close()
    torch.cuda.synchronize()
    for packed, g, start in outs:
        assert packed.cpu().numpy().tobytes() == oracle_pack(g, start).tobytes()
    for b in kept:
        b.close()


def test_two_streams_and_grids(cuda, mpi_init):
    """Two chains of pack and unpack on two streams, issued in turn; each reads
    only what the launch before it on its own stream wrote."""
    import torch

    chains = []
    for k, shape in enumerate(((70, 45, 33), (29, 64, 51))):
        g, start, data = grid(shape, 2 + k, 10 + k)
        packed, pack = packer(g, data)
        fill = halo.HaloBatch([g], [data.data_ptr()], [packed.data_ptr()], unpack=True)
        chains.append((g, start.copy(), data, packed, pack, fill, torch.cuda.Stream()))
    torch.cuda.synchronize()
    for _ in range(30):
        for g, _, data, packed, pack, fill, s in chains:
            pack.launch(s.cuda_stream)
            fill.launch(s.cuda_stream)
            with torch.cuda.stream(s):
                data.add_(1)
    torch.cuda.synchronize()
    for g, want, data, packed, pack, fill, s in chains:
        for _ in range(30):
            last = oracle_pack(g, want)
            want = oracle_unpack(g, last, want) + np.uint8(1)
        assert packed.cpu().numpy().tobytes() == last.tobytes()
        assert data.cpu().numpy().tobytes() == want.tobytes()
        pack.close()
        fill.close()
