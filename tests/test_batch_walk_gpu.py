"""The compact batch kernels step from word to word by adding to a word's
digits instead of dividing its index: every way a step of 32 words can carry
(row lengths and counts around 32, one word, one row), at every word width,
with few regions (their table in the kernel's parameters) and with many (in
device memory, its first chunks in shared memory or not)."""
import ctypes

import numpy as np
import pytest

from tempi_b200 import _lib

from . import helpers as H
from .test_canon import desc_pack
from .test_exchange_gpu import desc_unpack

pytestmark = pytest.mark.gpu

WORDS_PER_ROW = (1, 2, 3, 31, 32, 33, 65)
COUNTS = ((), (2,), (33,), (1, 5), (3, 7), (31, 2), (32, 3), (70, 2))


def layouts(width):
    """Descriptors of `width`-byte words: every row length x every count."""
    out = []
    for wpr in WORDS_PER_ROW:
        for counts in COUNTS:
            inner, strides = wpr * width, []
            for c in counts:
                strides.append(inner + width * 3)
                inner = c * strides[-1]
            out.append(_lib.Desc.make(width * 2, inner + width * 2, wpr * width, list(counts),
                                      strides))
    return out


def place(descs, width):
    regs, typed, packed = [], 0, 0
    for d in descs:
        regs.append((typed, d, packed))
        typed += d.extent + 64 // width * width
        packed += d.size + 2 * width
    return regs, typed + 64, packed + 64


def launch(regs, tp, pp, unpack):
    arr = (_lib.Region * len(regs))()
    for k, (b, d, off) in enumerate(regs):
        arr[k].origin, arr[k].packed = tp + b, pp + off
        arr[k].desc, arr[k].incount = d, 1
    h = ctypes.c_void_p()
    _lib.check(_lib.tempi().tempi_batch_create(arr, len(regs), unpack, ctypes.byref(h)))
    _lib.check(_lib.tempi().tempi_batch_launch(h, None))
    return h


@pytest.mark.parametrize("per_batch", [28, 10000])
@pytest.mark.parametrize("width", [1, 2, 4, 8, 16])
def test_every_carry(cuda, mpi_init, width, per_batch):
    import torch

    descs = layouts(width)
    regs, nt, npk = place(descs, width)
    typed_np, packed_np = H.splitmix_bytes(nt, width), H.splitmix_bytes(npk, 50 + width)
    typed = torch.from_numpy(typed_np).cuda()
    packed = torch.full((npk,), 0x5A, dtype=torch.uint8, device="cuda")
    into = torch.full((nt,), 0xAA, dtype=torch.uint8, device="cuda")
    source = torch.from_numpy(packed_np).cuda()
    handles = []
    for i in range(0, len(regs), per_batch):
        part = regs[i: i + per_batch]
        handles.append(launch(part, typed.data_ptr(), packed.data_ptr(), 0))
        handles.append(launch(part, into.data_ptr(), source.data_ptr(), 1))
    torch.cuda.synchronize()
    for h in handles:
        _lib.tempi().tempi_batch_destroy(h)
    want, back = np.full(npk, 0x5A, np.uint8), np.full(nt, 0xAA, np.uint8)
    for b, d, off in regs:
        want[off: off + d.size] = desc_pack(d, typed_np[b:], 1)
        desc_unpack(d, packed_np[off: off + d.size], back[b:], 1)
    assert packed.cpu().numpy().tobytes() == want.tobytes()
    assert into.cpu().numpy().tobytes() == back.tobytes()


def test_more_regions_than_shared_memory_holds(cuda, mpi_init):
    """9,000 regions: the search for a chunk's region reads the table."""
    import torch

    descs = [_lib.Desc.make(4 * (k % 3), 256, 4 * (k % 7 + 1), [k % 4 + 1], [44])
             for k in range(9000)]
    regs, nt, npk = place(descs, 4)
    typed_np = H.splitmix_bytes(nt, 9)
    typed = torch.from_numpy(typed_np).cuda()
    packed = torch.full((npk,), 0x5A, dtype=torch.uint8, device="cuda")
    h = launch(regs, typed.data_ptr(), packed.data_ptr(), 0)
    torch.cuda.synchronize()
    _lib.tempi().tempi_batch_destroy(h)
    want = np.full(npk, 0x5A, np.uint8)
    for b, d, off in regs:
        want[off: off + d.size] = desc_pack(d, typed_np[b:], 1)
    assert packed.cpu().numpy().tobytes() == want.tobytes()


@pytest.mark.parametrize("width", [1, 4, 8, 16])
def test_copy_between_walks(cuda, mpi_init, width):
    """Copy pairs whose two sides step differently through the same words."""
    import torch

    sides = [d for d in layouts(width) if d.ndims]
    pairs, ns, nd = [], 0, 0
    for s in sides:
        words = s.size // width
        row = max(r for r in (1, 2, 5, 33) if words % r == 0)
        d = _lib.Desc.make(width, words // row * (row + 1) * width + width, row * width,
                           [words // row], [(row + 1) * width])
        pairs.append((ns, s, nd, d))
        ns += s.extent + 16 * width
        nd += d.extent + 16 * width
    src_np = H.splitmix_bytes(ns + 64, 3)
    src = torch.from_numpy(src_np).cuda()
    dst = torch.full((nd + 64,), 0xAA, dtype=torch.uint8, device="cuda")
    for i in range(0, len(pairs), 30):
        part = pairs[i: i + 30]
        arr = (_lib.CopyRegion * len(part))()
        for k, (sb, s, db, d) in enumerate(part):
            arr[k].src_origin, arr[k].dst_origin = src.data_ptr() + sb, dst.data_ptr() + db
            arr[k].src_desc, arr[k].dst_desc = s, d
            arr[k].src_count = arr[k].dst_count = 1
        h = ctypes.c_void_p()
        _lib.check(_lib.tempi().tempi_batch_create_copy(arr, len(part), ctypes.byref(h)))
        _lib.check(_lib.tempi().tempi_batch_launch(h, None))
        torch.cuda.synchronize()
        _lib.tempi().tempi_batch_destroy(h)
    want = np.full(nd + 64, 0xAA, np.uint8)
    for sb, s, db, d in pairs:
        desc_unpack(d, desc_pack(s, src_np[sb:], 1), want[db:], 1)
    assert dst.cpu().numpy().tobytes() == want.tobytes()


def test_dependent_launches_overlap_safely(cuda, mpi_init):
    """Batches launched back to back on one stream, each reading what the one
    before wrote: a kernel may start early but touches no buffer before the
    kernels ahead of it have finished."""
    import torch

    from tempi_b200 import halo, mpi

    g = halo.Grid((70, 45, 33), 2)
    start = H.splitmix_bytes(g.nbytes, 77)
    data = torch.from_numpy(start).cuda()
    packed = torch.zeros(g.packed_bytes, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()
    pack = halo.HaloBatch([g], [data.data_ptr()], [packed.data_ptr()])
    fill = halo.HaloBatch([g], [data.data_ptr()], [packed.data_ptr()], unpack=True)
    want = start.copy()
    order = [(d, tuple(-x for x in d)) for d in halo.directions()]
    descs = {}
    for d, _ in order:
        descs[d, False] = mpi.describe(g.send[d])[1]
        descs[d, True] = mpi.describe(g.recv[d])[1]
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for k in range(40):
            pack.launch(stream.cuda_stream)
            fill.launch(stream.cuda_stream)
            data.add_(1)  # an ordinary kernel between overlapped ones
    stream.synchronize()
    for k in range(40):
        bytes_of = {d: desc_pack(descs[d, False], want, 1) for d, _ in order}
        for d, opposite in order:
            desc_unpack(descs[opposite, True], bytes_of[d], want, 1)
        last = np.concatenate([bytes_of[d] for d, _ in order])
        want += np.uint8(1)
    assert packed.cpu().numpy().tobytes() == last.tobytes()
    assert data.cpu().numpy().tobytes() == want.tobytes()
    # two batches straight after each other, many times: the second undoes
    # nothing and reads only finished bytes
    for k in range(50):
        pack.launch(stream.cuda_stream)
        fill.launch(stream.cuda_stream)
    stream.synchronize()
    bytes_of = {d: desc_pack(descs[d, False], want, 1) for d, _ in order}
    for d, opposite in order:
        desc_unpack(descs[opposite, True], bytes_of[d], want, 1)
    assert data.cpu().numpy().tobytes() == want.tobytes()
    # launches inside a capture become ordinary nodes
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        data.add_(3)
        pack.launch(stream.cuda_stream)
        fill.launch(stream.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    want += np.uint8(3)
    bytes_of = {d: desc_pack(descs[d, False], want, 1) for d, _ in order}
    for d, opposite in order:
        desc_unpack(descs[opposite, True], bytes_of[d], want, 1)
    assert data.cpu().numpy().tobytes() == want.tobytes()
    pack.close()
    fill.close()


@pytest.mark.parametrize("edges", [3, 32, 33])
@pytest.mark.parametrize("counts", [(1,), (1, 2), (1, 0, 3)])
@pytest.mark.parametrize("offset", [0, 1, 4, 8])
def test_exchange_of_committed_types(cuda, mpi_init, edges, counts, offset):
    """MPI_Neighbor_alltoallw over self-edges, single objects (whose geometries
    come from the commit) and several, at displacements that narrow the words,
    among one, two and three strided dimensions, up to and past the number of
    edges that fit the kernel's parameters."""
    import torch

    from tempi_b200 import mpi

    def commit(shape):
        block, c, s = shape
        inner, t = block, mpi.Type_contiguous(block, mpi.BYTE)
        for n, gap in zip(c, s):
            t = mpi.Type_create_hvector(n, 1, inner + gap, t)
            inner = (n - 1) * (inner + gap) + inner
        t = mpi.Type_create_resized(t, 0, inner + 16 - inner % 16)
        assert mpi.Type_commit(t) == 0
        return t

    kinds = [(48, (4,), (16,)), (16, (6, 2), (32, 16)), (24, (2, 2, 2), (8, 8, 8)), (192, (), ())]
    types = [commit(k) for k in kinds]
    descs = [mpi.describe(t)[1] for t in types]
    assert len({d.size for d in descs}) == 1
    sends = [k % 4 for k in range(edges)]
    recvs = [(k + k // 4 + 1) % 4 for k in range(edges)]
    n = [counts[k % len(counts)] for k in range(edges)]
    at, sd, rd = 0, [], []
    for k in range(edges):
        sd.append(at + (offset if k % 3 else 0))
        rd.append(at + 16)
        at += 3 * 1024 + 64
    src_np = H.splitmix_bytes(at + 64, edges)
    src = torch.from_numpy(src_np).cuda()
    dst = torch.full((at + 64,), 0xAA, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    err, comm = mpi.Dist_graph_create_adjacent([0] * edges, [0] * edges)
    assert err == 0
    before = _lib.counter("neighbor_fused")
    for _ in range(2):
        assert mpi.Neighbor_alltoallw(
            src.data_ptr(), n, sd, [types[k] for k in sends], dst.data_ptr(), n, rd,
            [types[k] for k in recvs], comm) == 0, _lib.last_error()
    assert _lib.counter("neighbor_fused") == before + 2
    want = np.full(at + 64, 0xAA, np.uint8)
    for k in range(edges):
        if n[k]:
            got = desc_pack(descs[sends[k]], src_np[sd[k]:], n[k])
            desc_unpack(descs[recvs[k]], got, want[rd[k]:], n[k])
    assert dst.cpu().numpy().tobytes() == want.tobytes()
    mpi.Comm_free(comm)
