"""The work whose speed this library is judged by, as cases that a program can time.

Every case goes through a public entry point: the interposed MPI calls
(MPI_Pack, MPI_Unpack, MPI_Isend/Irecv/Wait, MPI_Neighbor_alltoallw), called
as a C program calls them with its argument arrays already in hand, or the
batch handles of ``tempi_b200.halo``.  A case is a dict of plain values; its
``kind`` says what one pass does:

  strided   MPI_Pack and/or MPI_Unpack of `incount` objects of one datatype
  calls     one MPI_Pack per send region and one MPI_Unpack per ghost region
            of a 3-D grid (52 synchronous calls)
  batch     the same regions of one or several grids by one batched pack and
            one batched unpack
  exchange  the periodic self-exchange of a grid by MPI_Neighbor_alltoallw
  send      MPI_Irecv + MPI_Isend + MPI_Wait x2 of an object to this rank

Datatypes are described by ``elem`` (the named type) and either a subarray
(``sizes``/``subs``/``starts``, slowest dimension first, written as texts like
"256x256x64") or nested vectors (``block`` bytes, then ``counts`` and byte
``strides``, fastest first, after ``offset`` bytes).
"""
from __future__ import annotations

import ctypes
import math

import torch

from tempi_b200 import _lib, halo, mpi

ELEMS = {"byte": (mpi.BYTE, 1), "float": (mpi.FLOAT, 4), "double": (mpi.DOUBLE, 8)}
# interiors of the mixed batch: the grids of halo.mixed_shapes()
MIXED = "mixed8"


def listed():
    return [
        # a small message of a row-strided array: 1024 blocks of 64 B, both
        # ways; the call's fixed cost is all that counts
        dict(name="vector_1024x64", kind="strided", direction="both", elem="byte", offset=0,
             block=64, counts="1024", strides="512", incount=1),
        # an application that packs and unpacks its 26 neighbour regions one
        # call at a time, as MPI programs are mostly written
        dict(name="halo256_calls", kind="calls", grids="256x256x256", radius=2, elem="double"),
        # data that lives in pinned host memory: rows of a 2-D float array
        # over the host link, in and out
        dict(name="host_2d_rows1k", kind="strided", direction="both", where="host", elem="float",
             sizes="1024x1024", subs="1024x256", starts="0x531", incount=4),
        # short rows of a 3-D float volume (64 B at an odd offset in a line):
        # a thin slab of the fastest dimension, both ways
        dict(name="sub3d_rows64", kind="strided", direction="both", elem="float",
             sizes="256x256x256", subs="256x256x16", starts="0x0x190", incount=4),
        # medium rows of the same volume received into place
        dict(name="sub3d_rows256_unpack", kind="strided", direction="unpack", elem="float",
             sizes="256x256x256", subs="256x256x64", starts="0x0x135", incount=4),
        # whole volumes: the largest message, one contiguous run
        dict(name="sub3d_whole_pack", kind="strided", direction="pack", elem="float",
             sizes="256x256x256", subs="256x256x256", starts="0x0x0", incount=4),
        # a crop of an 8-bit image with odd width and offset: long rows whose
        # two sides never agree modulo 16
        dict(name="bytes2d_crop_pack", kind="strided", direction="pack", elem="byte",
             sizes="8209x4001", subs="8191x2999", starts="7x13", incount=1),
        # a ragged box of an 8-bit volume received into place: short odd rows
        dict(name="bytes3d_box_unpack", kind="strided", direction="unpack", elem="byte",
             sizes="397x401x403", subs="193x211x201", starts="5x11x17", incount=1),
        # the batched halo step of one grid: pack the sends, fill the ghosts
        dict(name="halo256_batch", kind="batch", grids="256x256x256", radius=2, elem="double"),
        # several unlike grids in one step (208 regions a direction)
        dict(name="halo_mixed8_batch", kind="batch", grids=MIXED, radius=0, elem="double"),
        # a periodic halo exchange by the collective
        dict(name="halo256_alltoallw", kind="exchange", grids="256x256x256", radius=2,
             elem="double"),
        # a non-blocking transfer of a strided volume to the same rank
        dict(name="self_send_3d_16MiB", kind="send", elem="float", sizes="256x256x256",
             subs="256x256x64", starts="0x0x67", incount=1),
    ]


# ---- the ranges the listed cases stand for -----------------------------------


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _ints(s):
    return [int(x) for x in str(s).split("x")]


def _text(v):
    return "x".join(str(int(x)) for x in v)


def _draw_vectors(rng, total_hi, span_hi):
    """1 to 3 dimensions, blocks of 1 B to 64 KiB, totals from 1 KiB, strides
    up to 16 times the inner extent at every alignment."""
    while True:
        nd, align = rng.randint(1, 3), rng.choice((1, 2, 4, 8, 16))
        total = _log(rng, 1024, total_hi)
        block = _log(rng, 1, 65536)
        incount = 1 if rng.random() < 0.7 else rng.randint(2, 16)
        offset = align * rng.randint(0, 3)
        rows = max(1, total // (block * incount))
        if nd == 1:
            block, counts = max(1, total // incount), []
        elif nd == 2:
            counts = [rows]
        else:
            c1 = _log(rng, 1, rows)
            counts = [c1, max(1, rows // c1)]
        inner, strides = block, []
        for c in counts:
            s = max(inner, int(inner * rng.uniform(1, 16)))
            strides.append(-(-s // align) * align)
            inner = c * strides[-1]
        n = block * math.prod(counts) * incount
        span = (offset + inner + 16) * incount
        if n <= total_hi and span <= span_hi:
            return dict(offset=offset, block=block, counts=_text(counts), strides=_text(strides),
                        incount=incount)


def _draw_subarray(rng):
    """2-D and 3-D subarrays of bytes, floats and doubles: the strided sweep's
    inner extents and odd ones, at every start."""
    nd = rng.choice((2, 3))
    elem = rng.choice(("byte", "float", "float", "double"))
    if nd == 2:
        sizes = [_log(rng, 256, 4096), _log(rng, 256, 4096)]
    else:
        sizes = [_log(rng, 64, 384) for _ in range(3)]
    subs = [rng.randint(max(1, s // 3), s) for s in sizes]
    subs[-1] = _log(rng, 1, sizes[-1])
    starts = [rng.randint(0, s - b) for s, b in zip(sizes, subs)]
    es = ELEMS[elem][1]
    most = max(1, min(16, (256 << 20) // (math.prod(sizes) * es)))
    return dict(elem=elem, sizes=_text(sizes), subs=_text(subs), starts=_text(starts),
                incount=rng.randint(1, most))


def draw(rng):
    pick = rng.random()
    if pick < 0.55:  # packs and unpacks on the device
        c = dict(kind="strided", direction=rng.choice(("pack", "unpack", "both")))
        if rng.random() < 0.5:
            c.update(_draw_subarray(rng))
        else:
            c.update(elem="byte", **_draw_vectors(rng, 128 << 20, 1 << 30))
        return c
    if pick < 0.62:  # pinned host memory
        return dict(kind="strided", direction=rng.choice(("pack", "unpack")), where="host",
                    elem="byte", **_draw_vectors(rng, 4 << 20, 16 << 20))
    if pick < 0.72:  # self-sends, 4 KiB to 64 MiB, inner blocks of 4 B to 4 KiB
        block = _log(rng, 4, 4096)
        rows = max(1, _log(rng, 4096, 64 << 20) // block)
        stride = block * rng.randint(2, 4) + rng.choice((0, 0, 4, 16))
        return dict(kind="send", elem="byte", offset=0, block=block, counts=str(rows),
                    strides=str(stride), incount=1)
    # halos: each interior dimension log-uniform, radius 1 to 3
    kind = rng.choice(("batch", "batch", "exchange", "calls"))
    dims = [_log(rng, 32, 320) for _ in range(3)]
    return dict(kind=kind, grids=_text(dims), radius=rng.randint(1, 3),
                elem=rng.choice(("float", "double", "double")))


# ---- a program's set-up -------------------------------------------------------


def _random_bytes(n, seed, host=False):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=gen)
    return t.cpu().pin_memory() if host else t


def _buffer(n, fill, host=False):
    t = torch.full((n,), fill, dtype=torch.uint8, device="cuda")
    return t.cpu().pin_memory() if host else t


def _datatype(case):
    """(committed datatype, bytes from the origin that its objects span)"""
    elem, es = ELEMS[case["elem"]]
    n = case["incount"]
    if "sizes" in case:
        sizes = _ints(case["sizes"])
        t = mpi.Type_create_subarray(sizes, _ints(case["subs"]), _ints(case["starts"]),
                                     mpi.ORDER_C, elem)
        span = math.prod(sizes) * es * n
    else:
        counts = _ints(case["counts"]) if case["counts"] else []
        strides = _ints(case["strides"]) if case["strides"] else []
        t = mpi.Type_contiguous(case["block"], elem)
        hi = case["offset"] + case["block"]
        for c, s in zip(counts, strides):
            t = mpi.Type_create_hvector(c, 1, s, t)
            hi += (c - 1) * s
        if case["offset"]:
            t = mpi.Type_create_hindexed([1], [case["offset"]], t)
        t = mpi.Type_create_resized(t, 0, hi)
        span = hi * n
    if mpi.Type_commit(t):
        raise RuntimeError("MPI_Type_commit failed")
    return t, span


def _grids(case):
    elem, es = ELEMS[case["elem"]]
    if case["grids"] == MIXED:
        shapes = halo.mixed_shapes()
    else:
        shapes = [(_ints(case["grids"]), case["radius"])]
    return [halo.Grid(interior, r, elem, es) for interior, r in shapes]


def _packed_bytes(case):
    if case["kind"] in ("strided", "send"):
        es = ELEMS[case["elem"]][1]
        if "subs" in case:
            n = math.prod(_ints(case["subs"])) * es
        else:
            n = case["block"] * math.prod(_ints(case["counts"]) if case["counts"] else [])
        return n * case["incount"]
    shapes = halo.mixed_shapes() if case["grids"] == MIXED else [
        (_ints(case["grids"]), case["radius"])]
    es = ELEMS[case["elem"]][1]
    total = 0
    for (nx, ny, nz), r in shapes:
        for d in halo.directions():
            ext = [r if di else m for di, m in zip(d, (nx, ny, nz))]
            total += math.prod(ext) * es
    return total


def prepare(case, seed):
    if mpi.Init():
        raise RuntimeError("MPI_Init failed")
    lib = _lib.tempi()
    kind = case["kind"]
    st = dict(kind=kind, lib=lib, n=case.get("incount", 1))
    if kind in ("strided", "send"):
        t, span = _datatype(case)
        nbytes = _packed_bytes(case)
        host = case.get("where") == "host"
        st.update(t=t, nbytes=nbytes, pos=ctypes.c_int(0), direction=case.get("direction"))
        if kind == "send" or st["direction"] != "unpack":
            st["src"] = _random_bytes(span, seed, host)
        if kind == "strided":
            if st["direction"] == "unpack":
                st["packed"] = _random_bytes(nbytes, seed, host)
            else:
                st["packed"] = _buffer(nbytes, 0, host)
        if kind == "send" or st["direction"] != "pack":
            st["dst"] = _buffer(span, 0xAA, host)
        if kind == "send":
            st.update(rq=ctypes.c_int(0), sq=ctypes.c_int(0), status=_lib.Status())
        return st
    grids = _grids(case)
    data = [_random_bytes(g.nbytes, seed + 101 * i) for i, g in enumerate(grids)]
    st["data"] = data
    if kind == "batch":
        st["packed"] = [_buffer(g.packed_bytes, 0) for g in grids]
        gp, pp = [d.data_ptr() for d in data], [p.data_ptr() for p in st["packed"]]
        st["pack"] = halo.HaloBatch(grids, gp, pp)
        st["unpack"] = halo.HaloBatch(grids, gp, pp, unpack=True)
    elif kind == "calls":
        g = grids[0]
        st["packed"] = _buffer(g.packed_bytes, 0)
        st["pos"] = ctypes.c_int(0)
        st["nbytes"] = g.packed_bytes
        st["sends"] = [g.send[d] for d in halo.directions()]
        st["recvs"] = [g.recv[tuple(-x for x in d)] for d in halo.directions()]
    else:
        sg = halo.SelfGraph(grids[0])
        m = len(sg.sendtypes)
        ones, zeros = (ctypes.c_int * m)(*[1] * m), (ctypes.c_ssize_t * m)(*[0] * m)
        p = data[0].data_ptr()
        st["graph"] = sg
        st["args"] = (p, ones, zeros, (ctypes.c_int * m)(*sg.sendtypes), p, ones, zeros,
                      (ctypes.c_int * m)(*sg.recvtypes), sg.comm)
    return st


# ---- one pass -----------------------------------------------------------------


def _check(err):
    if err:
        raise RuntimeError(f"MPI error {err}: {_lib.last_error()}")


def _run_strided(st):
    lib, t, n, nbytes, pos = st["lib"], st["t"], st["n"], st["nbytes"], st["pos"]
    packed = st["packed"].data_ptr()
    out = {}
    if st["direction"] != "unpack":
        pos.value = 0
        _check(lib.MPI_Pack(st["src"].data_ptr(), n, t, packed, nbytes, ctypes.byref(pos),
                            mpi.COMM_WORLD))
        out["packed"] = st["packed"]
    if st["direction"] != "pack":
        pos.value = 0
        _check(lib.MPI_Unpack(packed, nbytes, ctypes.byref(pos), st["dst"].data_ptr(), n, t,
                              mpi.COMM_WORLD))
        out["dst"] = st["dst"]
    return out


def _run_calls(st):
    lib, pos, nbytes = st["lib"], st["pos"], st["nbytes"]
    p, grid, packed = ctypes.byref(pos), st["data"][0].data_ptr(), st["packed"].data_ptr()
    pos.value = 0
    for t in st["sends"]:
        _check(lib.MPI_Pack(grid, 1, t, packed, nbytes, p, mpi.COMM_WORLD))
    pos.value = 0
    for t in st["recvs"]:
        _check(lib.MPI_Unpack(packed, nbytes, p, grid, 1, t, mpi.COMM_WORLD))
    return [st["packed"], st["data"][0]]


def _run_send(st):
    lib, t, n = st["lib"], st["t"], st["n"]
    rq, sq, status = ctypes.byref(st["rq"]), ctypes.byref(st["sq"]), ctypes.byref(st["status"])
    _check(lib.MPI_Irecv(st["dst"].data_ptr(), n, t, 0, 5, mpi.COMM_WORLD, rq))
    _check(lib.MPI_Isend(st["src"].data_ptr(), n, t, 0, 5, mpi.COMM_WORLD, sq))
    _check(lib.MPI_Wait(rq, status))
    _check(lib.MPI_Wait(sq, status))
    return st["dst"]


def run(state):
    kind = state["kind"]
    if kind == "strided":
        return _run_strided(state)
    if kind == "send":
        return _run_send(state)
    if kind == "calls":
        return _run_calls(state)
    if kind == "batch":
        state["pack"].launch()
        state["unpack"].launch()
        return [state["packed"], state["data"]]
    _check(state["lib"].MPI_Neighbor_alltoallw(*state["args"]))
    return state["data"][0]


def work(case):
    """Every described byte read once and written once, in each direction."""
    n = _packed_bytes(case)
    both = case["kind"] in ("calls", "batch") or case.get("direction") == "both"
    # a self-send must read the object and write the other one; the message
    # in between is the library's choice
    return {"bytes": 2 * n * (2 if both else 1), "flops": 0}
