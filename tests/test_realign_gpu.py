"""The realign kernel (kernel 5): rows of 16 B or more at any alignment, every
thread building whole 16-byte words of the destination.  Every pair of
alignments at row lengths around the word boundaries, zero to four strided
dimensions, one object and several; and the automatic rule's edges."""
import ctypes

import numpy as np
import pytest

from tempi_b200 import _lib

from . import helpers as H
from .test_canon import desc_pack
from .test_exchange_gpu import desc_unpack

pytestmark = pytest.mark.gpu


def roundtrip(d, incount, pmis, cfg, seed):
    """Pack and unpack by `cfg`; both against the descriptor's oracle, with the
    bytes around and between untouched.  Returns the two kernels' names."""
    import torch

    lib, total = _lib.tempi(), d.size * incount
    nbytes = d.start + d.extent * incount + 64
    src_np = H.splitmix_bytes(nbytes, seed)
    src = torch.from_numpy(src_np).cuda()
    out = torch.full((total + pmis + 32,), 0x5A, dtype=torch.uint8, device="cuda")
    back = torch.full((nbytes,), 0xAA, dtype=torch.uint8, device="cuda")
    pc = ctypes.byref(cfg) if cfg is not None else None
    torch.cuda.synchronize()
    _lib.check(lib.tempi_pack(ctypes.byref(d), src.data_ptr(), incount,
                              out.data_ptr() + pmis, pc, None))
    names = [lib.tempi_last_kernel().decode()]
    _lib.check(lib.tempi_unpack(ctypes.byref(d), out.data_ptr() + pmis, incount,
                                back.data_ptr(), pc, None))
    names.append(lib.tempi_last_kernel().decode())
    torch.cuda.synchronize()
    want = np.full(total + pmis + 32, 0x5A, np.uint8)
    want[pmis: pmis + total] = desc_pack(d, src_np, incount)
    assert out.cpu().numpy().tobytes() == want.tobytes(), (d.as_dict(), incount, pmis)
    exp = np.full(nbytes, 0xAA, np.uint8)
    desc_unpack(d, want[pmis: pmis + total], exp, incount)
    assert back.cpu().numpy().tobytes() == exp.tobytes(), (d.as_dict(), incount, pmis)
    return names


@pytest.mark.parametrize("words", [1, 4])
@pytest.mark.parametrize("block", [16, 17, 18, 24, 31, 32, 33, 47, 100, 255, 257, 4099])
def test_every_alignment(cuda, mpi_init, block, words):
    cfg = _lib.Config(5, 0, 0, words, 0, 0)
    for mis in range(16):
        pmis = (mis * 5 + block) % 16
        d = _lib.Desc.make(mis, 70 * (block + 21) + 5, block, [7, 5],
                           [block + mis % 5, 7 * (block + 4) + 9])
        assert roundtrip(d, 2, pmis, cfg, block + mis) == ["realign_pack", "realign_unpack"]


@pytest.mark.parametrize("nd", [0, 1, 2, 3, 4])
def test_dimensions(cuda, mpi_init, nd):
    """A contiguous run and up to four dimensions plus the object count."""
    for k, incount in enumerate((1, 3)):
        inner, counts, strides = 45, [], []
        for c in (6, 3, 5, 2)[:nd]:
            counts.append(c)
            strides.append(inner + 3)
            inner = c * (inner + 3)
        d = _lib.Desc.make(5, inner + 2, 45, counts, strides)
        for blocks_per_sm in (0, 1):
            cfg = _lib.Config(5, 0, 0, 4 if k else 1, blocks_per_sm, 0)
            roundtrip(d, incount, 3, cfg, nd)


@pytest.mark.parametrize("start,block,counts,strides,kernels", [
    (3, 1_000_001, [], [], ("realign", "realign")),        # a long odd run
    (3, 999_999, [], [], ("words", "words")),              # just too small for it
    (4, 33_554_436, [], [], ("realign", "realign")),       # 4-byte words from 32 MiB
    (4, 33_554_428, [], [], ("words", None)),
    (1, 127, [15_800], [130], ("realign", "realign")),     # short odd rows, 2 MB
    (1, 63, [32_000], [66], ("realign", None)),
    (1, 128, [15_800], [131], (None, "realign")),
    (1, 129, [31_100], [133], ("realign", "realign")),     # ... packs of up to 255 B, 4 MB
    (1, 256, [16_000], [259], (None, None)),
    (1, 4097, [2300], [4101], ("realign", "realign")),     # too few rows for a warp each
    (1, 4097, [2400], [4101], (None, None)),
    (1, 8193, [2400], [8201], ("realign", "realign")),
    (4, 260, [93_000], [264], (None, "realign")),          # rows that cut sectors, 60.3 MB
    (4, 260, [92_000], [264], (None, None)),               # ... 59.6 MB
    (2, 262, [74_000], [266], (None, "realign")),          # ... 48.2 MB of 2-byte words
    (16, 64, [240_000], [96], (None, "realign")),          # 16-byte words too
    (32, 64, [240_000], [96], (None, None)),               # whole sectors
    (4, 8196, [2300], [8212], ("realign", "realign")),     # long rows, too few of them
    (4, 8196, [2400], [8212], (None, None)),
    (16, 48, [250_000], [96], (None, None)),
    (16, 2048, [12_000], [2080], (None, None)),
])
def test_automatic_choice(cuda, mpi_init, start, block, counts, strides, kernels):
    sms = _sms()
    if sms != 148:
        pytest.skip("the edges are written for 148 SMs")
    hi = start + block + sum((c - 1) * s for c, s in zip(counts, strides))
    d = _lib.Desc.make(start, hi, block, counts, strides)
    names = roundtrip(d, 1, 0, None, block % 1000)
    for got, want in zip(names, kernels):
        if want is None:
            assert not got.startswith("realign"), names
        else:
            assert got.startswith(want), names


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count
