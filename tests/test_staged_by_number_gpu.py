"""Kernel 4 asked for by number where its bulk copies are not allowed (a packed
size that is no multiple of 16) takes the automatic rules, by kernel name."""
import ctypes

import pytest

from tempi_b200 import _lib

from . import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block,rows,gap,name", [
    (8_000_008, 1, 0, "words_unpack_w8"), (20, 1001, 12, "words_unpack_w4"),
    (1000, 601, 24, "rows_unpack_w8"), (520, 201, 24, "words_unpack_w8"),
    (16, 1001, 16, "staged_unpack_w16"),
])
def test_other_sizes_take_the_rules(cuda, mpi_init, block, rows, gap, name):
    import torch

    lib = _lib.tempi()
    d = _lib.Desc.make(0, rows * (block + gap), block, [rows], [block + gap])
    assert (d.size % 16 == 0) == name.startswith("staged")
    src = torch.from_numpy(H.splitmix_bytes(d.size, block % 1000)).cuda()
    back = torch.full((rows * (block + gap),), 0xAA, dtype=torch.uint8, device="cuda")
    cfg = _lib.Config(4, 0, 256, 0, 0, 0)
    torch.cuda.synchronize()
    for _ in range(2):  # the first staged launch may come before its failure word
        _lib.check(lib.tempi_unpack(ctypes.byref(d), src.data_ptr(), 1, back.data_ptr(),
                                    ctypes.byref(cfg), None))
    torch.cuda.synchronize()
    assert lib.tempi_last_kernel().decode() == name
    exp = torch.full((rows, block + gap), 0xAA, dtype=torch.uint8, device="cuda")
    exp[:, :block] = src.view(rows, block)
    assert torch.equal(back, exp.view(-1))
    _lib.check(lib.tempi_staged_check())
