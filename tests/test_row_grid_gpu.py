"""The shift and row kernels take rows of 64 B to 4 KiB in device memory once
each (the row kernel: from 32 MB), with as many CTAs of 128 threads as that
needs: row counts on both sides of the grid that fills the GPU (2368 such CTAs
on 148 SMs), a last CTA with one row, row lengths at the ends of the range and
beyond it, one and two strided dimensions."""
import ctypes

import pytest

from tempi_b200 import _lib

from . import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,lanes", [(2, 0), (3, 4), (3, 32)])
@pytest.mark.parametrize("block,planes,rows,gap", [
    (63, 1, 20_001, 5), (64, 1, 76_001, 3), (65, 3, 25_301, 63), (300, 2, 5_001, 20),
    (1027, 5, 6_501, 13), (4095, 1, 9_501, 2), (4096, 1, 301, 9), (4097, 7, 43, 31),
])
def test_rows_taken_once(cuda, mpi_init, kernel, lanes, block, planes, rows, gap):
    import torch

    lib = _lib.tempi()
    pitch, depth, start = block + gap, rows + 1, 2
    nbytes = planes * depth * pitch
    d = _lib.Desc.make(start, nbytes, block, [rows, planes], [pitch, depth * pitch])
    src = torch.from_numpy(H.splitmix_bytes(nbytes, block)).cuda()
    packed = torch.full((d.size + 32,), 0x5A, dtype=torch.uint8, device="cuda")
    back = torch.full((nbytes,), 0xAA, dtype=torch.uint8, device="cuda")
    cfg = _lib.Config(kernel, 0, 0, lanes, 0, 0)
    _lib.check(lib.tempi_pack(ctypes.byref(d), src.data_ptr(), 1, packed.data_ptr(),
                              ctypes.byref(cfg), None))
    _lib.check(lib.tempi_unpack(ctypes.byref(d), packed.data_ptr(), 1, back.data_ptr(),
                                ctypes.byref(cfg), None))
    torch.cuda.synchronize()
    box = (slice(None), slice(0, rows), slice(start, start + block))
    want = src.view(planes, depth, pitch)[box]
    assert torch.equal(packed[: d.size], want.reshape(-1))
    assert bool((packed[d.size:] == 0x5A).all())
    exp = torch.full((planes, depth, pitch), 0xAA, dtype=torch.uint8, device="cuda")
    exp[box] = want
    assert torch.equal(back, exp.view(-1))
