"""Kernels between two pinned host buffers run on a grid that keeps only a
bounded number of bytes in flight: every kernel walks its whole object in
several passes there, at row lengths that fill a lane group's pass and that
leave most of it idle, through tempi_pack (which looks the buffers up) and
through MPI_Pack (which knows them)."""
import ctypes

import numpy as np
import pytest

from tempi_b200 import _lib, mpi

from . import helpers as H
from .test_canon import desc_pack
from .test_exchange_gpu import desc_unpack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,lanes", [(0, 0), (1, 0), (2, 0), (3, 4), (3, 32)])
@pytest.mark.parametrize("block,rows,gap", [
    (2_000_003, 1, 5), (16, 70_000, 16), (12, 60_000, 4), (1024, 1500, 512), (301, 3500, 47),
    (5001, 300, 30),
])
def test_host_to_host(cuda, mpi_init, kernel, lanes, block, rows, gap):
    import torch

    lib = _lib.tempi()
    d = _lib.Desc.make(7 if block % 2 else 16, 32 + rows * (block + gap), block, [rows],
                       [block + gap])
    nbytes = d.extent
    src_np = H.splitmix_bytes(nbytes, block)
    src = torch.from_numpy(src_np).pin_memory()
    packed = torch.full((d.size + 16,), 0x5A, dtype=torch.uint8).pin_memory()
    back = torch.full((nbytes,), 0xAA, dtype=torch.uint8).pin_memory()
    cfg = _lib.Config(kernel, 0, 256, lanes, 0, 0)
    _lib.check(lib.tempi_pack(ctypes.byref(d), src.data_ptr(), 1, packed.data_ptr(),
                              ctypes.byref(cfg), None))
    _lib.check(lib.tempi_unpack(ctypes.byref(d), packed.data_ptr(), 1, back.data_ptr(),
                                ctypes.byref(cfg), None))
    torch.cuda.synchronize()
    want = np.full(d.size + 16, 0x5A, np.uint8)
    want[: d.size] = desc_pack(d, src_np, 1)
    assert packed.numpy().tobytes() == want.tobytes()
    exp = np.full(nbytes, 0xAA, np.uint8)
    desc_unpack(d, want[: d.size], exp, 1)
    assert back.numpy().tobytes() == exp.tobytes()


def test_mpi_pack_between_host_buffers(cuda, mpi_init):
    import torch

    ty = H.subarray([700, 3000], [700, 2200], [0, 5], mpi.ORDER_C, H.named("BYTE")).commit()
    src_np = H.splitmix_bytes(700 * 3000, 4)
    src = torch.from_numpy(src_np).pin_memory()
    packed = torch.zeros(700 * 2200, dtype=torch.uint8).pin_memory()
    back = torch.full_like(src, 0xAA).pin_memory()
    before = _lib.tempi().tempi_kernel_launches()
    assert mpi.Pack(src.data_ptr(), 1, ty.h, packed.data_ptr(), 700 * 2200) == (0, 700 * 2200)
    assert mpi.Unpack(packed.data_ptr(), 700 * 2200, back.data_ptr(), 1, ty.h)[0] == 0
    assert _lib.tempi().tempi_kernel_launches() > before
    box = src_np.reshape(700, 3000)[:, 5:2205]
    assert packed.numpy().tobytes() == np.ascontiguousarray(box).tobytes()
    exp = np.full((700, 3000), 0xAA, np.uint8)
    exp[:, 5:2205] = box
    assert back.numpy().tobytes() == exp.tobytes()
