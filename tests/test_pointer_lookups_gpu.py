"""tempi_pack asks the runtime where its buffers are only when the launch turns
on it, and for each buffer at most once."""
import ctypes

import pytest

from tempi_b200 import _lib

from . import helpers as H

pytestmark = pytest.mark.gpu

KB, MB = 1 << 10, 1 << 20


@pytest.mark.parametrize("where,nbytes,block,cfg,lookups", [
    ("cuda", 256 * KB, 64, (1, 0, 256, 0, 0, 0), 0),   # too small for any grid to differ
    ("cuda", 1 * MB, 64, (1, 0, 256, 0, 0, 0), 2),     # SMs without a block
    ("cuda", 8 * MB, 64, (1, 0, 256, 0, 0, 0), 1),     # a full grid: only whether it is the host
    ("cuda", 8 * MB, 64, (1, 0, 256, 0, 2, 0), 0),     # the caller's grid
    ("cuda", 8 * MB, 1024, (2, 0, 256, 0, 0, 0), 1),
    ("cuda", 8 * MB, 1024, (3, 0, 0, 32, 0, 0), 2),    # rows once each, in device memory
    ("cuda", 8 * MB, 1024, (3, 0, 256, 32, 0, 0), 1),
    ("cuda", 8 * MB, 1024, (4, 0, 0, 0, 0, 0), 2),     # bulk copies
    ("cuda", 8 * MB, 1023, (0, 0, 0, 0, 0, 0), 2),     # rules for odd rows, then the grid
    ("host", 8 * MB, 64, (1, 0, 256, 0, 0, 0), 2),
])
def test_lookups(cuda, mpi_init, where, nbytes, block, cfg, lookups):
    import torch

    lib, rows = _lib.tempi(), nbytes // block
    d = _lib.Desc.make(0, rows * 2 * block, block, [rows], [2 * block])
    src = torch.from_numpy(H.splitmix_bytes(d.extent, block))
    packed = torch.zeros(d.size, dtype=torch.uint8)
    want = src.view(rows, 2 * block)[:, :block].reshape(-1).clone()
    src, packed = ((src.cuda(), packed.cuda()) if where == "cuda"
                   else (src.pin_memory(), packed.pin_memory()))
    c = _lib.Config(*cfg)
    torch.cuda.synchronize()
    n = _lib.counter("pointer_lookups")
    assert n >= 0
    _lib.check(lib.tempi_pack(ctypes.byref(d), src.data_ptr(), 1, packed.data_ptr(),
                              ctypes.byref(c), None))
    torch.cuda.synchronize()
    assert _lib.counter("pointer_lookups") == n + lookups
    assert torch.equal(packed.cpu(), want)
