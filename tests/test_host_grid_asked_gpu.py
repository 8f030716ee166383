"""Between two pinned host buffers the library bounds the bytes in flight by
launching fewer blocks, but a caller's blocks_per_sm stands."""
import ctypes

import pytest

from tempi_b200 import _lib

from . import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,lanes,need", [(1, 0, 256), (2, 0, 512), (3, 32, 512)])
def test_blocks_per_sm_stands(cuda, mpi_init, kernel, lanes, need):
    """4 MiB in 4,096 rows of 1 KiB: `need` blocks of 256 threads would take
    every row or four words a thread once."""
    import torch

    lib, sms = _lib.tempi(), torch.cuda.get_device_properties(0).multi_processor_count
    d = _lib.Desc.make(0, 4096 * 1536, 1024, [4096], [1536])
    src = torch.from_numpy(H.splitmix_bytes(d.extent, kernel)).pin_memory()
    packed = torch.zeros(d.size, dtype=torch.uint8).pin_memory()
    want = src.view(4096, 1536)[:, :1024].reshape(-1)
    for asked, limit in ((8, 8 * sms), (1, sms), (0, None)):
        cfg = _lib.Config(kernel, 0, 256, lanes, asked, 0)
        packed.zero_()
        n = _lib.counter("pack_ctas")
        _lib.check(lib.tempi_pack(ctypes.byref(d), src.data_ptr(), 1, packed.data_ptr(),
                                  ctypes.byref(cfg), None))
        torch.cuda.synchronize()
        ctas = _lib.counter("pack_ctas") - n
        if asked:
            assert ctas == min(need, limit)
        else:
            assert 1 <= ctas <= 80
        assert torch.equal(packed, want)
