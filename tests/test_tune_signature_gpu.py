"""Tuned choices belong to the kernels they were timed on: regions of two
strided dimensions and regions of three, alike in words and row length, run
different kernels, and lines of a tune file written for earlier kernels are
not taken."""
import ctypes
import os
import subprocess
import sys

import pytest

from tempi_b200 import _lib

from . import helpers as H
from .test_batch_walk_gpu import launch
from .test_canon import desc_pack

pytestmark = pytest.mark.gpu

CLASS = 8 * 3 + 1  # 8-byte words, two or three to a row


def layout(dims):
    """96 rows of 24 bytes over `dims` strided dimensions."""
    counts = {2: [12, 8], 3: [12, 4, 2]}[dims]
    inner, strides = 24, []
    for c in counts:
        strides.append(inner + 8)
        inner = c * strides[-1]
    return _lib.Desc.make(0, inner, 24, counts, strides)


def config(h):
    th, cps = ctypes.c_int32(), ctypes.c_int32()
    cls, passes = (ctypes.c_int32 * 4)(), (ctypes.c_int32 * 4)()
    n = _lib.tempi().tempi_batch_config(h, ctypes.byref(th), ctypes.byref(cps), cls, passes, 4)
    assert n == 1 and cls[0] == CLASS
    return th.value, cps.value, passes[0]


def before(dims, regions, unpack=0):
    """The signature that earlier kernels stored: kind, then the keys."""
    h = 1469598103934665603
    for v in [unpack] + [CLASS << 8 | 8] * regions:  # 96 rows of 3 words: 2^8
        for i in range(4):
            h = ((h ^ (v >> 8 * i & 0xFF)) * 1099511628211) % 2**64
    return h


def test_choices_belong_to_their_kernels(cuda, tmp_path):
    (tmp_path / "tempi_b200_batch_tune.txt").write_text(
        f"{before(2, 3):x} 128 1" + " 4" * 40 + "\n")
    # a fresh process reads the file
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = ("import sys; sys.path.insert(0, %r)\n"
            "from tests import test_tune_signature_gpu as T\n"
            "T.fresh_process()\n" % root)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, TEMPI_CACHE_DIR=str(tmp_path)))
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr


def fresh_process():
    import torch

    from tempi_b200 import mpi

    assert mpi.Init() == 0
    lib = _lib.tempi()
    src_np = H.splitmix_bytes(1 << 16, 5)
    src = torch.from_numpy(src_np).cuda()
    out = torch.zeros(1 << 16, dtype=torch.uint8, device="cuda")

    def batch(dims):
        d = layout(dims)
        regs = [(k * (d.extent + 64), d, k * d.size) for k in range(3)]
        h = launch(regs, src.data_ptr(), out.data_ptr(), 0)
        torch.cuda.synchronize()
        for off, _, at in regs:
            want = desc_pack(d, src_np[off:], 1).tobytes()
            assert out[at: at + d.size].cpu().numpy().tobytes() == want
        return h

    two, three = batch(2), batch(3)
    # neither kernel takes the line of the file
    assert config(two) == (256, 0, 1) and config(three) == (256, 0, 1)
    # nor one kernel the choices of the other
    _lib.check(lib.tempi_batch_tune(three, None, 3))
    chosen = config(three)
    assert config(batch(2)) == (256, 0, 1)
    assert config(batch(3)) == chosen
    print("OK")
