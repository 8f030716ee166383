"""The realign kernel at the largest objects the library accepts (2^31 - 1
packed bytes): its index arithmetic on the CPU against 64 bits, then long odd
runs and rows of that size on the GPU, with guard bytes around both sides."""
import ctypes
import os
import subprocess

import pytest

from tempi_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MOST = 2**31 - 1


def test_index_arithmetic(tmp_path):
    exe = tmp_path / "realign_index"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=signed-integer-overflow",
                    "-fno-sanitize-recover", "-o", str(exe),
                    os.path.join(ROOT, "tests", "c", "realign_index.cpp"),
                    "-I" + os.path.join(ROOT, "tempi_b200", "csrc", "tempi")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "OK\n", r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("words", [0, 1, 4])  # 0: the library's own choice
@pytest.mark.parametrize("nbytes,start,pmis", [
    (MOST, 1, 0), (MOST, 0, 15), (MOST, 15, 3), (MOST - 7, 3, 0), (MOST - 15, 2, 1),
])
def test_long_runs(cuda, mpi_init, nbytes, start, pmis, words):
    import torch

    lib, guard = _lib.tempi(), 64
    gen = torch.Generator(device="cuda").manual_seed(nbytes % 1000 + pmis)
    src = torch.randint(0, 256, (nbytes + start + guard,), dtype=torch.uint8, device="cuda",
                        generator=gen)
    d = _lib.Desc.make(start, nbytes + start, nbytes, [], [])
    cfg = ctypes.byref(_lib.Config(5, 0, 0, words, 0, 0)) if words else None
    packed = torch.full((nbytes + pmis + guard,), 0x5A, dtype=torch.uint8, device="cuda")
    _lib.check(lib.tempi_pack(ctypes.byref(d), src.data_ptr(), 1, packed.data_ptr() + pmis, cfg,
                              None))
    assert lib.tempi_last_kernel() == b"realign_pack"
    torch.cuda.synchronize()
    assert torch.equal(packed[pmis: pmis + nbytes], src[start: start + nbytes])
    assert bool((packed[:pmis] == 0x5A).all()) and bool((packed[pmis + nbytes:] == 0x5A).all())
    back = torch.full_like(src, 0xAA)
    _lib.check(lib.tempi_unpack(ctypes.byref(d), packed.data_ptr() + pmis, 1, back.data_ptr(),
                                cfg, None))
    assert lib.tempi_last_kernel() == b"realign_unpack"
    torch.cuda.synchronize()
    assert torch.equal(back[start: start + nbytes], src[start: start + nbytes])
    assert bool((back[:start] == 0xAA).all()) and bool((back[start + nbytes:] == 0xAA).all())


@pytest.mark.gpu
@pytest.mark.parametrize("rows,block", [(2, 2**30 - 1), (3, 715_827_881), (134_000_001, 16)])
def test_large_rows(cuda, mpi_init, rows, block):
    """Rows whose last bytes lie just below 2^31 packed bytes."""
    import torch

    lib, gap = _lib.tempi(), 5
    assert rows * block <= MOST
    gen = torch.Generator(device="cuda").manual_seed(rows)
    src = torch.randint(0, 256, (rows * (block + gap),), dtype=torch.uint8, device="cuda",
                        generator=gen)
    d = _lib.Desc.make(0, src.numel(), block, [rows], [block + gap])
    cfg = ctypes.byref(_lib.Config(5, 0, 0, 0, 0, 0))
    packed = torch.full((rows * block + 64,), 0x5A, dtype=torch.uint8, device="cuda")
    _lib.check(lib.tempi_pack(ctypes.byref(d), src.data_ptr(), 1, packed.data_ptr(), cfg, None))
    assert lib.tempi_last_kernel() == b"realign_pack"
    torch.cuda.synchronize()
    want = src.view(rows, block + gap)[:, :block]
    assert torch.equal(packed[: rows * block].view(rows, block), want)
    assert bool((packed[rows * block:] == 0x5A).all())
    back = torch.full_like(src, 0xAA)
    _lib.check(lib.tempi_unpack(ctypes.byref(d), packed.data_ptr(), 1, back.data_ptr(), cfg,
                                None))
    assert lib.tempi_last_kernel() == b"realign_unpack"
    torch.cuda.synchronize()
    got = back.view(rows, block + gap)
    assert torch.equal(got[:, :block], want) and bool((got[:, block:] == 0xAA).all())
