"""Where the dispatcher picks the staged kernels, the word kernel runs below
16 MB of 4-byte and wider words in device memory (8 MB of 8-byte and wider ones
for rows below 64 B): both sides of each line, the widths it holds for and ones
it does not, and the staged kernel where a caller asks for it by number."""
import ctypes

import pytest

from tempi_b200 import _lib

from . import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mine", [True, False])
@pytest.mark.parametrize("block,rows,gap,words", [
    (16, 499_999, 32, True), (16, 500_000, 32, False), (60, 66_668, 4, False),
    (56, 71_428, 8, True),
    (64, 249_999, 64, True), (64, 250_000, 64, False), (4096, 3, 16, True),
    (8_000_008, 1, 0, True), (15_999_984, 1, 0, True), (16_000_000, 1, 0, False),
    (72, 27_776, 56, True), (254, 8_000, 2, False),
])
def test_staged_unpack_line(cuda, mpi_init, mine, block, rows, gap, words):
    import torch

    lib = _lib.tempi()
    nbytes = rows * (block + gap)
    d = _lib.Desc.make(0, nbytes, block, [rows], [block + gap])
    src = torch.from_numpy(H.splitmix_bytes(d.size, block)).cuda()
    back = torch.full((nbytes,), 0xAA, dtype=torch.uint8, device="cuda")
    cfg = _lib.Config(4, 0, 256, 0, 3, _lib.OWN_CHOICE if mine else 0)
    # the first staged launch of a process may come before its failure word
    _lib.check(lib.tempi_unpack(ctypes.byref(d), src.data_ptr(), 1, back.data_ptr(),
                                ctypes.byref(cfg), None))
    torch.cuda.synchronize()
    name = lib.tempi_last_kernel().decode()
    if mine and words:
        assert name.startswith("words_unpack")
    elif block != 254:  # odd rows: the realign kernel may take the dispatcher's pick
        assert name.startswith("staged_unpack" if d.size % 16 == 0 else "")
    exp = torch.full((rows, block + gap), 0xAA, dtype=torch.uint8, device="cuda")
    exp[:, :block] = src.view(rows, block)
    assert torch.equal(back, exp.view(-1))
    packed = torch.full((d.size + 16,), 0x5A, dtype=torch.uint8, device="cuda")
    _lib.check(lib.tempi_pack(ctypes.byref(d), back.data_ptr(), 1, packed.data_ptr(),
                              ctypes.byref(cfg), None))
    torch.cuda.synchronize()
    if mine and words and block % 16 == 0:
        assert lib.tempi_last_kernel().decode() == "words_pack_w16"
    assert torch.equal(packed[: d.size], src)
    assert bool((packed[d.size:] == 0x5A).all())
    _lib.check(lib.tempi_staged_check())
