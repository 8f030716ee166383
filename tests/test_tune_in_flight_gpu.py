"""tempi_batch_tune while a launch of the same batch is still queued on another
stream: that launch keeps the table and the chunk count it was issued with
(the tuner rewrites both for every plan it tries, so it waits first)."""
import pytest

from tempi_b200 import _lib, halo

from . import helpers as H
from .test_batch_gpu import oracle_pack, oracle_unpack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["pack", "exchange"])
def test_tune_waits_for_launches_of_the_batch(cuda, mpi_init, kind, tmp_path, monkeypatch):
    import torch

    monkeypatch.setenv("TEMPI_CACHE_DIR", str(tmp_path))
    _lib.tempi().tempi_reload_env()
    g = halo.Grid((46, 39, 21), 2)
    data_np = H.splitmix_bytes(g.nbytes, 17)
    data = torch.from_numpy(data_np).cuda()
    packed = torch.zeros(g.packed_bytes, dtype=torch.uint8, device="cuda")
    if kind == "pack":
        b = halo.HaloBatch([g], [data.data_ptr()], [packed.data_ptr()])
        out, want = packed, oracle_pack(g, data_np)
    else:
        b = halo.HaloExchange([g], [data.data_ptr()])
        out, want = data, oracle_unpack(g, oracle_pack(g, data_np), data_np)
    torch.cuda.synchronize()
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(2):  # the second time with the choices of the first
        with torch.cuda.stream(first):
            torch.cuda._sleep(100_000_000)
            b.launch(first.cuda_stream)
            got = out.clone()
        b.tune(second.cuda_stream, 1)
        torch.cuda.synchronize()
        assert got.cpu().numpy().tobytes() == want.tobytes()
        assert out.cpu().numpy().tobytes() == want.tobytes()
        if kind == "pack":
            packed.zero_()
            torch.cuda.synchronize()
    b.close()
    monkeypatch.undo()
    _lib.tempi().tempi_reload_env()
