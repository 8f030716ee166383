"""A measurement at run time (TEMPI_DISPATCH=exhaustive, or an ensemble that
disagrees) times the kernels that the candidates name, also where a rule puts
another kernel in the place of the cost model's pick, and the fixed rules
beside them; so it can find for the rule and against it."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from tempi_b200 import _lib, dispatch_train as DT, mpi

from . import helpers as H

pytestmark = pytest.mark.gpu

LONG = 60_000_001  # one run at an odd offset: words of a byte, or realigned


def times(d, what):
    t = (ctypes.c_float * DT.N_MEAS)()
    _lib.check(_lib.tempi().tempi_measure(ctypes.byref(d), 1, 0, 0, what, 3, t))
    return np.frombuffer(t, np.float32)


def test_named_kernels_are_timed(cuda, mpi_init):
    """The word kernel packs this run in 44 us beyond the call's cost, the
    realign kernel that the rule prefers in 20."""
    d = _lib.Desc.make(3, LONG + 3, LONG, [], [])
    t = times(d, 1 | 4)
    assert t[DT.PACK] > 1.3 * t[DT.FIXED_PACK]
    assert t[DT.UNPACK] > 1.3 * t[DT.FIXED_UNPACK]
    t = times(d, 1)  # what the cost model's pick would launch
    assert t[DT.PACK] < 1.3 * t[DT.FIXED_PACK]


@pytest.mark.parametrize("policy", ["exhaustive", "learned"])
def test_exhaustive_keeps_the_faster_rule(cuda, policy):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = ("import sys; sys.path.insert(0, %r)\n"
            "from tests import test_measured_kernels_gpu as T\n"
            "T.fresh_process(%r)\n" % (root, policy))
    # a spread limit of zero: the learned policy measures every layout
    env = dict(os.environ, TEMPI_DISPATCH=policy, TEMPI_DISPATCH_SPREAD="0")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=env)
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr


def fresh_process(policy):
    import torch

    assert mpi.Init() == 0
    lib = _lib.tempi()
    for block, rows, gap, realigned in ((LONG, 1, 0, True), (64, 4096, 64, False),
                                        (201, 40_000, 202, None)):
        t = mpi.Type_vector(rows, block, block + gap, mpi.BYTE)
        n = _lib.counter("dispatch_measured")
        assert mpi.Type_commit(t) == 0
        span = rows * (block + gap)
        src = torch.from_numpy(H.splitmix_bytes(span + 3, rows)).cuda()[3:]
        want = src.view(rows, block + gap)[:, :block].reshape(-1)
        packed = torch.zeros(rows * block, dtype=torch.uint8, device="cuda")
        back = torch.full_like(src, 0xAA)
        torch.cuda.synchronize()
        assert mpi.Pack(src.data_ptr(), 1, t, packed.data_ptr(), rows * block)[0] == 0
        name = lib.tempi_last_kernel().decode()
        assert _lib.counter("dispatch_measured") > n
        assert torch.equal(packed, want)
        if realigned is not None:
            assert name.startswith("realign") == realigned, name
        assert mpi.Unpack(packed.data_ptr(), rows * block, back.data_ptr(), 1, t)[0] == 0
        exp = torch.full_like(src, 0xAA).view(rows, block + gap)
        exp[:, :block] = packed.view(rows, block)
        assert torch.equal(back.view(rows, block + gap), exp)
    print("OK")
