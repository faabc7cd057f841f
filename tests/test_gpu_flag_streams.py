"""Flag fields in device memory that the default stream is still writing when
a solver on a non-blocking stream of its own is given them: every call waits
for them. (The delay is a kernel that spins for a bounded number of cycles.)"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (24, 18, 6)
DELAY = 50_000_000   # cycles, about 25 ms


@pytest.fixture(scope="module")
def fc(built_lib):
    import foil_cfd_gb300 as fc
    return fc


@pytest.fixture(scope="module")
def torch():
    import torch
    assert torch.cuda.is_available()
    return torch


def fields():
    rng = np.random.default_rng(7)
    n = int(np.prod(DIMS))
    return [(rng.random(n) < p).astype(np.uint8) for p in (0.05, 0.2)]


def late(torch, now, then):
    """A device field that holds `now` and will hold `then` once the default
    stream gets to it."""
    t, source = torch.from_numpy(now).cuda(), torch.from_numpy(then).cuda()
    torch.cuda.synchronize()
    torch.cuda._sleep(DELAY)
    t.copy_(source)
    return t


class Bytes:
    """n bytes of device memory at an address, for torch.as_tensor."""

    def __init__(self, address, n):
        self.__cuda_array_interface__ = {"data": (address, False), "shape": (n,), "typestr": "|u1", "version": 2}


@pytest.mark.parametrize("call", ["init", "set_flags", "apply_edited_flags"])
def test_fields_under_way_in_the_default_stream(fc, torch, call):
    a, b = fields()
    stream = torch.cuda.Stream()
    s = fc.LBMSolver()
    arg = late(torch, a, b) if call == "init" else a
    s.init(DIMS, fc.scaling_direct(0.55, 0.03), arg, stream=C.c_void_p(stream.cuda_stream), les_cs=0.1)
    if call == "set_flags":
        assert s.set_flags(late(torch, a, b)) == 0
    elif call == "apply_edited_flags":
        assert s.apply_edited_flags(late(torch, a, b)) == int((a != b).sum())
    s.synchronize()
    assert np.array_equal(torch.as_tensor(Bytes(s.device_flags(), b.size), device="cuda").cpu().numpy(), b)
    ref = fc.LBMSolver()
    ref.init(DIMS, fc.scaling_direct(0.55, 0.03), b if call == "init" else a, les_cs=0.1)
    if call == "set_flags":
        ref.set_flags(b)
    elif call == "apply_edited_flags":
        ref.apply_edited_flags(b)
    for x in (s, ref):
        assert x.step_n(4) == 0
        x.synchronize()
    keep = b == 0
    assert np.array_equal(s.export_f32().reshape(19, -1)[:, keep], ref.export_f32().reshape(19, -1)[:, keep])
