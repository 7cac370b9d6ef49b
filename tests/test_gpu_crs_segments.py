"""The seeded sampler writes in place and shifts only what a rejection moves: sizes
around one 2048-sample segment, rejections so rare that the first segments stay
in place, and an output buffer without 16-byte alignment. Word for word."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = 4294966657


def _host(t):
    return t.cpu().numpy().view(np.uint32).reshape(-1)


@pytest.mark.parametrize("npolys", [31, 32, 33, 64, 2049])
@pytest.mark.parametrize("accept_max", [0, (1 << 64) - (1 << 51), (1 << 64) - (1 << 56)])
def test_segments(cuda, oracle, npolys, accept_max):
    """About one sample in 8192, and one in 256, rejected by a lowered threshold."""
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.labrador import sample_uniform_polys
    plan = TwistedNttPlan(Q, 64)
    seed = bytes((npolys + 9 * i) & 0xFF for i in range(32))
    want = oracle.sample_uniform_polys(oracle.Field(Q), seed, npolys, 64, accept_max=accept_max)
    got = sample_uniform_polys(plan, seed, npolys, device=cuda, accept_max=accept_max)
    plan.check_device()
    assert np.array_equal(_host(got), want)


@pytest.mark.parametrize("shift", [1, 2])
def test_unaligned_output(cuda, oracle, shift):
    import torch
    from lattica_b200 import TwistedNttPlan, _lib
    plan, lib = TwistedNttPlan(Q, 64), _lib.load()
    npolys, seed = 65, bytes(range(32))
    nb = C.c_size_t()
    lib.grid_gpu_sample_uniform_polys_workspace(plan.handle, npolys, 0, C.byref(nb))
    ws = torch.empty(nb.value, dtype=torch.uint8, device=cuda)
    buf = torch.full((npolys * 64 + 8,), -1, dtype=torch.int32, device=cuda)
    sd = (C.c_uint8 * 32).from_buffer_copy(seed)
    st = lib.grid_gpu_sample_uniform_polys_dev(plan.handle, sd, npolys, 0,
                                               buf.data_ptr() + 4 * shift, ws.data_ptr(),
                                               ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert st == 0
    got = _host(buf)
    assert np.array_equal(got[shift:shift + npolys * 64],
                          oracle.sample_uniform_polys(oracle.Field(Q), seed, npolys, 64))
    assert (got[:shift] == 0xFFFFFFFF).all() and (got[shift + npolys * 64:] == 0xFFFFFFFF).all()
