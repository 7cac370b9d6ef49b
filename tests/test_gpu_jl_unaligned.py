"""The int8 entries go to any address: buffers that do not start on a 4-byte word are written
byte by byte."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = 4294966657


@pytest.mark.parametrize("rows", [256, 200])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_entries_at_any_address(cuda, oracle, rows, shift):
    import torch
    from lattica_b200 import TwistedNttPlan, _lib
    lib, d, parts, n = _lib.load(), 8, 2, 132
    plan, F = TwistedNttPlan(Q, d), oracle.Field(Q)
    seed = bytes((i * 13 + rows) & 0xFF for i in range(32))
    x = np.random.default_rng(rows).integers(0, Q, (parts, n * d), dtype=np.uint64).astype(np.uint32)
    want, flat = oracle.jl_project(F, seed, rows, x, parts, n * d, d)
    dx = torch.from_numpy(x.view(np.int32)).to(cuda)
    size = rows * parts * n * d
    out = torch.full((size + 8,), 7, dtype=torch.int8, device=cuda)
    p = torch.empty(rows, dtype=torch.int32, device=cuda)
    ws = torch.empty(1 << 16, dtype=torch.uint8, device=cuda)
    sd = (C.c_uint8 * 32).from_buffer_copy(seed)
    assert lib.grid_gpu_jl_project_dev(plan.handle, sd, rows, dx.data_ptr(), parts, n * d, d,
                                       p.data_ptr(), out.data_ptr() + shift, ws.data_ptr(),
                                       ws.numel(), torch.cuda.current_stream().cuda_stream) == 0
    got = out.cpu().numpy()
    assert np.array_equal(got[shift:shift + size], flat.reshape(-1))
    assert (got[:shift] == 7).all() and (got[shift + size:] == 7).all()
    assert np.array_equal(p.cpu().numpy().view(np.uint32), want)
    plan.check_device()
