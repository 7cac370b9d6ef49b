"""JL projection, entries and evaluations of more columns than one CTA per SM may accumulate
(148 x 2040 units of 32 columns): several waves of CTAs add up to the oracle's words."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q, D, PARTS, N = 4294966657, 64, 64, 2400  # 9,830,400 columns


def test_more_than_one_wave(cuda, oracle):
    import torch
    from lattica_b200 import TwistedNttPlan, _lib
    lib, plan, F = _lib.load(), TwistedNttPlan(Q, D), oracle.Field(Q)
    rng = np.random.default_rng(24)
    x = rng.integers(0, Q, (PARTS, N * D), dtype=np.uint64).astype(np.uint32)
    x[:, ::3] = Q - 1
    seed = bytes((7 * i) & 0xFF for i in range(32))
    sd = (C.c_uint8 * 32).from_buffer_copy(seed)
    st = torch.cuda.current_stream().cuda_stream
    dx = torch.from_numpy(x.view(np.int32)).to(cuda)
    ws = torch.empty(1 << 20, dtype=torch.uint8, device=cuda)
    want, _ = oracle.jl_project(F, seed, 256, x, PARTS, N * D, D, want_flat=False)

    p = torch.zeros(256, dtype=torch.int32, device=cuda)
    flat = torch.empty((256, PARTS, D, N), dtype=torch.int8, device=cuda)
    for entries in (None, flat.data_ptr()):
        p.zero_()
        assert lib.grid_gpu_jl_project_dev(plan.handle, sd, 256, dx.data_ptr(), PARTS, N * D, D,
                                           p.data_ptr(), entries, ws.data_ptr(), ws.numel(),
                                           st) == 0
        assert np.array_equal(p.cpu().numpy().view(np.uint32), want)
    words = (dx.to(torch.int64) & 0xFFFFFFFF).reshape(PARTS, N, D).transpose(1, 2)
    for row in (0, 137, 255):  # the entries themselves give the row's sum
        assert int((words * flat[row]).sum()) % Q == int(want[row])

    ev = torch.empty((256, D), dtype=torch.int32, device=cuda)
    assert lib.grid_gpu_jl_evals_dev(plan.handle, sd, 256, dx.data_ptr(), PARTS, N * D, D,
                                     ev.data_ptr(), ws.data_ptr(), ws.numel(), st) == 0
    got = ev.cpu().numpy().view(np.uint32)
    assert np.array_equal(got[:, 0], want)
    ext = np.concatenate([x.reshape(-1, D), (Q - x.reshape(-1, D).astype(np.uint64)) % Q], axis=1)
    rot = np.ascontiguousarray(ext[:, 5:5 + D].astype(np.uint32).reshape(PARTS, N * D))
    want5, _ = oracle.jl_project(F, seed, 256, rot, PARTS, N * D, D, want_flat=False)
    assert np.array_equal(got[:, 5], want5)
    plan.check_device()
