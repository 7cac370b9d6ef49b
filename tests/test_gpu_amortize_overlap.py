"""The amortized witness written over its own inputs: z over the rows of s (in place, or
shifted against them) and over c, where one launch would store while it still reads."""
import ctypes as C

import numpy as np
import pytest

Q, Q_RING, D = 4294966657, 4294967291, 64

pytestmark = pytest.mark.gpu


# 150 tiles of 128 polys: no split of the sum, and CTAs that start after others have stored
@pytest.mark.parametrize("q,r,n", [(Q, 3, 19190), (Q, 2, 300), (Q_RING, 2, 150)])
@pytest.mark.parametrize("z_at", [0, 64, -200, "c"])
def test_output_over_inputs(cuda, oracle, q, r, n, z_at):
    import torch
    from lattica_b200 import TwistedNttPlan, _lib
    from lattica_b200.ntt import RingPlan
    lib = _lib.load()
    rng = np.random.default_rng(r + n)
    S = rng.integers(0, q, (r, n, D), dtype=np.uint64).astype(np.uint32)
    c = rng.integers(0, q, (r, D), dtype=np.uint64).astype(np.uint32)
    if q == Q:
        plan, want = TwistedNttPlan(q, D), oracle.Plan(q, D).amortize(S, c, r, n)
    else:
        plan, want = RingPlan(q, D), oracle.Field(q).ring_amortize(D, S, c, r, n)
    want = want.reshape(n, D)
    pad = 256  # polys before s, and after it
    buf = torch.zeros((pad + r * n + pad + n + r, D), dtype=torch.int32, device=cuda)
    s_at, c_at = pad, pad + r * n + pad
    buf[s_at:s_at + r * n] = torch.from_numpy(S.reshape(-1, D).view(np.int32)).to(cuda)
    buf[c_at:c_at + r] = torch.from_numpy(c.view(np.int32)).to(cuda)
    at = c_at if z_at == "c" else s_at + z_at
    ptr = lambda poly: buf.data_ptr() + poly * D * 4
    nb = C.c_size_t()
    assert lib.grid_gpu_amortize_workspace(plan.handle, r, n, C.byref(nb)) == 0
    ws = torch.empty(nb.value, dtype=torch.uint8, device=cuda)
    assert lib.grid_gpu_amortize_dev(plan.handle, ptr(s_at), ptr(c_at), r, n, ptr(at),
                                     ws.data_ptr(), ws.numel(),
                                     torch.cuda.current_stream().cuda_stream) == 0
    assert np.array_equal(buf[at:at + n].cpu().numpy().view(np.uint32), want)
    plan.check_device()
