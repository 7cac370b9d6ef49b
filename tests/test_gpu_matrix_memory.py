"""A matrix whose evaluations fit the device's memory once, but not with the point-major
copy beside them, is prepared without the copy, and its products are the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = 4294966657
ROWS, COLS = 16, 65537  # 268 MB of evaluations


@pytest.mark.parametrize("ring", [False, True])
def test_prepared_without_the_copy(cuda, ring):
    import torch
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.commit import PreparedMatrix
    from lattica_b200.labrador import CommitKey, prover_round_dev
    from lattica_b200.ntt import RingPlan
    q = 4294967291 if ring else Q
    plan = RingPlan(q, 64) if ring else TwistedNttPlan(q, 64)
    g = torch.Generator(device=cuda).manual_seed(3)
    word = lambda *s: torch.randint(0, q, s, dtype=torch.int64, device=cuda,
                                    generator=g).to(torch.int32)
    A, s = word(ROWS, COLS, 64), word(6, COLS, 64)
    whole = CommitKey(plan, A, ROWS, COLS)
    want = whole.a.mul_vec(s)
    out = prover_round_dev(whole, s, 256, 4, 256, 4, None)
    rounds = [out.t_limbs, out.g, out.g_limbs]
    del whole, out
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    copies = 3 if ring else 1  # one per auxiliary prime
    one = ROWS * COLS * 256
    filler = torch.empty(free - (copies * 2 - 1) * one - one // 2, dtype=torch.uint8, device=cuda)
    key = CommitKey(plan, A, ROWS, COLS)
    del filler
    torch.cuda.empty_cache()
    assert torch.equal(key.a.mul_vec(s), want)
    out = prover_round_dev(key, s, 256, 4, 256, 4, None)
    assert all(torch.equal(x, y) for x, y in zip((out.t_limbs, out.g, out.g_limbs), rounds))
    plan.check_device()
