"""Grouped point-major products over blocks of 128 columns: lengths at the edges of blocks
and chunks, live counts beside the loads' boxes of 8 to 64 rows, K ranges that start inside
a block, gaps between the witnesses, against the oracle."""
import numpy as np
import pytest

Q, D = 4294966657, 64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths,ranks,k_split", [
    ([1], (1,), 32), ([128] * 9, (16,), 64), ([127, 128, 129, 31, 32, 33, 1], (8, 17), 96),
    ([300] * 63 + [129] * 2 + [257], (32,), 160), (list(range(1, 131)), (5,), 1024),
    ([385] * 121 + [96] * 8 + [2], (12, 31), 224)])
def test_blocks_match_the_oracle(cuda, oracle, lengths, ranks, k_split):
    import torch
    from lattica_b200 import TwistedNttPlan, _lib
    from lattica_b200.batch import UnevenCommitBatch
    from lattica_b200.commit import PreparedMatrix
    rng = np.random.default_rng(len(lengths))
    cols = max(lengths) + (-max(lengths)) % 4
    plan = TwistedNttPlan(Q, D)
    mats_host = [rng.integers(0, Q, (r, cols, D), dtype=np.uint64).astype(np.uint32) for r in ranks]
    mats = [PreparedMatrix(plan, A, A.shape[0], cols) for A in mats_host]
    items, so, to = [], 3, 0
    for i, n in enumerate(rng.permutation(lengths)):
        m = i % len(ranks)
        items.append((so, to, int(n), m))
        so += int(n) + (i % 3) * 70   # gaps: the packed buffer may exceed the padded blocks
        to += ranks[m]
    s_polys = max(a + n for a, _, n, _ in items)
    s_host = rng.integers(0, Q, (s_polys, D), dtype=np.uint64).astype(np.uint32)
    s_host[0:s_polys:5] = Q - 1
    s = torch.from_numpy(s_host.view(np.int32)).to(cuda)
    want = np.zeros((to, D), np.uint32)
    P = oracle.Plan(Q, D)
    for a, b, n, m in items:
        A = np.ascontiguousarray(mats_host[m][:, :n, :])
        want[b:b + ranks[m]] = P.matvec(A, ranks[m], n, s_host[a:a + n], 1).reshape(ranks[m], D)
    batch = UnevenCommitBatch(plan, mats, items)
    batch.set_config(k_split, 0, _lib.ENGINE_POINT_MAJOR)
    t = torch.full((to, D), -1, dtype=torch.int32, device=cuda)
    batch.commit_dev(s, t)
    torch.cuda.synchronize()
    assert np.array_equal(t.cpu().numpy().view(np.uint32), want)
