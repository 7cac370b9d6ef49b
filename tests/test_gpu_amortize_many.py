"""The amortized witness of thousands of vectors: more splits of the sum than SMs, and a
split that ends with a single term, against the oracle."""
import numpy as np
import pytest

Q, D = 4294966657, 64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r,n", [(4096, 3), (4097, 1), (5000, 10), (9473, 129)])
def test_amortize_matches_oracle(cuda, oracle, r, n):
    import torch
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.labrador import amortize_witness
    rng = np.random.default_rng(r + n)
    S = rng.integers(0, Q, (r, n, D), dtype=np.uint64).astype(np.uint32)
    c = rng.integers(0, Q, (r, D), dtype=np.uint64).astype(np.uint32)
    S[::2], c[::5] = Q - 1, Q - 1
    plan = TwistedNttPlan(Q, D)
    want = oracle.Plan(Q, D).amortize(S, c, r, n).reshape(n, D)
    dS, dc = (torch.from_numpy(x.view(np.int32)).to(cuda) for x in (S, c))
    assert np.array_equal(amortize_witness(plan, dS, dc).cpu().numpy().view(np.uint32), want)
    plan.check_device()
