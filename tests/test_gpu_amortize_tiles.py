"""The amortized witness without transforms: tiles of 128 polys and their edges, splits of
the sum over i, more than 64 terms, words at both ends of their range, against the oracle."""
import numpy as np
import pytest

Q, D = 4294966657, 64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [Q, 12289])
@pytest.mark.parametrize("r,n", [(1, 1), (2, 127), (5, 128), (7, 129), (65, 3), (9, 300), (130, 20),
                                 (149, 2), (2, 19001)])
def test_amortize_matches_oracle(cuda, oracle, q, r, n):
    import torch
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.labrador import amortize_witness
    rng = np.random.default_rng(r * 1000 + n)
    S = rng.integers(0, q, (r, n, D), dtype=np.uint64).astype(np.uint32)
    c = rng.integers(0, q, (r, D), dtype=np.uint64).astype(np.uint32)
    S[:, ::3], c[0] = q - 1, q - 1
    c[-1, ::2] = 0
    plan = TwistedNttPlan(q, D)
    want = oracle.Plan(q, D).amortize(S, c, r, n).reshape(n, D)
    dS, dc = (torch.from_numpy(x.view(np.int32)).to(cuda) for x in (S, c))
    got = amortize_witness(plan, dS, dc).cpu().numpy().view(np.uint32)
    assert np.array_equal(got, want)
    plan.check_device()
