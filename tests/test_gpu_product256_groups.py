"""d = 256 products in two groups of warps per CTA: tile counts around one, two and three
per CTA, words at both ends of the range, both operands the same tensor, against the
oracle."""
import numpy as np
import pytest

Q256 = 4294962689

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [Q256, 12289])
@pytest.mark.parametrize("tiles,ragged", [(0, 2), (1, 0), (148, 31), (2 * 148, 1), (3 * 148 - 1, 0)])
def test_product_matches_oracle(cuda, oracle, q, tiles, ragged):
    import torch
    from lattica_b200 import TwistedNttPlan
    n = 32 * tiles + ragged
    rng = np.random.default_rng(n + q % 97)
    a = rng.integers(0, q, (n, 256), dtype=np.uint64).astype(np.uint32)
    a[::3], a[1::5, ::2] = q - 1, 0
    plan, P = TwistedNttPlan(q, 256), oracle.Plan(q, 256)
    ta = torch.from_numpy(a.view(np.int32)).to(cuda)
    got = plan.ntt_mul_inverse(ta, ta).cpu().numpy().view(np.uint32)
    idx = np.unique(np.r_[0, n - 1, np.linspace(0, n - 1, 60).astype(int)])
    assert np.array_equal(got[idx], P.ntt_mul_inverse(a[idx], a[idx]).reshape(-1, 256))
    plan.check_device()
