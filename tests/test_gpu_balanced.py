"""Balanced limbs in 32-bit arithmetic: powers of two from 2 to 2^32, other bases,
carries that run past the magnitude, the limbs a half base away from zero, buffers
that take the four-word path and ones that do not; and the prover round's fused
limbs against the separate pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = 4294966657


def _dev(x, cuda):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).to(cuda)


def _edge_words(q, n, base):
    """Montgomery words of values around multiples of base / 2, q / 2 and zero."""
    half = base // 2
    vals = [0, 1, q - 1, q // 2, q // 2 + 1, q // 2 - 1]
    for m in (1, 2, 3, 255, 256, 257):
        for e in (-1, 0, 1):
            vals += [m * half + e, -(m * half + e)]
    rng = np.random.default_rng(base % 1000)
    vals += [int(v) for v in rng.integers(0, q, n - len(vals))]
    return np.array([(v % q) * (1 << 32) % q for v in vals[:n]], dtype=np.uint64).astype(np.uint32)


@pytest.mark.parametrize("q", [Q, 12289])
@pytest.mark.parametrize("base,limbs", [(2, 33), (4, 16), (256, 4), (1 << 16, 2), (1 << 31, 2),
                                        (1 << 32, 2), (3, 21), (10, 10), (257, 4),
                                        (4294967295, 1), (2147483647, 3), (256, 1)])
def test_limbs_match_oracle(cuda, oracle, q, base, limbs):
    import torch
    from lattica_b200 import TwistedNttPlan, _lib
    plan, F, lib = TwistedNttPlan(q, 64), oracle.Field(q), _lib.load()
    polys = _edge_words(q, 64 * 5, base)
    want = oracle.decompose_polys(F, 64, polys, base, limbs)
    for shift in (0, 1):  # 16-byte aligned, and not
        src = torch.empty(64 * 5 + 4, dtype=torch.int32, device=cuda)
        src[shift:shift + 64 * 5] = _dev(polys, cuda)
        out = torch.zeros(64 * 5 * limbs + 4, dtype=torch.int32, device=cuda)
        st = lib.grid_gpu_decompose_balanced_dev(plan.handle, src.data_ptr() + 4 * shift, 5, base,
                                                 limbs, out.data_ptr() + 4 * shift,
                                                 torch.cuda.current_stream().cuda_stream)
        assert st == 0
        got = out.cpu().numpy().view(np.uint32)[shift:shift + 64 * 5 * limbs]
        assert np.array_equal(got, want.reshape(-1))


@pytest.mark.parametrize("ring", [False, True])
@pytest.mark.parametrize("base,limbs", [(256, 4), (10, 10)])
def test_round_limbs_equal_the_separate_pass(cuda, oracle, ring, base, limbs):
    import torch
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.labrador import CommitKey, prover_round_dev
    from lattica_b200.ntt import RingPlan
    q = 4294967291 if ring else Q
    plan = RingPlan(q, 64) if ring else TwistedNttPlan(q, 64)
    F = oracle.Field(q)
    r, n, kappa = 9, 131, 5
    g = torch.Generator(device=cuda).manual_seed(base)
    word = lambda *s: torch.randint(0, q, s, dtype=torch.int64, device=cuda,
                                    generator=g).to(torch.int32)
    S, key = word(r, n, 64), CommitKey(plan, word(kappa, n, 64), kappa, n)
    out = prover_round_dev(key, S, base, limbs, base, limbs, None)
    host = lambda t: t.cpu().numpy().view(np.uint32).reshape(-1)
    t = host(key.inner_commit_slice(S))
    assert np.array_equal(host(out.t_limbs), oracle.decompose_polys(F, 64, t, base, limbs).reshape(-1))
    assert np.array_equal(host(out.g_limbs),
                          oracle.decompose_polys(F, 64, host(out.g), base, limbs).reshape(-1))
    plan.check_device()
