"""Ring plans transform their input words as they are: words between an auxiliary
prime and q (not reduced mod the prime) through every engine a transform can take,
point-major and gathering products, both CUDA-core fallbacks. Words equal the
oracle's schoolbook products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = 4294967291  # 2^32 - 5
AUX = (4294962689, 4294957057, 4294955009)


def _words(shape, seed):
    """Words around the auxiliary primes and up to q - 1, a quarter of them uniform."""
    rng = np.random.default_rng(seed)
    edge = np.array([p + e for p in AUX for e in (-1, 0, 1)] + [Q - 1, Q - 2], dtype=np.uint64)
    x = edge[rng.integers(0, edge.size, shape)]
    uni = rng.integers(0, Q, shape, dtype=np.uint64)
    return np.where(rng.integers(0, 4, shape) == 0, uni, x).astype(np.uint32)


def _dev(x, cuda):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).to(cuda)


def _host(t):
    return t.cpu().numpy().view(np.uint32)


# (r, n): K a multiple of 4 takes the point-major products, 37 the gathering ones,
# 65 rows the CUDA-core products
@pytest.mark.parametrize("engine", ["default", "cuda_core"])
@pytest.mark.parametrize("r,n", [(4, 8), (33, 36), (6, 37), (65, 4)])
def test_products_of_unreduced_words(cuda, oracle, monkeypatch, engine, r, n):
    from lattica_b200.commit import PreparedMatrix
    from lattica_b200.labrador import amortize_witness, compute_garbage_g, compute_garbage_h
    from lattica_b200.ntt import RingPlan
    if engine != "default":
        monkeypatch.setenv("GRID_GPU_NTT_ENGINE", engine)
    d = 64
    plan, F = RingPlan(Q, d), oracle.Field(Q)
    S, Phi, c = _words((r, n, d), r + n), _words((r, n, d), r * n), _words((r, d), 3)
    A = _words((5, n, d), 4)
    dS, dPhi = _dev(S, cuda), _dev(Phi, cuda)
    M = PreparedMatrix(plan, _dev(A, cuda), 5, n)
    assert np.array_equal(_host(M.mul_vec(dS)).reshape(-1),
                          F.ring_matvec(d, A, 5, n, S, r).reshape(-1))
    assert np.array_equal(_host(compute_garbage_g(plan, dS)).reshape(-1), F.ring_gram(d, S, r, n))
    assert np.array_equal(_host(compute_garbage_h(plan, dS, dPhi)).reshape(-1),
                          F.ring_garbage_h(d, S, Phi, r, n))
    assert np.array_equal(_host(amortize_witness(plan, dS, _dev(c, cuda))).reshape(-1),
                          F.ring_amortize(d, S, c, r, n))
    plan.check_device()


@pytest.mark.parametrize("d,n", [(8, 5), (64, 130), (128, 9), (256, 33)])
def test_single_products_of_unreduced_words(cuda, oracle, d, n):
    from lattica_b200.ntt import RingPlan
    plan, F = RingPlan(Q, d), oracle.Field(Q)
    a, b = _words((n, d), d), _words((n, d), n)
    lhs = _dev(a, cuda)
    plan.multiply_in_place(lhs, _dev(b, cuda))
    want = np.stack([F.ring_matvec(d, a[i:i + 1], 1, 1, b[i:i + 1], 1).reshape(d)
                     for i in range(n)])
    assert np.array_equal(_host(lhs), want)
    plan.check_device()
