"""Kernels that a rule of dispatch reaches for few of the sizes it accepts: the point-major
product's shapes for five to eight vectors, the matrix-vector kernel with a split K (more
rows than the vector products take, or another degree), and the gathering tensor-core
products on ring plans, whose inputs are not reduced mod the auxiliary primes. Against the
oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q, Q256, Q_RING = 4294966657, 4294962689, 4294967291
AUX = (4294962689, 4294957057, 4294955009)


def _words(q, shape, seed):
    rng = np.random.default_rng(seed)
    x = rng.integers(0, q, shape, dtype=np.uint64).astype(np.uint32)
    x.reshape(-1)[: x.size // 4] = q - 1
    return x


def _dev(x, cuda):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).to(cuda)


def _host(t):
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("q,d,rows,cols,batch", [
    (Q, 64, 16, 4100, 5), (Q, 64, 17, 4100, 8), (Q, 64, 32, 4100, 8), (Q, 64, 24, 515, 6),
    (Q, 64, 48, 1030, 7), (Q, 64, 64, 2049, 8),                # five to eight vectors
    (Q, 64, 65, 1000, 2), (Q, 64, 70, 129, 4), (Q256, 256, 16, 300, 1), (Q256, 128, 9, 520, 3)])
def test_commitments(cuda, oracle, q, d, rows, cols, batch):
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.commit import PreparedMatrix
    plan, P = TwistedNttPlan(q, d), oracle.Plan(q, d)
    A, s = _words(q, (rows, cols, d), rows), _words(q, (batch, cols, d), cols)
    got = PreparedMatrix(plan, _dev(A, cuda), rows, cols).mul_vec(_dev(s, cuda))
    want = P.matvec(A, rows, cols, s, batch, threads=0).reshape(batch, rows, d)
    assert np.array_equal(_host(got), want)
    plan.check_device()


@pytest.mark.parametrize("r,n", [(6, 37), (33, 36), (64, 65)])
def test_gathering_products_of_a_ring_plan(cuda, oracle, monkeypatch, r, n):
    from lattica_b200.commit import PreparedMatrix
    from lattica_b200.labrador import compute_garbage_g, compute_garbage_h
    from lattica_b200.ntt import RingPlan
    monkeypatch.setenv("GRID_GPU_CONTRACTION", "gather")
    plan, F, d = RingPlan(Q_RING, 64), oracle.Field(Q_RING), 64
    rng = np.random.default_rng(r * n)
    edge = np.array([p + e for p in AUX for e in (-1, 0, 1)] + [Q_RING - 1], dtype=np.uint64)
    word = lambda *s: np.where(rng.integers(0, 4, s) == 0,
                               rng.integers(0, Q_RING, s, dtype=np.uint64),
                               edge[rng.integers(0, edge.size, s)]).astype(np.uint32)
    S, Phi, A = word(r, n, d), word(r, n, d), word(20, n, d)
    dS, dPhi = _dev(S, cuda), _dev(Phi, cuda)
    assert np.array_equal(_host(compute_garbage_g(plan, dS)).reshape(-1), F.ring_gram(d, S, r, n))
    assert np.array_equal(_host(compute_garbage_h(plan, dS, dPhi)).reshape(-1),
                          F.ring_garbage_h(d, S, Phi, r, n))
    assert np.array_equal(_host(PreparedMatrix(plan, _dev(A, cuda), 20, n).mul_vec(dS)).reshape(-1),
                          F.ring_matvec(d, A, 20, n, S, r).reshape(-1))
    plan.check_device()
