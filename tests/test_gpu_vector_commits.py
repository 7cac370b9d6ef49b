"""A matrix times one to four vectors: every rows-per-thread variant at its edges,
columns around one block of 64 and past two CTAs' worth of SMs (several blocks per
CTA), sums of two products of different lengths, and the batch sizes around the
path's limit. Every word equals the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = 4294966657


def _words(q, shape, seed):
    rng = np.random.default_rng(seed)
    x = rng.integers(0, q, shape, dtype=np.uint64).astype(np.uint32)
    x.reshape(-1)[: x.size // 3] = q - 1
    return x


def _dev(x, cuda):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x).view(np.int32)).to(cuda)


def _host(t):
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("q,batch,rows,cols", [(Q, 1, 1, 129), (Q, 2, 8, 192), (Q, 3, 9, 1000),
                                               (Q, 4, 16, 131), (Q, 5, 16, 131), (Q, 1, 17, 4097),
                                               (Q, 2, 32, 190), (Q, 1, 33, 65), (Q, 1, 64, 300),
                                               (Q, 1, 65, 30), (Q, 2, 33, 130), (Q, 1, 2, 19100),
                                               (12289, 2, 5, 257)])
def test_vector_products(cuda, oracle, q, batch, rows, cols):
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.commit import PreparedMatrix
    plan, P = TwistedNttPlan(q, 64), oracle.Plan(q, 64)
    A, s = _words(q, (rows, cols, 64), rows), _words(q, (batch, cols, 64), cols)
    got = PreparedMatrix(plan, _dev(A, cuda), rows, cols).mul_vec(_dev(s, cuda))
    want = P.matvec(A, rows, cols, s, batch, threads=0).reshape(batch, rows, 64)
    assert np.array_equal(_host(got), want)
    plan.check_device()


@pytest.mark.parametrize("ring", [False, True])
@pytest.mark.parametrize("batch,rows,mc,oc", [(1, 16, 300, 129), (2, 9, 129, 2000), (1, 8, 150, 64),
                                              (1, 33, 40, 7), (5, 16, 200, 300)])
def test_sums_of_two_products(cuda, oracle, ring, batch, rows, mc, oc):
    """(1, 8, 150, 64): one of the two fits the one-launch kernel, so each runs by itself."""
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.commit import (BdlopCommitmentKey, CommitmentDimensions, LinearCommitmentKey)
    from lattica_b200.ntt import RingPlan
    q = 4294967291 if ring else Q
    plan, F = (RingPlan(q, 64) if ring else TwistedNttPlan(q, 64)), oracle.Field(q)
    if ring:
        mc, oc = mc // 4 + 100, oc // 4 + 100
        mul = lambda a, r, c, v: F.ring_matvec(64, a, r, c, v, batch)
    else:
        P = oracle.Plan(q, 64)
        mul = lambda a, r, c, v: P.matvec(a, r, c, v, batch, threads=0)
    A, B, K = (_words(q, (rows, c, 64), i) for i, c in enumerate((mc, oc, oc)))
    m, r = _words(q, (batch, mc, 64), 4), _words(q, (batch, oc, 64), 5)
    want = F.add_slice(mul(A, rows, mc, m).reshape(-1), mul(B, rows, oc, r).reshape(-1))
    key = LinearCommitmentKey(plan, _dev(A, cuda), _dev(B, cuda),
                              CommitmentDimensions(mc, oc, rows))
    assert np.array_equal(_host(key.recompute(_dev(m, cuda), _dev(r, cuda))).reshape(-1), want)
    assert np.array_equal(key.recompute(m, r).reshape(-1), want)  # host buffers
    bd = BdlopCommitmentKey(plan, _dev(K, cuda), _dev(A, cuda), _dev(B, cuda), rows, mc, oc)
    u, v = bd.recompute_parts(_dev(m, cuda), _dev(r, cuda))
    assert np.array_equal(_host(v).reshape(-1), want)
    assert np.array_equal(_host(u).reshape(-1), mul(K, rows, oc, r).reshape(-1))
    plan.check_device()
