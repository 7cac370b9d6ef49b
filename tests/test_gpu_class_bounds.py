"""The byte classes of the point-major products at their largest: every evaluation of both
operands is 0xFEFFFFFF, the word below q with the largest class sum (class 3: 2 * 255 * 254 +
2 * 255^2 a word), and K gives every CTA 8192 words, so that the class reaches 99 % of 2^31.
A constant evaluation is a constant polynomial, so the sums are known in closed form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q, W = 4294966657, 0xFEFFFFFF
PER_CTA = 8192
PRODUCT = W * W * pow(1 << 32, -1, Q) % Q


def _const(cuda, *shape):
    import torch
    x = torch.zeros((*shape, 64), dtype=torch.int32, device=cuda)
    x[..., 0] = W - (1 << 32)
    return x


def _first_words(t):
    """Words 0 of the polynomials; the others are zero."""
    assert not bool(t[..., 1:].any())
    return t[..., 0].cpu().numpy().view(np.uint32)


def test_the_class_sum_is_near_its_bound():
    b = [(W >> 8 * i) & 255 for i in range(4)]
    largest = max(sum(b[i] * b[s - i] for i in range(4) if 0 <= s - i < 4) for s in range(7))
    assert W < Q and 0.99 * 2 ** 31 < largest * PER_CTA < 2 ** 31


# K ranges per point of a product: nine with four CTAs per SM, four with two, two with one
@pytest.mark.parametrize("rows,batch,ranges", [(16, 8, 9), (16, 64, 9), (32, 7, 9), (32, 33, 4),
                                               (48, 64, 4), (64, 64, 2), (64, 100, 2)])
@pytest.mark.parametrize("extra", [0, 1])
def test_commitments(cuda, rows, batch, ranges, extra):
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.commit import PreparedMatrix
    K = ranges * PER_CTA + extra
    plan = TwistedNttPlan(Q, 64)
    t = PreparedMatrix(plan, _const(cuda, rows, K), rows, K).mul_vec(_const(cuda, batch, K))
    assert (_first_words(t) == K * PRODUCT % Q).all()
    plan.check_device()


@pytest.mark.parametrize("r,ranges", [(16, 9), (32, 4), (64, 2)])
@pytest.mark.parametrize("extra", [0, 3])
def test_gram_and_garbage_h(cuda, r, ranges, extra):
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.labrador import compute_garbage_g, compute_garbage_h
    K = ranges * PER_CTA + extra
    plan, S = TwistedNttPlan(Q, 64), _const(cuda, r, K)
    for out in (compute_garbage_g(plan, S), compute_garbage_h(plan, S, S)):
        assert (_first_words(out) == K * PRODUCT % Q).all()
    plan.check_device()


@pytest.mark.parametrize("rank", [16, 32])
def test_grouped_products(cuda, rank):
    import torch
    from lattica_b200 import TwistedNttPlan, _lib
    from lattica_b200.batch import UnevenCommitBatch
    from lattica_b200.commit import PreparedMatrix
    lengths = [PER_CTA, 2 * PER_CTA, PER_CTA - 1, 100, 2 * PER_CTA - 33]
    plan, cols = TwistedNttPlan(Q, 64), 2 * PER_CTA
    A = PreparedMatrix(plan, _const(cuda, rank, cols), rank, cols)
    starts = np.concatenate([[0], np.cumsum(lengths)])
    items = [(int(starts[i]), i * rank, n, 0) for i, n in enumerate(lengths)]
    batch = UnevenCommitBatch(plan, [A], items)
    batch.set_config(PER_CTA, 0, _lib.ENGINE_POINT_MAJOR)
    t = torch.full((len(lengths) * rank, 64), -1, dtype=torch.int32, device=cuda)
    batch.commit_dev(_const(cuda, int(starts[-1])), t)
    got = _first_words(t).reshape(len(lengths), rank)
    assert all((got[i] == n * PRODUCT % Q).all() for i, n in enumerate(lengths))
    plan.check_device()
