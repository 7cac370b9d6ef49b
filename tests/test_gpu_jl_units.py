"""The JL kernels' work split: units of 32 columns go round the SMs' producer
warps (20 per SM, in groups of four that share a barrier), so the sizes where it
can go wrong are a single unit, a last round that leaves groups partly idle, a
part that ends inside a unit and units of several parts in one warp. Exact
integers: every word equals the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = 4294966657


def _parts(q, num_parts, cols, seed):
    rng = np.random.default_rng(seed)
    x = rng.integers(0, q, (num_parts, cols), dtype=np.uint64).astype(np.uint32)
    x[0, :4] = [0, q - 1, 1, q - 1]
    return x


# units per part: 1 (8 of 32 columns), 2, 3 with a ragged end, and 2980 / 3001 in
# all: 20 and 41 past the 148 x 20 = 2960 warps of one round
@pytest.mark.parametrize("rows,num_parts,n,d", [(256, 1, 1, 8), (256, 1, 1, 64), (256, 5, 9, 8),
                                                (256, 1490, 1, 64), (200, 3001, 1, 16),
                                                (255, 2, 747, 64)])
def test_projection_units(cuda, oracle, rows, num_parts, n, d):
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.labrador import JLMatrix
    plan, F = TwistedNttPlan(Q, d), oracle.Field(Q)
    seed = bytes((5 * i + n) & 0xFF for i in range(32))
    parts = _parts(Q, num_parts, n * d, rows + n)
    want, _ = oracle.jl_project(F, seed, rows, parts, num_parts, n * d, d)
    jl = JLMatrix.from_seed(rows, n * d, seed)
    assert np.array_equal(jl.project_multi(plan, parts, num_parts, d), want)
    plan.check_device()


@pytest.mark.parametrize("num_parts,n", [(1, 2), (1490, 1), (3, 500)])
def test_evaluation_units(cuda, oracle, num_parts, n):
    """Coefficient t of evals[m] is the projection of the witness with every
    polynomial multiplied by X^-t (64 oracle projections would be slow: t = 0, 1, 63)."""
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.labrador import JLMatrix
    d = 64
    plan, F = TwistedNttPlan(Q, d), oracle.Field(Q)
    seed = bytes((3 * i + n) & 0xFF for i in range(32))
    parts = _parts(Q, num_parts, n * d, 7 + n)
    got = JLMatrix.from_seed(256, n * d, seed).conjugated_evals(plan, parts, num_parts, d)
    polys = parts.reshape(num_parts, n, d).astype(np.uint64)
    ext = np.concatenate([polys, (Q - polys) % Q], axis=2)
    for t in (0, 1, 63):
        rot = np.ascontiguousarray(ext[:, :, t:t + d].astype(np.uint32).reshape(num_parts, n * d))
        want, _ = oracle.jl_project(F, seed, 256, rot, num_parts, n * d, d)
        assert np.array_equal(got[:, t], want)
    plan.check_device()
