"""JL matrices of fewer than 253 rows: a column's bytes begin anywhere in a keystream block,
and the next block is made only where they reach into it. Byte counts that divide a block,
end with one, or cross it by one byte, with the int8 entries in groups of four polynomials
and singly, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = 4294966657


@pytest.mark.parametrize("rows", [1, 4, 5, 12, 60, 64, 68, 85, 128, 129, 132, 200, 248, 252])
@pytest.mark.parametrize("num_parts,n,d", [(3, 12, 8), (2, 33, 16)])
def test_rows_match_oracle(cuda, oracle, rows, num_parts, n, d):
    from lattica_b200 import TwistedNttPlan
    from lattica_b200.labrador import JLMatrix
    plan, F = TwistedNttPlan(Q, d), oracle.Field(Q)
    seed = bytes((9 * i + rows) & 0xFF for i in range(32))
    rng = np.random.default_rng(rows * n)
    parts = rng.integers(0, Q, (num_parts, n * d), dtype=np.uint64).astype(np.uint32)
    want, flat = oracle.jl_project(F, seed, rows, parts, num_parts, n * d, d)
    p, got = JLMatrix.from_seed(rows, n * d, seed).project_and_extract_jl_rows(plan, parts,
                                                                               num_parts, d)
    assert np.array_equal(p, want)
    assert np.array_equal(got, flat)
    plan.check_device()
