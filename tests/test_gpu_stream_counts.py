"""The stream kernel's counts of equal (value, group) pairs at their 16 bits: one value that a target
stores 65,534 to 131,073 times (counted, or where the count overflows left to the rank kernel), and a
target of more than 65,535 cells whose values hardly repeat. U1 and P equal the plain form's (the
rank kernel), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("equal", [0, 65_534, 65_535, 65_536, 65_537, 131_073])
def test_counts_at_16_bits(equal, dtype):
    from hpdex_gb300.resident import PLAIN, ResidentMatrix
    rng = np.random.default_rng(equal)
    n_rows, genes, ref, other = max(equal, 70_000) + 1_500, 3, 300, 700
    gid = np.concatenate([np.zeros(ref), np.full(other, 2), np.ones(n_rows - ref - other)]).astype(np.int32)
    data = np.sort(rng.standard_normal((genes, n_rows)).astype(dtype), axis=1)
    data = data[:, np.argsort(rng.permutation(n_rows))]
    for c in range(genes):
        data[c, n_rows - equal:] = 0.7265625
        data[c, :17 * c] = 0.7265625  # reference cells among the ties
        data[c, ref:ref + 5] = 0.7265625
    m = ResidentMatrix(data.reshape(-1), np.tile(np.arange(n_rows, dtype=np.int64), genes),
                       np.arange(genes + 1, dtype=np.int64) * n_rows, n_rows)
    plan = m.plan(gid, 2, zero_handling="min", use_continuity=True)
    plan.run(PLAIN)
    want = [x.copy() for x in plan.download()]
    for mode in (1, -1, 1):
        plan.set_stream(mode)
        plan.run()
        for a, b in zip(plan.download(), want):
            np.testing.assert_array_equal(a, b)
