"""The layout tuner on plans whose genes the stream or the histogram kernel takes: the rank kernel's
candidates differ by noise only, so the plan keeps its layout (counters by the number of groups, 2^13
buckets, or what was set), and the results stay the same, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,T,counters", [("normal", 9, "shared"), ("normal", 1_200, "global"), ("counts", 9, "shared")])
def test_keeps_its_layout(kind, T, counters):
    from hpdex_gb300.resident import ResidentMatrix
    rng = np.random.default_rng(T)
    cells, genes = (8_000, 40) if kind == "normal" else (400, 600)
    x = rng.standard_normal(genes * cells) if kind == "normal" else rng.integers(0, 9, genes * cells)
    m = ResidentMatrix(x.astype(np.float32), np.tile(np.arange(cells, dtype=np.int64), genes),
                       np.arange(genes + 1, dtype=np.int64) * cells, cells)
    gid = rng.permutation(np.arange(cells) % (T + 1)).astype(np.int32)
    for bits in (13, 13, 11):
        plan = m.plan(gid, T, zero_handling="min")
        plan.set_bucket_bits(bits)
        plan.run()
        assert plan.timings()[1] == 3
        want = [a.copy() for a in plan.download()]
        tuned = plan.autotune(reps=1)
        assert (tuned["run_counters"], tuned["bucket_bits"]) == (counters, bits)
        assert len(tuned["ms"]) == 4 and all(t > 0.0 for t in tuned["ms"].values())
        plan.run()
        assert plan.timings()[1] == 3
        for a, b in zip(plan.download(), want):
            np.testing.assert_array_equal(a, b)
