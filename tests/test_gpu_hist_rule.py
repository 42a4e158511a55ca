"""Integer matrices with one gene far longer than the others: the histogram kernel's CTAs are slower
with a gene than the rank kernel's, so it takes a launch only while the longest gene does not outlast
the rest. The launch count shows the choice; U1 and P are the bucket path's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("longest,genes,length,hist", [(2_000, 600, 2_000, True), (60_000, 600, 2_000, True),
                                                       (200_000, 600, 2_000, False), (200_000, 2_000, 500, True),
                                                       (400_000, 2_000, 500, False), (90_000, 500, 90_000, True)])
def test_one_long_gene(longest, genes, length, hist):
    from hpdex_gb300.resident import ResidentMatrix
    rng = np.random.default_rng(1)
    sizes = [length] * (genes // 2) + [longest] + [length] * (genes - genes // 2)
    indptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n_rows = max(sizes)
    data = rng.integers(1, 30, indptr[-1]).astype(np.uint8)
    rows = np.concatenate([np.arange(k, dtype=np.int32) * (n_rows // k) for k in sizes])
    gid = (np.arange(n_rows) * 7919 % n_rows % 12).astype(np.int32)
    plan = ResidentMatrix(data, rows, indptr, n_rows).plan(gid, 11, zero_handling="min")
    plan.run()
    assert plan.timings()[1] == (3 if hist else 2)
    got = [x.copy() for x in plan.download()]
    plan.set_histogram(False)
    plan.run()
    assert plan.timings()[1] == 2
    for a, b in zip(plan.download(), got):
        np.testing.assert_array_equal(a, b)
