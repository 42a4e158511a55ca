"""Float matrices in which some columns hold whole numbers only: these go to the histogram kernel (or,
where they are few, to the rank kernel), the others to the stream kernel or the rank kernel by their own
values. The launches of a batched run show the division; U1 and P are the plain form's (the rank
kernel for every gene), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_ROWS = 6_000


def _columns(rng, kind, count):
    for j in range(count):
        if kind == "continuous":
            yield rng.standard_normal(N_ROWS), np.arange(N_ROWS)
        elif kind == "steps":  # many of each value, not whole
            yield rng.integers(1, 9, N_ROWS) / 4 + 0.125, np.arange(N_ROWS)
        elif kind == "flag":
            yield (rng.random(N_ROWS) < 0.3).astype(float), np.arange(N_ROWS)
        elif kind == "wide":  # whole numbers that span more than the histogram kernel counts
            yield rng.integers(0, 500_000, 2_000).astype(float), np.sort(rng.permutation(N_ROWS)[:2_000])
        else:
            k = int(rng.integers(0, 90))
            yield rng.integers(1, 30, k).astype(float), np.sort(rng.permutation(N_ROWS)[:k])


@pytest.mark.parametrize("zero", ["min", "mix"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kinds,launches", [
    (dict(continuous=20), 3),                                  # stream kernel, rank kernel
    (dict(continuous=20, flag=1), 3),
    (dict(continuous=20, counts=30, wide=1), 3),
    (dict(continuous=20, flag=2, wide=2, counts=700), 4),      # histogram kernel too
    (dict(steps=20, flag=2, counts=700), 3),                   # histogram kernel, rank kernel
    (dict(steps=20, flag=1), 2),
    (dict(continuous=4, steps=3, flag=1), 2),                  # too few seldom repeat
])
def test_division(kinds, launches, dtype, zero):
    from hpdex_gb300.resident import PLAIN, ResidentMatrix
    rng = np.random.default_rng(5)
    cols = [c for kind, count in kinds.items() for c in _columns(rng, kind, count)]
    cols = [cols[i] for i in rng.permutation(len(cols))]
    m = ResidentMatrix(np.concatenate([x for x, _ in cols]).astype(dtype),
                       np.concatenate([r for _, r in cols]).astype(np.int64),
                       np.concatenate([[0], np.cumsum([x.size for x, _ in cols])]).astype(np.int64), N_ROWS)
    gid = rng.permutation(np.arange(N_ROWS) % 8 - (np.arange(N_ROWS) % 80 == 0)).astype(np.int32)
    plan = m.plan(gid, 7, zero_handling=zero, use_continuity=True)
    plan.run(PLAIN)
    want = [x.copy() for x in plan.download()]

    def check(expected=None):
        plan.run()
        assert expected is None or plan.timings()[1] == expected
        for a, b in zip(plan.download(), want):
            np.testing.assert_array_equal(a, b)

    check(launches)
    plan.set_stream(1)
    check(3)
    plan.set_histogram(False)
    check(3)
    plan.set_stream(0)
    check(2)
    plan.set_histogram(True)
    check()
    plan.set_stream(-1)
    check(launches)
