"""Which genes a plan gives to the stream kernel: plans of up to and above 100 groups, columns whose
values repeat seldom, often and nearly always, references that fit and do not, a few long genes left
behind. The plan's own choice, the stream kernel for all and the rank kernel for all give the
same U1 and P bit for bit (no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 98, 99, 100, 101, 300])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("steps,ref,long_rest", [(100_000, 900, 0), (700, 900, 0), (700, 900, 2), (60, 900, 0),
                                                 (700, 19_500, 0)])
def test_choice_changes_nothing(steps, ref, long_rest, dtype, T):
    from hpdex_gb300.resident import ResidentMatrix
    n_rows = 22_000
    rng = np.random.default_rng(steps + T)
    sizes = [1_500, 2_048, 1_023, 40, 0] + [1_800] * 30 + [n_rows if long_rest else 3_000] * 2
    rows = [np.sort(rng.permutation(n_rows)[:k]) for k in sizes]
    data = []
    for j, k in enumerate(sizes):
        few = 20 if long_rest and j >= len(sizes) - long_rest else steps
        data.append((np.round(rng.standard_normal(k) * few / 6) + 0.25) / few)
    indptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    gid = rng.integers(1, T + 1, n_rows).astype(np.int32)
    gid[rng.permutation(n_rows)[:ref]] = 0
    gid[:2 * T] = np.tile(np.arange(1, T + 1), 2)  # every target holds two rows
    m = ResidentMatrix(np.concatenate(data).astype(dtype), np.concatenate(rows).astype(np.int64), indptr, n_rows)
    plan = m.plan(gid, T, zero_handling="min", use_continuity=True)
    got = []
    for mode in (-1, 1, 0):
        plan.set_stream(mode)
        plan.run()
        got.append([x.copy() for x in plan.download()])
    for other in got[1:]:
        for a, b in zip(got[0], other):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("dtype,held", [(np.float32, 19_744), (np.float64, 10_968)])
def test_references_at_the_capacity(dtype, held):
    """Dense genes whose references fill the stream kernel's shared memory to the last entries, and
    exceed it (held: (230,400 - 96 - 32,800, in whole 16 bytes, - 64) / (2 * key bytes + 2))."""
    from hpdex_gb300.resident import ResidentMatrix
    rng = np.random.default_rng(3)
    for ref in (held - 9, held - 1, held, held + 1, held + 9):
        n_rows = ref + 700
        data = (np.round(rng.standard_normal(3 * n_rows) * 3000) + 0.25) / 3000
        indptr = np.arange(4, dtype=np.int64) * n_rows
        gid = np.zeros(n_rows, np.int32)
        gid[rng.permutation(n_rows)[:700]] = np.repeat([1, 2], 350)
        m = ResidentMatrix(data.astype(dtype), np.tile(np.arange(n_rows, dtype=np.int64), 3), indptr, n_rows)
        plan = m.plan(gid, 2, zero_handling="min")
        got = []
        for mode in (-1, 1, 0):
            plan.set_stream(mode)
            plan.run()
            got.append([x.copy() for x in plan.download()])
        for other in got[1:]:
            for a, b in zip(got[0], other):
                np.testing.assert_array_equal(a, b)
