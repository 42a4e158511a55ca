"""Which plans of a float matrix the stream kernel takes: by how often equal values meet in a group
(values, length of the genes, number and evenness of the targets) and by the genes' length. A
batched run then has three launches (group ids, stream kernel, rank kernel) instead of two; either
way U1 and P are those of the rank kernel alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# dtype, cells (dense genes), distinct values (0: continuous), targets, share of the first target, stream
CASES = [
    (np.float32, 6_000, 0, 5, 0.0, True),
    (np.float32, 6_000, 0, 400, 0.0, True),
    (np.float32, 50_000, 5_000, 1, 0.0, False),    # 9 of a value in the group
    (np.float32, 50_000, 5_000, 90, 0.0, True),    # 0.1
    (np.float32, 50_000, 5_000, 90, 0.95, False),  # 0.1, but nearly all cells in one target
    (np.float32, 50_000, 0, 1, 0.0, True),
    (np.float32, 50_000, 500, 120, 0.0, False),    # 0.75
    (np.float32, 20_000, 500, 120, 0.0, True),     # 0.3
    (np.float32, 20_000, 500, 60, 0.0, False),     # one value in four repeats: not up to 100 groups
    (np.float32, 80_000, 20_000, 20, 0.0, True),   # 0.18 and a bitmap with room
    (np.float32, 170_000, 20_000, 60, 0.0, False),  # 0.13, but little room beside the reference
    (np.float32, 1_300, 0, 5, 0.0, False),
    (np.float32, 2_000, 0, 5, 0.0, True),
    (np.float32, 2_200, 0, 50, 0.0, True),
    (np.float32, 2_200, 0, 80, 0.0, False),
    (np.float64, 2_800, 0, 5, 0.0, False),
    (np.float64, 4_000, 0, 5, 0.0, True),
    (np.float64, 4_000, 0, 50, 0.0, False),
    (np.float64, 8_000, 0, 50, 0.0, True),
    (np.float64, 8_000, 0, 150, 0.0, False),
    (np.float64, 14_000, 0, 150, 0.0, True),
]


@pytest.mark.parametrize("dtype,cells,distinct,targets,first,stream", CASES)
def test_route(dtype, cells, distinct, targets, first, stream):
    from hpdex_gb300.resident import ResidentMatrix
    rng = np.random.default_rng(7)
    genes = 6
    if distinct:
        x = (rng.integers(0, distinct, genes * cells) + 0.25) / distinct + 1.0
    else:
        x = rng.standard_normal(genes * cells)
    gid = (1 + np.arange(cells) % targets).astype(np.int32)
    gid[2 * targets:2 * targets + int(first * cells)] = 1
    gid[cells - cells // 10:] = 0
    gid = rng.permutation(gid)
    m = ResidentMatrix(x.astype(dtype), np.tile(np.arange(cells, dtype=np.int64), genes),
                       np.arange(genes + 1, dtype=np.int64) * cells, cells)
    plan = m.plan(gid, targets, zero_handling="min")
    plan.run()
    assert plan.timings()[1] == (3 if stream else 2)
    got = [a.copy() for a in plan.download()]
    plan.set_stream(0)
    plan.run()
    assert plan.timings()[1] == 2
    for a, b in zip(plan.download(), got):
        np.testing.assert_array_equal(a, b)
