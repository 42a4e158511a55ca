"""Group means where a gene's fixed-point sums are given up for double sums (a value whose bits they cannot
hold, early, late or many), also with non-finite values, and where they are not (all-negative genes,
large integers). Compared with math.fsum: equal where the sums are exact, within one rounding per addition else."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_ROWS = 9_001


def _gene(kind, rng):
    x = rng.standard_normal(N_ROWS)
    if kind == "negative":
        return -np.abs(x).astype(np.float32).astype(np.float64) - 0.001, True
    if kind == "first":  # the lowest bits lie 2^-300 below the top
        x[0] = 1e-90
    elif kind == "last":
        x[-1] = -1e-90
    elif kind == "many":
        x[::3] = 10.0 ** rng.uniform(-90, 5, x[::3].size)
    elif kind == "positive":
        return np.exp2(rng.uniform(-60, 60, N_ROWS)), False
    elif kind == "integers":
        return rng.integers(-(1 << 62), 1 << 62, N_ROWS).astype(np.float64), True
    return x, False


@pytest.mark.parametrize("include_zeros", [True, False])
@pytest.mark.parametrize("dirty", [False, True])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n_groups", [3, 700])
def test_group_mean_repeat(n_groups, dtype, dirty, include_zeros):
    from hpdex_gb300.resident import ResidentMatrix
    rng = np.random.default_rng(n_groups)
    kinds = ["negative", "first", "last", "many", "positive", "integers"]
    genes, exact = zip(*(_gene(k, rng) for k in kinds))
    data = np.stack(genes)
    if dirty:
        data[:, ::11] = np.nan
        data[:, 5::13] = -np.inf
        data[:, 7::17] = 0.0
    with np.errstate(over="ignore"):
        data = data.astype(dtype)
    gid = rng.integers(-1, n_groups, N_ROWS).astype(np.int32)
    m = ResidentMatrix(data.reshape(-1), np.tile(np.arange(N_ROWS, dtype=np.int32), len(kinds)),
                       np.arange(len(kinds) + 1, dtype=np.int64) * N_ROWS, N_ROWS)
    got = m.group_mean(gid, n_groups, include_zeros=include_zeros).reshape(len(kinds), n_groups)
    for c, kind in enumerate(kinds):
        for g in range(n_groups):
            v = data[c, gid == g].astype(np.float64)
            fine = v[np.isfinite(v)]
            denom = int((gid == g).sum()) - (v.size - fine.size) if include_zeros else fine.size
            want = math.fsum(fine) / denom if denom > 0 else 0.0
            if exact[c]:
                assert got[c, g] == want, (kind, g)
            else:
                tol = (fine.size + 1) * 2.0 ** -53 * (np.abs(fine).sum() / max(denom, 1) + abs(want))
                assert abs(got[c, g] - want) <= tol, (kind, g)
