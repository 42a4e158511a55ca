"""Group means on the GPU against exactly summed values (math.fsum), where the fixed-point sums
can go wrong: word carries and signs, wide value ranges (the repeat with double atomics),
subnormals, 64-bit integers above 2^53, accumulator sets, many groups, ragged columns."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_ROWS = 4001


def _values(kind, rng, n):
    if kind == "log":
        return np.log1p(rng.poisson(2.0, n) + 0.25).astype(np.float32)
    if kind == "signed":
        return rng.standard_normal(n).astype(np.float32)
    if kind == "signed64":
        return rng.standard_normal(n)
    if kind == "positive64":  # full mantissas over 20 binades: three words
        return np.exp2(rng.uniform(-10, 10, n))
    if kind == "spread":  # one value dwarfs the others: their bits need the double sums
        x = rng.standard_normal(n).astype(np.float32)
        x[::97] = np.float32(3e30)
        return x
    if kind == "subnormal":
        return (rng.integers(-(1 << 20), 1 << 20, n) * 2.0 ** -149).astype(np.float32)
    if kind == "nonfinite":
        x = rng.standard_normal(n).astype(np.float32)
        x[::5] = np.nan
        x[1::7] = -np.inf
        x[2::11] = 0.0
        return x
    info = np.iinfo(kind)
    return rng.integers(info.min, info.max, n, dtype=kind, endpoint=True)


@pytest.mark.parametrize("include_zeros", [True, False])
@pytest.mark.parametrize("kind,n_groups", [
    ("log", 1), ("log", 50), ("log", 65), ("log", 501), ("log", 3000), ("log", 12000),
    ("signed", 7), ("signed", 300), ("signed64", 50), ("positive64", 33), ("spread", 20),
    ("subnormal", 9), ("nonfinite", 40), ("int8", 64), ("uint16", 129), ("int32", 5),
    ("uint32", 50), ("int64", 50), ("uint64", 17)])
def test_group_mean_sums(kind, n_groups, include_zeros):
    from hpdex_gb300.resident import ResidentMatrix
    rng = np.random.default_rng(len(kind) * 1000 + n_groups)
    sizes = [0, 1, 3, 31, 33, 511, 512, 513, 2047, 2049, N_ROWS]
    rows = [np.sort(rng.choice(N_ROWS, k, replace=False)) for k in sizes]
    data = np.concatenate([_values(kind, rng, k) for k in sizes])
    indices = np.concatenate(rows).astype(np.int64)
    indptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    gid = rng.integers(-2, n_groups + 3, N_ROWS).astype(np.int32)
    m = ResidentMatrix(data, indices, indptr, N_ROWS)
    got = m.group_mean(gid, n_groups, include_zeros=include_zeros).reshape(len(sizes), n_groups)
    n_rows = np.bincount(gid[(gid >= 0) & (gid < n_groups)], minlength=n_groups)
    # the double sums of the repeat (and of more groups than shared memory holds) may round once
    # per addition; every other sum is exact
    rounds = kind in ("signed", "signed64", "spread", "nonfinite") or n_groups > 11000
    for c in range(len(sizes)):
        x, g = data[indptr[c]:indptr[c + 1]], gid[rows[c]]
        for k in np.unique(np.clip(g, 0, n_groups - 1)):
            v = x[g == k].astype(np.float64)
            fine = v[np.isfinite(v)]
            denom = int(n_rows[k]) - (v.size - fine.size) if include_zeros else fine.size
            want = math.fsum(fine) / denom if denom > 0 else 0.0
            if rounds:
                tol = (fine.size + 1) * 2.0 ** -53 * (np.abs(fine).sum() / max(denom, 1) + abs(want))
                assert abs(got[c, k] - want) <= tol, (c, k)
            else:
                assert got[c, k] == want, (c, k)
        empty = np.setdiff1d(np.arange(n_groups), g)
        assert not got[c, empty].any()
