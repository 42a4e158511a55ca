"""The stream kernel (all genes forced onto it, and the plan's own choice) against the rank kernel
(the plain form runs it for every gene): U1 and P bit for bit, where the stream kernel can go
wrong: pairs of equal (value, group) found through the bitmap and counted in one or more
partitions, genes it leaves (too many reference elements, crowded buckets), signed and wide
ranges, heavy ties, empty and tiny genes, explicit zeros, non-finite values, row ids outside the
matrix, few and many groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values(kind, rng, n):
    if kind == "log":
        return np.log1p(1e4 * (1 + rng.poisson(0.7, n)) / rng.integers(1500, 2100, n))
    if kind == "normal":
        return rng.standard_normal(n)
    if kind == "few":  # half-integers: not small integers, a handful of values
        return rng.integers(-2, 4, n) + 0.5
    if kind == "one":
        return np.full(n, 0.75)
    if kind == "crowded":  # distinct values far below the range's resolution, and one far above
        x = 1.0 + np.arange(n) * 2.0 ** -23
        if n:
            x[rng.permutation(n)[0]] = 3e38
        return x
    if kind == "wide":
        x = rng.standard_normal(n) * 10.0 ** rng.uniform(-44, 37, n)
        x[rng.random(n) < 0.3] = 1e-40
        return x
    x = rng.standard_normal(n).round(1)  # "dirty": ties, zeros, non-finite
    x[rng.random(n) < 0.1] = 0.0
    x[rng.random(n) < 0.05] = np.nan
    x[rng.random(n) < 0.03] = np.inf
    x[rng.random(n) < 0.03] = -0.0
    return x


def _check(kind, dtype, n_rows, sizes, ref, T, in_group=1.0, bad_rows=False, **options):
    from hpdex_gb300.resident import PLAIN, ResidentMatrix
    rng = np.random.default_rng(n_rows + T)
    rows = [np.sort(rng.permutation(n_rows)[:k]) for k in sizes]
    data = np.concatenate([_values(kind, rng, k) for k in sizes]).astype(dtype)
    indices = np.concatenate(rows).astype(np.int64)
    if bad_rows:
        indices[::37] = n_rows + 5
        indices[1::41] = -3
    indptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    gid = rng.integers(1, T + 1, n_rows).astype(np.int32)
    gid[rng.random(n_rows) >= in_group] = -1
    gid[:2 * T] = np.tile(np.arange(1, T + 1), 2)  # every target holds two rows
    gid[2 * T:2 * T + ref] = 0
    perm = rng.permutation(n_rows)
    gid = gid[perm]
    m = ResidentMatrix(data, indices, indptr, n_rows)
    plan = m.plan(gid, T, **options)
    plan.run(PLAIN)
    want = [x.copy() for x in plan.download()]
    for mode, fused in ((1, True), (1, False), (-1, True), (0, True)):
        plan.set_stream(mode)
        plan.set_fused_pvalues(fused and options.get("method") != "exact")
        for _ in range(2):
            plan.run()
            for a, b in zip(plan.download(), want):
                np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("zero", ["min", "max", "mix"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["log", "normal", "few", "one", "crowded", "wide", "dirty"])
def test_stream_equals_rank(kind, dtype, zero):
    """Genes from empty to 20,000 entries (fewer where the rank kernel, which gives the expected
    values, compares a gene's elements pairwise)."""
    sizes = [0, 1, 2, 31, 33, 127, 129, 1_000, 4_097, 9_000, 13_001, 20_000]
    if kind in ("crowded", "wide"):
        sizes = [0, 1, 33, 600, 4_097]
    _check(kind, dtype, 20_000, sizes, 2_500, 23, zero_handling=zero, use_continuity=True,
           bad_rows=kind == "dirty")


@pytest.mark.parametrize("kind,T,ref", [("log", 1, 4_000), ("log", 501, 12_000), ("normal", 60, 9_000),
                                        ("few", 501, 12_000), ("few", 1, 100), ("log", 37, 90_000)])
def test_stream_large_genes(kind, T, ref):
    """120,000 entries: several partitions, 16-bit counts exceeded ("few", one target), references
    that do not fit (left to the rank kernel)."""
    _check(kind, np.float32, 120_000, [120_000, 60_000, 119_999, 5], ref, T, zero_handling="min")


@pytest.mark.parametrize("T", [2, 700, 1_500, 4_000])
def test_stream_many_groups(T):
    _check("normal", np.float32, 30_000, [30_000, 29_000, 0, 900], 40, T, in_group=0.6, zero_handling="mix")


@pytest.mark.parametrize("options", [dict(tie_correction=False), dict(alternative="less"),
                                     dict(alternative="greater", use_continuity=True), dict(fast_norm=True)])
def test_stream_options(options):
    _check("dirty", np.float32, 9_000, [9_000, 4_000, 17], 900, 12, zero_handling="min", **options)


@pytest.mark.parametrize("method", ["asymptotic", "exact"])
def test_stream_zero_handling_none(method):
    _check("normal", np.float64, 3_000, [3_000] * 5, 40, 30, zero_handling="none", method=method)
