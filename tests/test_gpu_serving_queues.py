"""Batches of the server that use all three kernels: integer counts (histogram kernel), continuous
values (stream kernel, some genes of which it leaves: crowded buckets), a matrix of both, and log counts
(rank kernel), queries of one to 40 targets together. Every result equals the plain form's
plan on the same matrix and groups, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dense(x, dtype):
    from hpdex_gb300.resident import ResidentMatrix
    genes, cells = x.shape
    return ResidentMatrix(x.astype(dtype).reshape(-1), np.tile(np.arange(cells, dtype=np.int64), genes),
                          np.arange(genes + 1, dtype=np.int64) * cells, cells)


def _matrices(rng, dtype):
    """(matrix, whether its plans take the stream kernel)"""
    from hpdex_gb300 import synthetic
    from hpdex_gb300.resident import ResidentMatrix
    normal = rng.standard_normal((90, 7_001))
    for c in range(3):  # a few hundred values within a bucket, and one far above
        normal[c] = 1 + rng.integers(0, 3_000, 7_001) * 2.0 ** -23
        normal[c, c] = 3e37
    both = rng.standard_normal((70, 6_500))
    both[::9] = rng.integers(0, 12, both[::9].shape)
    counts = rng.poisson(2.0, (300, 3_000))
    counts[::50, 5] = 1_000_000
    log = synthetic.perturb_screen(seed=41, n_rows=9_000, n_cols=120, n_targets=10, ref_size=2_000)
    return [(_dense(normal, dtype), True), (_dense(counts, dtype), False), (_dense(both, dtype), True),
            (ResidentMatrix(log.data.astype(dtype), log.indices, log.indptr, log.n_rows), False)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_three_kernels_in_a_batch(dtype):
    from hpdex_gb300.resident import PLAIN
    from hpdex_gb300.serving import Server
    rng = np.random.default_rng(3)
    mats = _matrices(rng, dtype)
    queries = []
    for i in range(16):
        m = i % len(mats)
        T = [1, 40, 7, 18][(i // len(mats) + i) % 4]
        gid = rng.permutation(np.arange(mats[m][0].n_rows) % (T + 4) - 3).astype(np.int32)
        gid[gid < 0] = rng.integers(-1, 1, (gid < 0).sum())  # no group, or the reference
        queries.append((m, gid, T, dict(zero_handling=["min", "max", "mix"][i % 3], use_continuity=bool(i % 2))))
    want = []
    for m, gid, T, options in queries:
        plan = mats[m][0].plan(gid, T, **options)
        plan.run(PLAIN)
        want.append([x.copy() for x in plan.download()])
        plan.run()
        assert plan.timings()[1] == (3 if mats[m][1] else 2)
    with Server(workspace_bytes=8 << 30, max_batch=16) as server:
        ids = [server.add_matrix(m) for m, _ in mats]
        for _ in range(3):
            sent = [server.submit(ids[m], gid, T, **options) for m, gid, T, options in queries]
            for q, w in zip(sent, want):
                for a, b in zip(q.result(), w):
                    np.testing.assert_array_equal(a, b)
        assert server.stats()["batches"] < 3 * len(queries)
