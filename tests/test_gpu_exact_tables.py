"""Exact p-values around the size where the tables leave shared memory (n1 * n2 = 4,095) and with
sample sizes that differ by gene (marked pairs): against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ref,target", [(2, 2), (1023, 4), (2047, 2), (2048, 2), (63, 65), (64, 64), (64, 63),
                                        (5, 819), (40, 40), (30, 200)])
@pytest.mark.parametrize("zero", ["min", "none"])
def test_tables(ref, target, zero, oracle_lib):
    from hpdex_gb300.resident import ResidentMatrix
    rng = np.random.default_rng(ref)
    T, C = 3, 300
    sizes = [target, max(2, target - 1), max(2, target // 2)]
    gid = np.concatenate([np.zeros(ref, np.int32)] + [np.full(k, i + 1, np.int32) for i, k in enumerate(sizes)])
    n_rows = gid.size
    gid = gid[rng.permutation(n_rows)]
    x = rng.standard_normal((C, n_rows)).astype(np.float32)
    if zero == "none":  # some genes store fewer values: their samples are smaller
        drop = rng.random((C, n_rows)) < 0.05
        for g in range(T + 1):
            cells = np.flatnonzero(gid == g)[:2]
            drop[:, cells] = False
        x[drop] = np.nan
    indptr = np.arange(C + 1, dtype=np.int64) * n_rows
    indices = np.tile(np.arange(n_rows, dtype=np.int64), C)
    plan = ResidentMatrix(x.reshape(-1), indices, indptr, n_rows).plan(gid, T, zero_handling=zero, method="exact")
    plan.run()
    U1, P = plan.download()
    U1o, Po = oracle_lib.mannwhitneyu(x.reshape(-1), indices, indptr, gid, T,
                                      zero_handling={"none": 0, "min": 1}[zero], method=1)
    np.testing.assert_array_equal(U1, U1o.reshape(C, T).T)
    np.testing.assert_array_equal(P, Po.reshape(C, T).T)
