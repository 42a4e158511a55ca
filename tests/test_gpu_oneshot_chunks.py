"""The one-shot call cuts a matrix into chunks of at least 2^19 entries (at most 12): matrices
just below and above one, two and three chunks, with columns of odd lengths (chunks then start
at any alignment), empty columns and one long column, give the resident matrix's results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHUNK = 1 << 19


@pytest.mark.parametrize("index", [np.int32, np.int64])
@pytest.mark.parametrize("dtype", [np.uint8, np.float32, np.float64])
@pytest.mark.parametrize("nnz", [CHUNK - 1, CHUNK, 2 * CHUNK - 1, 2 * CHUNK + 1, 3 * CHUNK + 77,
                                 14 * CHUNK + 5])
def test_chunked_call_equals_resident(nnz, dtype, index):
    from hpdex_gb300.backend.bin import kernel
    from hpdex_gb300.resident import ResidentMatrix
    rng = np.random.default_rng(nnz)
    n_rows = 9_001
    sizes = [0, n_rows]
    while sum(sizes) < nnz:
        sizes.append(min(int(rng.integers(0, n_rows)), nnz - sum(sizes)))
    sizes.append(0)
    indices = np.concatenate([np.sort(rng.permutation(n_rows)[:k]) for k in sizes]).astype(index)
    indptr = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    data = rng.integers(1, 200, indices.size).astype(dtype)
    if dtype != np.uint8:
        data = np.log1p(data).astype(dtype)
    gid = rng.integers(-1, 9, n_rows).astype(np.int32)
    U1, P = kernel.mannwhitneyu(data, indices, indptr, gid, 8, zero_handling=1, use_continuity=True,
                                fast_norm=False)
    m = ResidentMatrix(data, indices, indptr, n_rows)
    plan = m.plan(gid, 8, zero_handling="min", use_continuity=True)
    plan.run()
    for a, b in zip((U1, P), plan.download()):
        np.testing.assert_array_equal(a, b)
