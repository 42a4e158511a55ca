"""Host arrays at addresses that are no multiple of their element size, as numpy views into byte
buffers are: the resident matrix, the one-shot call and the group means take them (by the driver's
copies) with the results of aligned arrays, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shifted(a, by):
    """The array's values `by` bytes behind an aligned address."""
    raw = np.empty(a.nbytes + 64, np.uint8)
    at = -raw.ctypes.data % 64 + by
    out = raw[at:at + a.nbytes].view(a.dtype)
    out[:] = a
    assert out.ctypes.data % 64 == by
    return out


@pytest.mark.parametrize("index", [np.int32, np.int64])
@pytest.mark.parametrize("dtype,by_data,by_rows", [(np.float32, 1, 0), (np.float32, 0, 2), (np.float32, 4, 4),
                                                   (np.float64, 4, 4), (np.uint16, 1, 1), (np.int8, 3, 3)])
def test_misaligned_arrays(dtype, by_data, by_rows, index):
    from hpdex_gb300 import synthetic
    from hpdex_gb300.backend.bin import kernel
    from hpdex_gb300.resident import ResidentMatrix
    w = synthetic.umi_counts(seed=3, n_rows=4_000, n_cols=60, n_targets=3)
    data, rows = np.minimum(w.data, 100).astype(dtype), w.indices.astype(index)
    moved = _shifted(data, by_data), _shifted(rows, by_rows)

    def results(d, r):
        m = ResidentMatrix(d, r, w.indptr, w.n_rows)
        plan = m.plan(w.group_id, w.n_targets, zero_handling="min")
        plan.run()
        return [*plan.download(), m.group_mean(w.group_id, w.n_targets + 1),
                *kernel.mannwhitneyu(d, r, w.indptr, w.group_id, w.n_targets, zero_handling=1, fast_norm=False),
                kernel.group_mean(d, r, w.indptr, w.group_id, w.n_targets + 1)]

    for a, b in zip(results(*moved), results(data, rows)):
        np.testing.assert_array_equal(a, b)
