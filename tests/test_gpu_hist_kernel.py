"""The histogram kernel (batched runs of integer counts) against the rank kernel's bucket path: U1
and P bit for bit at the edges of what it takes: value spans below, at and far above its counters'
room (few and many elements above the first range, several ranges), one to 3,000 groups, empty and one-entry genes, genes of other values (left to the
rank kernel), negative values, explicit zeros, sample sizes per gene (zero_handling none)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sms():
    import ctypes
    from hpdex_gb300 import _lib
    n = ctypes.c_int32()
    _lib.check(_lib.lib().hpdex_device_sm_count(ctypes.byref(n)))
    return n.value


@pytest.mark.parametrize("zero", ["none", "min", "mix"])
@pytest.mark.parametrize("dtype", [np.int8, np.uint16, np.int32, np.float32, np.float64, np.int64])
@pytest.mark.parametrize("T", [1, 7, 49, 255, 1_000, 3_000])
def test_hist_kernel_equals_bucket_path(T, dtype, zero):
    from hpdex_gb300.resident import PLAIN, ResidentMatrix
    rng = np.random.default_rng(T)
    n_rows = 13_007
    integer = np.issubdtype(dtype, np.integer)
    cap = np.iinfo(dtype).max if integer else 10 ** 6
    low = -3 if dtype in (np.int8, np.int32, np.float32) else 0
    cols, rows = [], []
    for span, tail in ((1, 0), (2, 0), (5, 0), (31, 0), (33, 0), (100, 0), (130, 0), (50, 255), (50, 256),
                       (50, 257), (9, 30), (700, 0), (2_047, 0), (3_064, 0), (3_065, 0), (8_191, 0), (9_000, 0)):
        x = low + np.minimum(rng.integers(0, span, n_rows), cap - 4)
        x[:2] = low, low + min(span - 1, cap - 4)
        if tail:  # values far above the others, with repeats
            x[2:2 + tail] = low + np.minimum(4_000 + rng.integers(0, 60, tail), cap - 4)
        if not integer and span == 33:
            x = x + 0.5  # another kind of gene
        cols.append(x[rng.permutation(n_rows)].astype(dtype))
        rows.append(np.arange(n_rows))
    if zero != "none":  # (every group must store two values under none)
        for k in (0, 1, 2, 255, 257, 4_001):
            cols.append(rng.integers(1, 9, k).astype(dtype))
            rows.append(np.sort(rng.permutation(n_rows)[:k]))
    # enough genes for the launch to choose the kernel (short ones, but under none)
    filler = 3 * _sms() * max(48, T + 1) // 48 if T < 300 else 0
    for k in range(filler):
        n = 2 * (T + 1) if zero == "none" else int(rng.integers(0, 90))
        cols.append(rng.integers(1, 5, n).astype(dtype))
        rows.append(np.arange(n))
    data, indices = np.concatenate(cols), np.concatenate(rows).astype(np.int64)
    indptr = np.concatenate([[0], np.cumsum([x.size for x in cols])]).astype(np.int64)
    gid = rng.integers(-1, T + 1, n_rows).astype(np.int32)
    gid[:2 * T + 2] = np.tile(np.arange(T + 1), 2)
    plan = ResidentMatrix(data, indices, indptr, n_rows).plan(gid, T, zero_handling=zero, use_continuity=True)
    plan.set_histogram(False)
    plan.run(PLAIN)
    want = [x.copy() for x in plan.download()]
    plan.set_histogram(True)
    for fused in (True, False):
        plan.set_fused_pvalues(fused)
        for _ in range(2):
            plan.run()
            for a, b in zip(plan.download(), want):
                np.testing.assert_array_equal(a, b)
