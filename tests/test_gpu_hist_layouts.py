"""The histogram kernel with two CTAs and one CTA to an SM (plans of 350 to 1,000 targets), where a CTA
has room for a few dozen values of every group: genes at the edges of a range, of several ranges and
above them, and with few elements above the first. The launch count shows that the kernel ran; U1
and P equal the bucket path's, bit for bit."""
import numpy as np
import pytest

from test_gpu_hist_kernel import _sms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zero", ["min", "mix"])
@pytest.mark.parametrize("dtype", [np.int32, np.float32, np.uint8])
@pytest.mark.parametrize("T", [350, 501, 1_000])
def test_many_groups(T, dtype, zero):
    from hpdex_gb300.resident import PLAIN, ResidentMatrix
    rng = np.random.default_rng(T)
    n_rows, G = 9_001, T + 1
    cap = 255 if dtype == np.uint8 else 10 ** 6
    # values of a range: the counters of a CTA over the groups, a multiple of 4
    room = (113_664 if T == 350 else 230_400) - (24 * G + 15) // 16 * 16
    W = (room // 16 * 4 - 4) // G & ~3
    cols, rows = [], []
    for span, tail in ((1, 0), (W - 1, 0), (W, 0), (W + 1, 0), (2 * W, 0), (8 * W - 1, 0), (8 * W, 0), (8 * W + 1, 0),
                       (9 * W, 0), (W // 2, 255), (W // 2, 256), (W // 2, 257)):
        x = rng.integers(1, max(span, 1) + 1, n_rows)
        x[:2] = 1, max(span, 1)
        if tail:
            x[2:2 + tail] = 3 * W + rng.integers(0, 40, tail)
        cols.append(np.minimum(rng.permutation(x), cap).astype(dtype))
        rows.append(np.arange(n_rows))
    for k in range(_sms() * G // 16 + 1):  # enough genes for the launch to choose the kernel
        n = int(rng.integers(0, 12))
        cols.append(rng.integers(1, 5, n).astype(dtype))
        rows.append(rng.integers(0, n_rows - 12) + np.arange(n))
    m = ResidentMatrix(np.concatenate(cols), np.concatenate(rows).astype(np.int64),
                       np.concatenate([[0], np.cumsum([x.size for x in cols])]).astype(np.int64), n_rows)
    gid = rng.integers(-1, G, n_rows).astype(np.int32)
    gid[:2 * G] = np.tile(np.arange(G), 2)
    plan = m.plan(gid, T, zero_handling=zero, use_continuity=True)
    plan.set_histogram(False)
    plan.run(PLAIN)
    want = [x.copy() for x in plan.download()]
    plan.set_histogram(True)
    plan.run()
    assert plan.timings()[1] == 3
    for a, b in zip(plan.download(), want):
        np.testing.assert_array_equal(a, b)
