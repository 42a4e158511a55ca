"""BH FDR on the GPU at the edges of the sort's tiles (4,096 entries) and of its scan's rows (256
tiles at a time), with long runs of one digit, signed zeros and equal p-values: scipy's values
bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("values", ["uniform", "equal", "ties", "tiny"])
@pytest.mark.parametrize("n", [31, 255, 257, 4095, 4096, 4097, 8193, 256 * 4096 - 1, 256 * 4096 + 1])
def test_bh_at_tile_edges(n, values):
    from scipy.stats import false_discovery_control
    from hpdex_gb300._lib import bh_fdr
    rng = np.random.default_rng(n)
    p = {"uniform": lambda: rng.random(n), "equal": lambda: np.full(n, 0.25),
         "ties": lambda: rng.integers(0, 9, n) / 8.0,
         "tiny": lambda: 10.0 ** -rng.uniform(0, 320, n)}[values]()
    p[::7] = np.where(p[::7] == 0.0, -0.0, p[::7])
    np.testing.assert_array_equal(bh_fdr(p), false_discovery_control(np.abs(p), method="bh"))
