"""BH adjusted p-values at the edges of the small tiles (1,024 entries) and of the line above which tiles
of 4,096 are taken: scipy's values bit for bit, with ties, zeros, ones and negative zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 255, 257, 1_023, 1_024, 1_025, 2_049, 5_040, 262_145, (1 << 19) - 1, 1 << 19,
                               (1 << 19) + 1])
def test_small_tiles(n):
    stats = pytest.importorskip("scipy.stats")
    from hpdex_gb300 import _lib
    rng = np.random.default_rng(n)
    p = rng.random(n)
    p[::3] = np.round(p[::3], 2)
    p[::11] = 0.0
    p[5::13] = -0.0
    p[7::17] = 1.0
    p[9::19] = 10.0 ** -rng.uniform(0, 300, p[9::19].size)
    np.testing.assert_array_equal(_lib.bh_fdr(p), stats.false_discovery_control(np.abs(p), method="bh"))
