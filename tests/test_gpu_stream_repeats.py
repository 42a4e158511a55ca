"""The stream kernel's repeat pass, where each warp moves the elements of cells hit more than once to
the front of its own part of the slice and counts them from there: target counts around one
tile of a warp (128) and one tile of every warp (4,096), all elements, some or few of them moved,
against the rank kernel bit for bit (no tolerance)."""
import numpy as np
import pytest

from test_gpu_stream import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind,T", [("one", 1), ("few", 9), ("log", 3), ("log", 300)])
def test_repeats_at_the_edges_of_parts(kind, T, dtype):
    """Dense genes: 30 reference cells, so a gene of n entries over n_rows rows holds about that many
    targets; the sizes run through the edges exactly for the whole-column genes."""
    for ntar in (127, 128, 129, 4_095, 4_096, 4_097, 8_191, 8_193):
        n = max(ntar + 30, 2 * T + 30)
        _check(kind, dtype, n, [n, n - 1, n - 2, n], 30, T, zero_handling="min")
