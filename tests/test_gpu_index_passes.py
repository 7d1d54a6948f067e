"""The passes over the points before the index: column statistics in one
stream whatever the row length, reference-point distances 32 columns at a
time.

Row lengths around the column tiles (32 staged columns, 256-column statistics
tiles) and row counts around the blocks; reference points from the bounding
box (RP box), the principal axes and the caller, on every input type, must
all give the oracle's pairs.  Non-finite values are found wherever they are,
and the statistics skip NaN as before when the check is off."""
import numpy as np
import pytest

from helpers import diff_pairs
from oracle import oracle as O

import mistic
from mistic import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n,d,k", [(2, 1, 1), (257, 31, 3), (513, 32, 8), (1000, 33, 9), (300, 64, 16), (700, 255, 5),
                                   (256, 256, 8), (400, 257, 6), (60, 600, 4)])
def test_row_lengths_around_the_tiles(handle, dtype, n, d, k):
    rng = np.random.default_rng(n + d)
    x = (rng.normal(size=(n, d)) * rng.uniform(0.1, 2.0, size=d)).astype(dtype)
    x[n // 2:] = x[:n - n // 2] + (rng.normal(size=(n - n // 2, d)) * 0.01).astype(dtype)
    eps = 0.02 * np.sqrt(d)
    ref = O.brute_pairs(x, eps)
    for rp in ("pca", "box", "user"):
        kw = {"rp_user": rng.normal(size=(k, d)) * 5} if rp == "user" else {}
        r = handle.selfjoin(x, k, eps, rp=rp, pairs="host", sort_pairs=True, **kw)
        assert np.array_equal(r.pairs, ref), (rp, diff_pairs(r.pairs, ref))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n,d", [(5, 1), (1000, 2), (300, 18), (50, 300)])
@pytest.mark.parametrize("value", [np.nan, -np.nan, np.inf, -np.inf])
def test_non_finite_values_are_found(handle, dtype, n, d, value):
    x = np.random.default_rng(1).random((n, d)).astype(dtype)
    for i, j in ((0, 0), (n - 1, d - 1), (n // 2, d // 2)):
        y = x.copy()
        y[i, j] = value
        with pytest.raises(mistic.MisticError) as e:
            handle.selfjoin(y, 2, 0.1)
        assert e.value.status == L.ERR_NOT_FINITE


def test_signs_and_zeros_in_the_statistics(handle):
    """All-negative, mixed and signed-zero columns: a wrong minimum or maximum
    moves the box reference points or the centre, never the pairs; a spread of
    1e-300 .. 1e300 must not overflow into a wrong key."""
    rng = np.random.default_rng(2)
    x = rng.random((900, 4)) * [-1.0, 1.0, 1.0, 1e-3] + [-5.0, 0.0, -0.5, 0.0]
    x[::3, 1] = -0.0
    ref = O.brute_pairs(x, 0.07)
    for rp in ("box", "pca"):
        r = handle.selfjoin(x, 3, 0.07, rp=rp, pairs="host", sort_pairs=True)
        assert np.array_equal(r.pairs, ref), (rp, diff_pairs(r.pairs, ref))
