"""Streamed pair ring whose band list overflows too.

The band list of a pass has a fixed length as well.  A flush that crosses its
end leaves slots that hold nothing, which the band decisions have to skip, and
its unit runs again.  Bounds wide enough that every candidate pair goes to the
band list, which MISTIC_BAND_CAP keeps shorter than the band of a pass; the
length is no multiple of a flush's."""
import numpy as np
import pytest

from helpers import diff_pairs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,d,eps", [("tf32", 3, 0.005), ("tf32", 40, 0.005), ("bf16", 3, 0.001), ("bf16", 40, 0.001)])
@pytest.mark.parametrize("band_cap", [9001, 40003])
def test_band_list_overflows_in_a_ring_pass(handle, monkeypatch, mode, d, eps, band_cap):
    rng = np.random.default_rng(d)
    x = np.repeat(rng.random((400, d)), 30, axis=0)[rng.permutation(12000)]
    ref = O.brute_pairs(x, eps)
    monkeypatch.setenv("MISTIC_TC_MIN_BIN", "1")
    monkeypatch.setenv("MISTIC_TC_WIDE", "1")
    monkeypatch.setenv("MISTIC_BAND_CAP", str(band_cap))
    r = handle.selfjoin(x, 6, eps, mode=mode, pairs="host", sort_pairs=True, ring_capacity=50000)
    assert r.n_units_tc > 0 and r.band_pairs > 0
    assert r.ring_passes > 1 and r.ring_units_redone > 0
    assert np.array_equal(r.pairs, ref), diff_pairs(r.pairs, ref)
