"""Unit counts of very large bins.

A bin of n points holds n^2 / (2 chunk segment) units when it is cut into
segments of fixed length, which passes the work lists' 32-bit offsets at 12M
points of long rows in one bin.  Segments grow with the work instead, so that a
join whose home chunks alone fit the lists is never refused.
MISTIC_TEST_WORKLIST_LIMIT lowers the limit to half the units of the join as it
is cut by default."""
import numpy as np
import pytest

from helpers import diff_pairs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ring", [0, 40000])
@pytest.mark.parametrize("mode,d", [("fp64", 2), ("fp64", 140), ("fp32", 2), ("fp32", 140), ("bf16", 18), ("bf16", 140)])
def test_one_bin_of_more_units_than_the_lists_hold(handle, monkeypatch, mode, d, ring):
    n = 40000 if ring else 12000
    if ring and mode != "fp64":
        pytest.skip("home chunks of one list: enough units at this size only there")
    x = np.random.default_rng(d).random((n, d))
    eps = {2: 0.004, 18: 0.75, 140: 3.9}[d]
    a = handle.selfjoin(x, 0, eps, mode=mode, pairs="host", sort_pairs=True, ring_capacity=ring)
    assert a.n_bins == 1
    if n <= 12000:
        ref = O.brute_pairs(x, eps)
        assert np.array_equal(a.pairs, ref), diff_pairs(a.pairs, ref)
    monkeypatch.setenv("MISTIC_TEST_WORKLIST_LIMIT", str(max(a.n_units, a.n_units_tc) // 2))
    b = handle.selfjoin(x, 0, eps, mode=mode, pairs="host", sort_pairs=True, ring_capacity=ring)
    assert 0 < max(b.n_units, b.n_units_tc) <= max(a.n_units, a.n_units_tc) // 2
    assert np.array_equal(b.pairs, a.pairs), diff_pairs(b.pairs, a.pairs)
