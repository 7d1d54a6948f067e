"""The short-row tensor-core join at K = 48 to 128 (rows of 31 to 126 columns,
the K-chunked kernel switched off): units of many candidate tiles.

Two or three operand stages are used again and again within a unit while only
some of the four MMA warps hold work of a given tile (one or two home chunks),
so every stage's reuse has to wait for all of them.  d is at both edges of each
padded width with an instance of its own; home bins of one, one and a bit and
several chunks, alone and as members of a fused batch."""
import numpy as np
import pytest

from helpers import diff_pairs
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DIMS = [31, 46, 47, 62, 63, 78, 79, 90, 94, 95, 110, 111, 126]


def _points(n, d, seed):
    """Points whose nearest pairs are about the radius apart: few bins, long candidate lists."""
    x = np.random.default_rng(seed).random((n, d))
    eps = float(np.sqrt(d / 6.0) * 0.8)
    return x, eps


@pytest.mark.parametrize("d", DIMS)
@pytest.mark.parametrize("n", [129, 3000, 6001])
def test_many_tiles_a_unit(handle, monkeypatch, n, d):
    x, eps = _points(n, d, n + d)
    monkeypatch.setenv("MISTIC_TC_WIDE", "0")
    r = handle.selfjoin(x, 1, eps, mode="bf16", pairs="host", sort_pairs=True)
    assert r.tc_kernel == "short-rows" and r.n_units_tc > 0
    ref = O.brute_pairs(x, eps)
    assert np.array_equal(r.pairs, ref), diff_pairs(r.pairs, ref)


def test_batch_members(handle):
    inst = [(*_points(n, d, n + d), 1) for n, d in [(5000, 31), (130, 31), (3000, 90), (4100, 90), (2000, 126), (900, 62)]]
    res = handle.batch_selfjoin([(x, k, e) for x, e, k in inst], mode="bf16", pairs="host", sort_pairs=True)
    for (x, eps, _), r in zip(inst, res):
        ref = O.brute_pairs(x, eps)
        assert np.array_equal(r.pairs, ref), diff_pairs(r.pairs, ref)
