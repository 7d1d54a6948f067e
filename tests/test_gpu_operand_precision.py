"""Operands of the K-chunked kernel for rows that the short-row kernel takes
with split ones: 31 and 32 columns, and medium rows in a batch, stay split even
where the bound would let single bf16 do (a radius near the data's own)."""
import numpy as np
import pytest

from helpers import diff_pairs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _points(n, d):
    """Uniform points in a cube, ε at 0.8 of the mean pair distance."""
    return np.random.default_rng(n + d).random((n, d)), float(0.8 * np.sqrt(d / 6.0))


@pytest.mark.parametrize("d", [31, 32])
def test_short_rows_on_the_k_chunked_kernel(handle, d):
    x, eps = _points(5000, d)
    r = handle.selfjoin(x, 2, eps, mode="bf16", pairs="host", sort_pairs=True)
    assert r.tc_kernel == "k-chunked" and r.tc_operands == "split-bf16"
    ref = O.brute_pairs(x, eps)
    assert np.array_equal(r.pairs, ref), diff_pairs(r.pairs, ref)


@pytest.mark.parametrize("d", [31, 57, 126])
def test_medium_rows_of_a_batch(handle, d):
    inst = [(*_points(n, d)[:1], 2, _points(n, d)[1]) for n in (16384, 17001)]
    res = handle.batch_selfjoin(inst, mode="bf16", pairs="host", sort_pairs=True)
    for (x, _, eps), r in zip(inst, res):
        assert r.tc_kernel == "k-chunked" and r.tc_operands == "split-bf16"
        ref = O.brute_pairs(x, eps)
        assert np.array_equal(r.pairs, ref), diff_pairs(r.pairs, ref)
