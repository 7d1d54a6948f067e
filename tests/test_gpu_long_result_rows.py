"""Result rows above 8,192 entries: a point amid thousands of others that are
not near one another.

Rows of at least n / 32 entries are sorted by a bitmap of the ids, shorter ones
by a radix sort.  Points far from everything else raise n to put a row on either
side of that line; the rest of the pairs are compared with the CPU oracle."""
import numpy as np
import pytest

from helpers import diff_pairs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _star(leaves, n, d, seed, first):
    """A centre, `leaves` points at 0.99 from it, and far points; the centre at
    row 0 or anywhere.  Also the rows of the star."""
    rng = np.random.default_rng(seed)
    x = np.zeros((n, d))
    x[: leaves + 1] = rng.standard_normal((leaves + 1, d))
    x[: leaves + 1] *= 0.99 / np.linalg.norm(x[: leaves + 1], axis=1)[:, None]
    x[0] = 0.0
    x[leaves + 1:, 0] = 100.0 * np.arange(1, n - leaves)
    order = rng.permutation(n) if not first else np.concatenate([[0], 1 + rng.permutation(n - 1)])
    rows = np.flatnonzero(order <= leaves)
    return x[order], rows


@pytest.mark.parametrize("leaves,n", [(8192, 8193), (8193, 40000), (8193, 262144), (8193, 262209), (8300, 300000),
                                      (10300, 300000), (9400, 300800), (9401, 300800), (30000, 300000)])
@pytest.mark.parametrize("out", ["pairs", "csr"])
def test_one_long_row(handle, leaves, n, out):
    x, rows = _star(leaves, n, 48, leaves + n, first=out == "pairs")
    ref = rows[O.brute_pairs(np.ascontiguousarray(x[rows]), 1.0)].astype(np.uint32)  # rows ascend
    assert len(ref) >= leaves
    if out == "pairs":
        r = handle.selfjoin(x, 6, 1.0, pairs="host", sort_pairs=True)
        assert np.array_equal(r.pairs, ref), diff_pairs(r.pairs, ref)
    else:
        r = handle.selfjoin(x, 6, 1.0, csr="host")
        me = np.arange(n, dtype=np.uint32)
        i, j = np.concatenate([ref[:, 0], ref[:, 1], me]), np.concatenate([ref[:, 1], ref[:, 0], me])
        o = np.lexsort((j, i))
        assert np.array_equal(r.csr_offsets, np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.uint64))
        assert np.array_equal(r.csr_nbrs, j[o])


def test_a_lone_long_row_is_not_sorted_slowly(handle):
    """200,001 rows, one with 200,000 entries: the list takes 0.58 ms, a tenth of
    the join (2.7 ms, 0.46 of it, where one block ranked an entry a thread); a
    quarter is the limit, whatever the clocks."""
    x, _ = _star(200000, 200001, 90, 1, first=True)
    r = [handle.selfjoin(x, 6, 1.0, pairs="device", sort_pairs=True).ms for _ in range(6)]
    assert min(m["d2h"] for m in r) < 0.25 * min(m["join"] for m in r)
