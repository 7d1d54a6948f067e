"""Sorted pair lists and neighbour tables, row by row (rows.cu).

Rows of every length class: empty, below and at 32 (sorted several at a
time), 33 to 256 (one row in a warp's registers), up to 8,192 (shared memory)
and above (through global memory).  Tight groups a long way apart give rows of
exactly known content; a random set is compared with the CPU oracle."""
import numpy as np
import pytest

from helpers import diff_pairs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _groups(sizes, seed):
    """Points in tight groups 10 apart, rows shuffled, and the group of each row."""
    rng = np.random.default_rng(seed)
    g = rng.permutation(np.repeat(np.arange(len(sizes)), sizes))
    return np.stack([10.0 * g, np.zeros(len(g))], axis=1) + rng.random((len(g), 2)) * 0.1, g


@pytest.mark.parametrize("sizes", [
    [1] * 70 + [2, 3, 31, 32, 33, 34, 1, 1, 63, 64, 65, 66, 127, 128, 129, 130, 255, 256, 257, 258, 513],
    [5] * 200 + [1] * 33,
    [40] * 20 + [1] * 5,
    [1, 2500, 1, 300],
    [8190, 3],
    [8193],
    [8700, 40],
])
@pytest.mark.parametrize("out", ["pairs", "csr"])
def test_rows_of_every_length(handle, sizes, out):
    x, g = _groups(sizes, len(sizes))
    n = len(x)
    members = [np.flatnonzero(g == k).astype(np.uint32) for k in range(len(sizes))]
    if out == "csr":
        r = handle.selfjoin(x, 2, 1.0, csr="host")
        want = np.concatenate([members[k] for k in g])
        off = np.concatenate([[0], np.cumsum(np.array(sizes)[g])]).astype(np.uint64)
        assert np.array_equal(r.csr_offsets, off)
        assert np.array_equal(r.csr_nbrs, want)
    else:
        r = handle.selfjoin(x, 2, 1.0, pairs="host", sort_pairs=True)
        rows = [m[np.searchsorted(m, i, side="right"):] for i, m in ((i, members[k]) for i, k in enumerate(g))]
        want = np.stack([np.repeat(np.arange(n, dtype=np.uint32), [len(q) for q in rows]), np.concatenate(rows)], axis=1)
        assert np.array_equal(r.pairs, want)


@pytest.mark.parametrize("n,eps", [(2, 2.0), (33, 0.2), (4000, 0.05), (4000, 0.4)])
def test_table_and_pairs_match_the_oracle(handle, n, eps):
    x = np.random.default_rng(n).random((n, 3))
    ref = O.brute_pairs(x, eps)
    r = handle.selfjoin(x, 3, eps, pairs="host", sort_pairs=True, csr="host")
    assert np.array_equal(r.pairs, ref), diff_pairs(r.pairs, ref)
    i = np.concatenate([ref[:, 0], ref[:, 1], np.arange(n, dtype=np.uint32)])
    j = np.concatenate([ref[:, 1], ref[:, 0], np.arange(n, dtype=np.uint32)])
    o = np.lexsort((j, i))
    assert np.array_equal(r.csr_nbrs, j[o])
    assert np.array_equal(r.csr_offsets, np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.uint64))
