"""Work units cut at exact candidate ranks, and the two enumerations.

A unit takes a run of candidate points that may begin and end inside a
neighbour bin, the home bin among them.  The inputs put the cuts where they
can go wrong: one bin larger than any segment, bins whose sizes are multiples
of the shortest segments (256 and 512 points) and one off them, segments that
end at a bin's last point, and bin counts on both sides of the line between
the warp-per-bin and the thread-per-bin enumeration.  Pair sets are compared
with the CPU oracle; counts of one large bin are exact by construction."""
import numpy as np
import pytest

from helpers import diff_pairs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp32", "bf16", "fp64", "tf32"])
@pytest.mark.parametrize("n", [255, 256, 257, 511, 513, 4097])
def test_one_bin_cut_across_units(handle, mode, n):
    """Near-duplicates: one bin, every pair a result."""
    x = np.random.default_rng(n).random((n, 9)) * 1e-3
    r = handle.selfjoin(x, 3, 0.5, mode=mode, pairs="host", sort_pairs=True)
    i, j = np.triu_indices(n, 1)
    assert np.array_equal(r.pairs, np.stack([i, j], axis=1).astype(np.uint32))


@pytest.mark.parametrize("mode", ["fp32", "bf16", "fp64", "tf32"])
def test_bins_of_segment_multiples(handle, mode):
    """A line of tight groups of 1, 127, 128, 255, 256, 257, 512 and 1,025
    points one ε apart: each group is a bin or two, with its neighbours on
    either side among its candidates."""
    rng = np.random.default_rng(5)
    sizes = [1, 127, 128, 255, 256, 257, 512, 1025, 1, 512, 256, 3]
    x = np.concatenate([np.array([1.0 * g, 0, 0, 0]) + rng.random((s, 4)) * 0.2 for g, s in enumerate(sizes)])
    x = x[rng.permutation(len(x))]
    eps = 0.95
    ref = O.brute_pairs(x, eps)
    r = handle.selfjoin(x, 4, eps, mode=mode, pairs="host", sort_pairs=True)
    assert np.array_equal(r.pairs, ref), diff_pairs(r.pairs, ref)


@pytest.mark.parametrize("n,d,k,eps", [(3000, 2, 2, 0.004), (20000, 2, 2, 0.0035), (9000, 3, 3, 0.02),
                                       (30000, 6, 6, 0.06), (5000, 8, 8, 0.2)])
def test_enumerations_find_every_pair(handle, n, d, k, eps):
    """Uniform points: bin counts from a few thousand to tens of thousands."""
    x = np.random.default_rng(n + d).random((n, d))
    ref = O.brute_pairs(x, eps)
    r = handle.selfjoin(x, k, eps, pairs="host", sort_pairs=True)
    assert np.array_equal(r.pairs, ref), diff_pairs(r.pairs, ref)
    s = handle.selfjoin(x, k, eps, mode="fp64", csr="host", home_sample=0)
    assert s.pairs_ij == len(ref) and s.candidates == r.candidates


@pytest.mark.parametrize("mode", ["fp32", "fp64"])
@pytest.mark.parametrize("rows,cols", [(560, 561), (640, 641), (1001, 999)])
def test_many_small_units(handle, mode, rows, cols):
    """Unit lattices whose bins hold a point or two: unit counts on both sides
    of where a warp begins to claim several units at a time.  At ε = 1.1 the
    pairs are the lattice's edges."""
    ids = np.arange(rows * cols, dtype=np.uint32).reshape(rows, cols)
    x = np.stack(np.divmod(ids.ravel(), cols), axis=1).astype(np.float64)
    edges = [(ids[:, :-1], ids[:, 1:]), (ids[:-1], ids[1:])]
    ref = np.concatenate([np.stack([a.ravel(), b.ravel()], axis=1) for a, b in edges])
    ref = ref[np.lexsort((ref[:, 1], ref[:, 0]))]
    r = handle.selfjoin(x, 2, 1.1, mode=mode, pairs="host", sort_pairs=True)
    assert np.array_equal(r.pairs, ref)


@pytest.mark.parametrize("n,d,k,eps", [(12000, 3, 3, 0.012), (24000, 4, 4, 0.04), (40000, 5, 5, 0.05),
                                       (24000, 8, 8, 0.16), (36000, 6, 4, 0.05)])
@pytest.mark.parametrize("clusters", [0, 5])
def test_threads_sharing_a_walk(handle, n, d, k, eps, clusters):
    """Bins beyond the warp-per-bin line, walked by 8, 4, 2 or one thread
    each: uniform points, and a third of them in tight groups whose long lists
    are cut into segments inside a thread's share.  The home samples add up to
    no more than the whole."""
    rng = np.random.default_rng(n + d + clusters)
    x = rng.random((n, d))
    g = n // 15
    for c in range(clusters):
        x[c * g:(c + 1) * g] = rng.random(d) + rng.random((g, d)) * eps
    ref = O.brute_pairs(x, eps)
    r = handle.selfjoin(x, k, eps, pairs="host", sort_pairs=True)
    assert np.array_equal(r.pairs, ref), diff_pairs(r.pairs, ref)
    s = handle.selfjoin(x, k, eps, pairs="host", sort_pairs=True, home_sample=3)
    assert s.candidates < r.candidates
    key = lambda p: p[:, 0].astype(np.uint64) << 32 | p[:, 1]
    assert np.isin(key(s.pairs), key(ref)).all()
