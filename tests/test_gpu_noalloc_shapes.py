"""mistic_selfjoin_noalloc over its row classes and segment lengths: rows of 1
to 8 float4 chunks in registers, longer ones a chunk at a time, point counts
around the 32-row chunks and 256-point segments; and the plain FP64 join,
which leaves out home rows whose partial sums already exceed the bound, at odd
and even row lengths, ties on the bound included.  Pair sets are the oracle's."""
import ctypes

import numpy as np
import pytest

from helpers import canon, diff_pairs
from oracle import oracle as O

from mistic import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 33, 256, 257, 3001])
@pytest.mark.parametrize("d", [1, 4, 5, 8, 12, 16, 19, 24, 28, 32, 33, 128])
def test_noalloc_row_classes(d, n):
    torch = pytest.importorskip("torch")
    lib = L.load()
    rng = np.random.default_rng(100 * d + n)
    x = rng.normal(size=(n, d)).astype(np.float32)
    x[n // 2:] = x[:n - n // 2] + rng.normal(scale=0.05, size=(n - n // 2, d)).astype(np.float32)
    eps = 0.08 * np.sqrt(d)
    ref = O.brute_pairs(x, eps)
    xt = torch.from_numpy(x).cuda()
    buf = torch.zeros((len(ref) + 8,), dtype=torch.int64, device="cuda")
    cnt = ctypes.c_uint64(0)
    torch.cuda.synchronize()
    st = lib.mistic_selfjoin_noalloc(ctypes.c_void_p(xt.data_ptr()), n, d, L.F32, eps,
                                     ctypes.c_void_p(buf.data_ptr()), len(ref) + 8, ctypes.byref(cnt), None)
    assert st == L.OK and cnt.value == len(ref)
    got = buf[:cnt.value].cpu().numpy().view(np.uint32).reshape(-1, 2)
    assert (got[:, 0] < got[:, 1]).all()
    assert np.array_equal(canon(got), ref), diff_pairs(got, ref)


@pytest.mark.parametrize("n,d,eps", [(700, 1, 0.01), (900, 2, 0.05), (1500, 3, 0.1), (1500, 18, 0.8), (900, 19, 0.9),
                                     (400, 200, 4.2), (300, 1100, 12.5)])
def test_fp64_join_leaves_no_pair_out(handle, n, d, eps):
    x = np.random.default_rng(n + d).random((n, d))
    ref = O.brute_pairs(x, eps)
    r = handle.selfjoin(x, min(6, d), eps, mode="fp64", pairs="host", sort_pairs=True)
    assert np.array_equal(r.pairs, ref), diff_pairs(r.pairs, ref)


def test_fp64_join_on_a_grid_of_ties(handle):
    """Integer grid, ε = sqrt(2): every accepted distance but the nearest lies on the bound."""
    g = np.stack(np.meshgrid(*[np.arange(7.0)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    ref = O.brute_pairs(g, float(np.sqrt(2.0)))
    r = handle.selfjoin(g, 3, float(np.sqrt(2.0)), mode="fp64", pairs="host", sort_pairs=True)
    assert np.array_equal(r.pairs, ref), diff_pairs(r.pairs, ref)
