"""Device pair lists that the result owns: a block of their own size beside
the join's buffer.

- Asked for twice on one handle with more than 16 pairs a point (the join's
  buffer is sized by the first call and stays with the handle).
- Where device memory ends during the sort and the call fails, nothing is left
  in its result, and the handle works on.  MISTIC_TEST_DEVICE_GROWTH sets the
  bytes a call may add to what its handle holds.
- Where it ends between the sort's scratch and that block, the list is sorted
  in the join's buffer: 16 bytes a pair instead of 24."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

import mistic
from mistic import _lib as L

pytestmark = pytest.mark.gpu


def _points(n=20000):
    return np.random.default_rng(n).random((n, 2)), 0.03


def _device_list(h, x, eps, sort):
    """(status, raw result) of one call."""
    r = L.Result()
    o = h.opts(pairs="device", sort_pairs=sort)
    st = h.lib.mistic_selfjoin(h.h, x.ctypes.data_as(ctypes.c_void_p), x.shape[0], x.shape[1], L.F64, 2, eps,
                               ctypes.byref(o), ctypes.byref(r))
    return st, r


def _host(r):
    import torch

    class View:
        __cuda_array_interface__ = {"shape": (int(r.pairs_len), 2), "typestr": "<i4", "version": 2,
                                    "data": (ctypes.cast(r.pairs, ctypes.c_void_p).value, False)}

    return torch.as_tensor(View(), device="cuda").cpu().numpy().view(np.uint32)


def test_twice_with_many_pairs_a_point():
    x, eps = _points()
    ref = O.brute_pairs(x, eps)
    assert len(ref) > 16 * len(x)
    with mistic.Handle(0) as h:
        kept = []
        for _ in range(3):
            st, r = _device_list(h, x, eps, True)
            assert st == L.OK and r.pairs_on_device and r.pairs_len == len(ref)
            kept.append(r)
        for r in kept:  # earlier lists are untouched by later calls
            assert np.array_equal(_host(r), ref)
            h.lib.mistic_result_free(ctypes.byref(r))


@pytest.mark.parametrize("room", [2, 10])
def test_a_failed_call_leaves_nothing(monkeypatch, room):
    """room: bytes a pair beyond the join's buffer (sort scratch 8, block 8)."""
    x, eps = _points()
    ref = O.brute_pairs(x, eps)
    with mistic.Handle(0) as h:
        st, r = _device_list(h, x, eps, False)  # sizes every buffer of the join
        assert st == L.OK
        h.lib.mistic_result_free(ctypes.byref(r))
        monkeypatch.setenv("MISTIC_TEST_DEVICE_GROWTH", str(room * len(ref)))
        st, r = _device_list(h, x, eps, True)
        if st != L.OK:
            assert st == L.ERR_OUT_OF_MEMORY
            assert not r.pairs and not r._owner
        h.lib.mistic_result_free(ctypes.byref(r))
        monkeypatch.delenv("MISTIC_TEST_DEVICE_GROWTH")
        st, r = _device_list(h, x, eps, True)
        assert st == L.OK and np.array_equal(_host(r), ref)
        h.lib.mistic_result_free(ctypes.byref(r))


def test_sorted_in_place_without_room_for_a_block(monkeypatch):
    x, eps = _points()
    ref = O.brute_pairs(x, eps)
    with mistic.Handle(0) as h:
        st, r = _device_list(h, x, eps, False)  # sizes every buffer of the join
        assert st == L.OK
        h.lib.mistic_result_free(ctypes.byref(r))
        monkeypatch.setenv("MISTIC_TEST_DEVICE_GROWTH", str(10 * len(ref)))
        st, r = _device_list(h, x, eps, True)
        assert st == L.OK and r.pairs_on_device
        assert np.array_equal(_host(r), ref)
        h.lib.mistic_result_free(ctypes.byref(r))
