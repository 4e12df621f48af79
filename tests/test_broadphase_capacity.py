"""Context.broadphase without a capacity (CPU, the library replaced by a count per pair of objects): one search per call
once the pair's count is known, whatever other pairs the program searches in between, and buffers of each pair's own size."""
import ctypes

import numpy as np
import pytest

from distbvh_b200 import _abi


class Lib:
    def __init__(self, counts):
        self.counts, self.calls = counts, []

    def bvhg_broadphase(self, h, a, b, out, capacity, cnt, mem):
        n = self.counts[a, b]
        cnt._obj.value = n
        self.calls.append((a, b, capacity))
        m = min(n, capacity)
        buf = np.ctypeslib.as_array(ctypes.cast(out, ctypes.POINTER(ctypes.c_uint64)), (2 * m,)) if m else np.empty(0)
        buf[:] = np.arange(2 * m)
        return _abi.OK if n <= capacity else _abi.ERR_OVERFLOW


@pytest.fixture
def ctx(monkeypatch):
    lib = Lib({(0, 1): 500000, (2, 3): 7, (1, 0): 0})
    monkeypatch.setattr(_abi, "lib", lib)
    c = _abi.Context.__new__(_abi.Context)
    c._h, c._pair_caps = None, {}
    c.counting = lib
    return c


def test_alternating_pairs_are_searched_once(ctx):
    for a, b in ((0, 1), (2, 3), (1, 0)) * 3:
        got = ctx.broadphase(a, b)
        n = ctx.counting.counts[a, b]
        assert got.shape == (n, 2) and np.array_equal(got.ravel(), np.arange(2 * n))
    calls = ctx.counting.calls
    assert len(calls) == 10  # the first search of the large pair ran twice
    assert all(c < 20000 for a, b, c in calls if a != 0)  # the others never take its buffer


def test_a_count_that_drifts_upwards_is_searched_once(ctx):
    ctx.broadphase(0, 1)
    before = len(ctx.counting.calls)
    for _ in range(5):
        ctx.counting.counts[0, 1] += 20000
        assert ctx.broadphase(0, 1).shape[0] == ctx.counting.counts[0, 1]
    assert len(ctx.counting.calls) == before + 5


def test_a_given_capacity_is_kept(ctx):
    assert ctx.broadphase(2, 3, capacity=7).shape == (7, 2)
    with pytest.raises(_abi.BvhgError):
        ctx.broadphase(2, 3, capacity=6)
    assert ctx.broadphase(1, 0, capacity=0).shape == (0, 2)


def test_many_pairs_are_not_all_kept(ctx):
    for i in range(10000):
        ctx.counting.counts[i, i + 1] = 3
        ctx.broadphase(i, i + 1)
    assert len(ctx._pair_caps) <= 4096
