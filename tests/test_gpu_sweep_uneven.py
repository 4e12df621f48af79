"""Sort-and-sweep of unevenly spread objects (bvhg_sort_and_sweep): the cells must follow B's elements wherever they lie,
so that the cost stays that of the elements near one another, and the pair set stays the oracle's."""
import time

import numpy as np
import pytest

import distbvh_b200 as bvhg
from distbvh_b200 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def seconds(a, b):
    """The fastest of several calls, and the pairs."""
    with bvhg.Context(k=18) as ctx:
        oa, ob = ctx.object(), ctx.object()
        for o, x in ((oa, a), (ob, b)):
            ctx.set_elements(o, np.ascontiguousarray(x))
            ctx.build(o)
        best = float("inf")
        for _ in range(8):
            t = time.perf_counter()
            pairs, _ = ctx.sort_and_sweep(oa, ob)
            best = min(best, time.perf_counter() - t)
        return best, orc.canonical(pairs)


def test_cost_of_outliers_and_of_a_wide_object():
    """One element 1,000 extents away on every axis, in either object, and an A spread 100 times as wide as B. Each meets
    the same neighbours as the plain soups (or fewer), so each call takes at most twice their time; cells of even steps
    over the extents put all 262,144 elements of B into one of them (about 400 times the time)."""
    n = 262144
    a, b = meshes.random_soup(n, 3, seed=1, size=0.004), meshes.random_soup(n, 3, seed=2, size=0.004, stream=1)
    plain, pairs = seconds(a, b)
    assert pairs.shape[0] > 10000
    a_far, b_far = a.copy(), b.copy()
    a_far[7] += np.array([-1e3, 1e3, 5e2])
    b_far[5] += 1e3
    for x, y in ((a, b_far), (a_far, b), (a_far, b_far)):
        t, got = seconds(x, y)
        assert abs(got.shape[0] - pairs.shape[0]) < 10
        assert t < 2 * plain, (t, plain)
    centre = a.mean(axis=1, keepdims=True)
    t, _ = seconds((a - centre) + 100.0 * (centre - 0.5), b)
    assert t < 2 * plain, (t, plain)


def check(a, b, k, eps=0.0):
    want = orc.pair_set(a, b, k, eps)
    with bvhg.Context(k=k, epsilon=eps) as ctx:
        oa, ob = ctx.object(), ctx.object()
        for o, x in ((oa, a), (ob, b)):
            ctx.set_elements(o, np.ascontiguousarray(x))
            ctx.build(o)
        for axis in (-1, 0, 1, 2):
            got, _ = ctx.sort_and_sweep(oa, ob, axis)
            assert np.array_equal(orc.canonical(got), want), axis
    return want.shape[0]


@pytest.mark.parametrize("k", [6, 18, 26])
def test_clusters_and_tails(k):
    """Two far clusters of B, minima over ten orders of magnitude, and B on a few planes (many equal borders)."""
    rng = np.random.default_rng(3)
    a = meshes.random_soup(3000, 4, seed=11, size=0.02)
    b = meshes.random_soup(4000, 4, seed=12, size=0.02, stream=1)
    b2 = b.copy()
    b2[1::2] += 1e6
    assert check(a, b2, k) > 0
    s = 10.0 ** rng.uniform(-8, 2, (4000, 1, 1))
    assert check(a * s[:3000], b * s, k) > 0
    b3 = b.copy()
    b3[..., 0] = np.round(b3[..., 0] * 3) / 3 + 0.01 * (b[..., 0] - b[:, :1, 0])
    assert check(a, b3, k, 0.01) > 0


@pytest.mark.parametrize("nb", [1, 2, 7, 255, 256, 257, 2047, 2048, 2049, 4097])
def test_sizes_around_the_sample(nb):
    a = meshes.random_soup(1500, 3, seed=21, size=0.03)
    b = meshes.random_soup(nb, 3, seed=22, size=0.03, stream=1)
    check(a, b, 18, 0.01)
