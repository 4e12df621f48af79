"""Sort-and-sweep in strips and bins (bvhg_sort_and_sweep) where they can go wrong: elements wider than many strips,
minima exactly on strip and bin borders, a degenerate second axis, all elements in one cell, and sizes of A around the
steps of the elements-per-warp rule. The pair set must be the oracle's, bit for bit."""
import numpy as np
import pytest

import distbvh_b200 as bvhg
from distbvh_b200 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def check(a, b, k=18, eps=0.0, axes=(-1, 0, 1, 2)):
    want = orc.pair_set(a, b, k, eps)
    with bvhg.Context(k=k, epsilon=eps) as ctx:
        oa, ob = ctx.object(), ctx.object()
        for o, x in ((oa, a), (ob, b)):
            ctx.set_elements(o, np.ascontiguousarray(x))
            ctx.build(o)
        for axis in axes:
            got, _ = ctx.sort_and_sweep(oa, ob, axis)
            assert np.array_equal(orc.canonical(got), want), axis
    return want.shape[0]


@pytest.mark.parametrize("k", [6, 26])
@pytest.mark.parametrize("wide", [0.1, 0.9])
def test_wide_elements(k, wide):
    a = meshes.random_soup(700, 3, seed=31, size=0.01)
    b = meshes.random_soup(900, 3, seed=32, size=0.01, stream=1)
    b[::97] = meshes.random_soup(10, 3, seed=33, size=wide, stream=2)[: b[::97].shape[0]]
    a[::101] = meshes.random_soup(7, 3, seed=34, size=wide, stream=3)[: a[::101].shape[0]]
    assert check(a, b, k) > 0 and check(b, a, k) > 0


@pytest.mark.parametrize("eps", [0.0, 1.0 / 512])
def test_minima_on_the_borders(eps):
    """Triangles on a grid of 1/256 over the unit cube: every minimum is a strip border, and neighbours touch."""
    rng = np.random.default_rng(5)
    def grid(n):
        p = rng.integers(0, 256, (n, 1, 3)).astype(np.float64)
        tri = np.array([[0, 0, 0], [1, 0, 1], [0, 1, 1]], dtype=np.float64)
        return np.ascontiguousarray(np.concatenate([(p + tri), [[[0, 0, 0], [1, 0, 0], [0, 1, 0]]],
                                                    [[[256, 256, 256], [255, 256, 256], [256, 255, 256]]]]) / 256.0)
    check(grid(4000), grid(3000), 18, eps)


def test_degenerate_axes_and_one_cell():
    a = meshes.random_soup(600, 3, seed=41, size=0.02)
    b = meshes.random_soup(500, 3, seed=42, size=0.02, stream=1)
    a2, b2 = a.copy(), b.copy()
    a2[..., 1] = b2[..., 1] = 0.25  # flat: the second axis and then the sweep axis have no extent
    check(a2, b2, 18, 0.001)
    a3, b3 = a2.copy(), b2.copy()
    a3[..., 2] = b3[..., 2] = 0.5  # a line
    check(a3, b3, 18, 0.001)
    tri = np.array([[[0.0, 0.0, 0.0], [1.0, 0.0, 0.5], [0.0, 1.0, 0.25]]])
    assert check(np.repeat(tri, 70, 0), np.repeat(tri, 40, 0)) == 70 * 40


@pytest.mark.parametrize("na", [1, 31, 4735, 4736, 9473, 160001])
def test_elements_per_warp(na):
    """One element of A per warp below 148 x 32 x 2 elements, up to 32 from 148 x 32 x 32 on."""
    a = meshes.random_soup(na, 3, seed=50, size=0.01)
    b = meshes.random_soup(3001, 4, seed=51, size=0.01, stream=1)
    check(a, b, 18, 0.0, axes=(-1,))
