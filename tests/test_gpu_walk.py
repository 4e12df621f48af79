"""The packet walk of the traversal (computed and stored element slabs) on inputs that its steps can get wrong: packets
whose ranks lie far apart (small children are checked against every query), gathers that end exactly on or just past a
full group, survivors beyond one slab test, ragged last packets and buckets, one-bucket trees and self-collision. Every
pair set must be the oracle's, bit for bit."""
import numpy as np
import pytest

import distbvh_b200 as bvhg
from distbvh_b200 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def check(a, b, k, precision=bvhg.PLAIN_FP64, eps=0.0):
    want, want_self = orc.pair_set(a, b, k, eps), orc.self_pair_set(b, k, eps)
    with bvhg.Context(k=k, precision=precision, epsilon=eps) as ctx:
        oa, ob = ctx.object(), ctx.object()
        for rep in range(3):  # computed slabs, then (in dense contact) stored ones
            for o, x in ((oa, a), (ob, b)):
                ctx.set_elements(o, np.ascontiguousarray(x))
                ctx.build(o)
            assert np.array_equal(orc.canonical(ctx.broadphase(oa, ob)), want), rep
            assert np.array_equal(orc.canonical(ctx.broadphase(ob, oa)), orc.canonical(want[:, ::-1])), rep
        for rep in range(2):
            assert np.array_equal(orc.canonical(ctx.self_collision(ob)), want_self), rep
            ctx.build(ob)
    return want.shape[0]


FORMS = [(6, bvhg.PLAIN_FP64), (18, bvhg.PLAIN_FP64), (26, bvhg.PLAIN_FP64), (18, bvhg.FILTER_FP32), (26, bvhg.FILTER_FP32)]


@pytest.mark.parametrize("k,precision", FORMS)
def test_scattered_queries(k, precision):
    """A few elements all over a large target, and two clusters at opposite corners: union boxes that cover it."""
    b = meshes.random_soup(40000, 3, seed=1, size=0.01)
    a = meshes.random_soup(45, 3, seed=2, size=0.02, stream=1)
    assert check(a, b, k, precision) > 0
    c = np.concatenate([meshes.random_soup(17, 3, seed=3, size=0.01) * 0.02,
                        1.0 - 0.02 * meshes.random_soup(20, 3, seed=4, size=0.01)])
    check(c, b, k, precision)


@pytest.mark.parametrize("k,precision", FORMS)
@pytest.mark.parametrize("n", [(1, 1), (8, 9), (15, 16), (17, 33), (257, 8), (999, 1000)])
def test_ragged_sizes_all_overlapping(k, precision, n):
    """Every element overlaps every other: full gathers, and many more survivors than one slab test holds."""
    a = 0.4 + meshes.random_soup(n[0], 4, seed=5, size=1.0) * 0.1
    b = 0.4 + meshes.random_soup(n[1], 4, seed=6, size=1.0, stream=1) * 0.1
    check(a, b, k, precision, 0.25)


@pytest.mark.parametrize("k,precision", FORMS)
def test_mixed_extents(k, precision):
    """Needles and large elements among small ones, hexahedra against hexahedra."""
    a = meshes.random_soup(2500, 8, seed=7, size=0.02)
    b = meshes.random_soup(3100, 8, seed=8, size=0.02, stream=1)
    a[::50] = meshes.random_soup(50, 8, seed=9, size=0.3, stream=2)
    b[::31] *= np.array([1.0, 1.0, 0.01])
    assert check(a, b, k, precision) > 0
