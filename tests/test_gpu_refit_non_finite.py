"""A refit after some elements' coordinates became NaN or infinite (a rebuild refuses them, a refit does not look): an
element whose slab is not a number overlaps nothing, and the elements that share its bucket or its query group keep all
their pairs. The pair set must be the oracle's over the finite elements, bit for bit."""
import numpy as np
import pytest

import distbvh_b200 as bvhg
from distbvh_b200 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

FORMS = [(6, bvhg.PLAIN_FP64), (18, bvhg.PLAIN_FP64), (26, bvhg.PLAIN_FP64), (18, bvhg.FILTER_FP32)]


def expected(a, b, k):
    ia, ib = (np.flatnonzero(np.isfinite(x).all(axis=(1, 2))).astype(np.uint64) for x in (a, b))
    p = orc.pair_set(np.ascontiguousarray(a[ia]), np.ascontiguousarray(b[ib]), k)
    return np.stack([ia[p[:, 0]], ib[p[:, 1]]], axis=1)


def spoil(xyz, perm, ranks, value):
    out = xyz.copy()
    out[perm[ranks]] = value
    return out


@pytest.mark.parametrize("k,precision", FORMS)
@pytest.mark.parametrize("V", [3, 4, 5, 8])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("n,size", [(1003, 0.05), (6007, 0.007)])
def test_neighbours_of_a_non_finite_element(k, precision, V, value, n, size):
    """The first element of many buckets and groups, a whole bucket, and the last element of the ragged one; objects in
    dense and in sparse contact, alone (narrow packets) and in a batch (packets of 32)."""
    a = meshes.random_soup(n, V, seed=7, size=size)
    b = meshes.random_soup(n + 20, V, seed=8, size=size, stream=1)
    with bvhg.Context(k=k, precision=precision) as ctx:
        oa, ob = ctx.object(), ctx.object()
        for rep in range(2):  # the second build of dense objects stores their slabs
            for o, x in ((oa, a), (ob, b)):
                ctx.set_elements(o, x)
                ctx.build(o)
            assert ctx.broadphase(oa, ob).shape[0] > 30
        ranks = np.unique(np.concatenate([[0, 9, 100, n - 1], np.arange(320, 328), 8 * np.arange(n // 16) + n // 16 * 8]))
        a2 = spoil(a, ctx.morton(oa, n)[1], ranks, value)
        b2 = spoil(b, ctx.morton(ob, n + 20)[1], ranks, value)
        for x, y in ((a2, b), (a, b2), (a2, b2)):
            want = expected(x, y, k)
            assert want.shape[0] > 10
            ctx.set_elements(oa, x)
            ctx.set_elements(ob, y)
            ctx.build(oa, bvhg.REFIT)
            ctx.build(ob, bvhg.REFIT)
            assert np.array_equal(orc.canonical(ctx.broadphase(oa, ob)), orc.canonical(want))
            assert np.array_equal(orc.canonical(ctx.broadphase(ob, oa)), orc.canonical(want[:, ::-1]))
            for _ in range(2):
                got = ctx.batch_broadphase([(oa, ob)], mode=bvhg.REFIT)
                assert np.array_equal(orc.canonical(got[0]), orc.canonical(want))
            if precision == bvhg.PLAIN_FP64:
                ctx.validate_tree(oa)
                ctx.validate_tree(ob)
