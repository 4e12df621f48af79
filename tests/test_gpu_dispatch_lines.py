"""Sizes on both sides of the lines at which a search or a build changes its form: packets of 8 or 32 queries in dense
contact (18,944 queries), chunks of one or more packets in sparse contact, and builds whose launches are chained (up to
524,288 elements). Every pair set must be the oracle's, bit for bit."""
import numpy as np
import pytest

import distbvh_b200 as bvhg
from distbvh_b200 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def check(a, b, k, precision, dense):
    want = orc.pair_set(a, b, k)
    assert want.shape[0] > 20 and (want.shape[0] * 50 >= a.shape[0] + b.shape[0]) == dense
    with bvhg.Context(k=k, precision=precision) as ctx:
        oa, ob = ctx.object(), ctx.object()
        for rep in range(2):  # computed slabs, then (in dense contact) stored ones
            for o, x in ((oa, a), (ob, b)):
                if rep == 0:
                    ctx.set_elements(o, x)
                ctx.build(o)
            assert np.array_equal(orc.canonical(ctx.broadphase(oa, ob)), want), rep
            assert np.array_equal(orc.canonical(ctx.broadphase(ob, oa)), orc.canonical(want[:, ::-1])), rep
        ctx.validate_tree(oa)


@pytest.mark.parametrize("n", [18943, 18944, 18945, 18953])
@pytest.mark.parametrize("k,precision", [(18, bvhg.PLAIN_FP64), (26, bvhg.PLAIN_FP64), (18, bvhg.FILTER_FP32)])
def test_packet_width(n, k, precision):
    check(meshes.random_soup(n, 3, seed=1, size=0.015), meshes.random_soup(18945, 3, seed=2, size=0.015, stream=1), k,
          precision, True)


@pytest.mark.parametrize("precision", [bvhg.PLAIN_FP64, bvhg.FILTER_FP32])
@pytest.mark.parametrize("chunk", [1, 2, 3])
def test_chunk_of_packets(chunk, precision):
    """A chunk holds packets / (2 x 148 x 16) of them: one below 2 x 4,736 packets, two there, three from 3 x 4,736 on; the
    last packet and the last chunk ragged."""
    n = 32 * 4736 * chunk + (-33 if chunk == 1 else 7)
    check(meshes.random_soup(n, 3, seed=3, size=0.002), meshes.random_soup(5000, 3, seed=4, size=0.01, stream=1), 18,
          precision, False)


@pytest.mark.parametrize("n", [524287, 524288, 524289])
def test_chained_launches(n):
    check(meshes.random_soup(n, 3, seed=5, size=0.001), meshes.random_soup(4001, 3, seed=6, size=0.01, stream=1), 18,
          bvhg.PLAIN_FP64, False)
