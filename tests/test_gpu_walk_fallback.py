"""The rerun of a dense search whose walk reaches its stack bound. The walk's own bound is never reached (it turns to a
depth-first walk before), so this is a defensive path, and a test hook lowers the bound: the first search over stored slabs
must then launch twice (the rerun computes its slabs), later ones once, and every pair set is the oracle's."""
import numpy as np
import pytest

import distbvh_b200 as bvhg
from distbvh_b200 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [bvhg.PLAIN_FP64, bvhg.FILTER_FP32])
@pytest.mark.parametrize("limit,first", [(1, 2), (3, 2), (0, 1)])
def test_the_rerun_happens_once(precision, limit, first):
    m = 14
    xyz = meshes.tet_lattice(m)
    even = meshes.checkerboard(m)
    a, b = np.ascontiguousarray(xyz[even]), np.ascontiguousarray(xyz[~even])
    want = orc.pair_set(a, b, 18)
    with bvhg.Context(k=18, precision=precision, stage_timing=True) as ctx:
        ctx.test_dense_stack(limit)
        oa, ob = ctx.object(), ctx.object()
        launches = []
        for rep in range(4):
            for o, x in ((oa, a), (ob, b)):
                if rep == 0:
                    ctx.set_elements(o, x)
                ctx.build(o)
            ctx.stage_times()
            assert np.array_equal(orc.canonical(ctx.broadphase(oa, ob)), want)
            launches.append(ctx.stage_times()[1]["traverse"])
        assert launches == [1, first, 1, 1]  # computed slabs, then stored ones
