"""Batches whose scenes share the recheck and id-output launches: more scenes than one running sum holds (512), most of
them empty, with scenes of no, few and many pairs side by side. Counts and pairs must be the oracle's, scene by scene."""
import numpy as np
import pytest

import distbvh_b200 as bvhg
from distbvh_b200 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nscenes", [511, 513, 1300])
@pytest.mark.parametrize("precision", [bvhg.PLAIN_FP64, bvhg.FILTER_FP32])
def test_many_uneven_scenes(nscenes, precision):
    rng = np.random.default_rng(nscenes)
    bodies = [meshes.random_soup(int(n), 3, seed=60 + i, size=0.15) + rng.integers(0, 3, 3)
              for i, n in enumerate(rng.integers(1, 60, 40))]
    bodies[7] = meshes.random_soup(900, 3, seed=59, size=0.2)  # many pairs, several groups of 32 candidates
    bodies[8] = meshes.random_soup(700, 3, seed=58, size=0.2, stream=1)
    scenes = [(int(a), int(b)) for a, b in rng.integers(0, 40, (nscenes - 2, 2))] + [(7, 8), (7, 7)]
    want = {}
    for a, b in set(scenes):
        want[a, b] = orc.self_pair_set(bodies[a], 18) if a == b else orc.pair_set(bodies[a], bodies[b], 18)
    assert any(w.shape[0] == 0 for w in want.values()) and want[7, 8].shape[0] > 1000
    with bvhg.Context(k=18, precision=precision) as ctx:
        ctx.test_batch_form(3, 2)
        objs = [ctx.object() for _ in bodies]
        for o, x in zip(objs, bodies):
            ctx.set_elements(o, x)
        for rep in range(2):
            got = ctx.batch_broadphase([(objs[a], objs[b]) for a, b in scenes])
            for s, ab in enumerate(scenes):
                assert np.array_equal(orc.canonical(got[s]), want[ab]), (rep, s, ab)
