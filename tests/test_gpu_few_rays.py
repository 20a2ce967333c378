"""Calls of few rays, whose warps take 1, 2, 4, ... 32 rays at a time: the
hits of any prefix of a ray set equal those of the whole set, in every kind of
traversal, at the counts where the number of rays a warp changes."""
import numpy as np
import pytest

from obvhs_gb300 import scenes as S
from obvhs_gb300 import test_util as T
from obvhs_gb300.params import BvhBuildParams
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    import obvhs_gb300 as G

    tris = S.scene1(5000)[0]
    cw = G.build_cwbvh_from_tris(tris, BvhBuildParams.medium_build())
    cw.set_triangles_compressed(tris)
    rng = np.random.default_rng(8)
    o = rng.uniform(-1.5, 1.5, size=(60_000, 3)).astype(np.float32)
    d = T.uniform_sample_sphere(rng.random(len(o)).astype(np.float32), rng.random(len(o)).astype(np.float32))
    rays = T.make_rays(o, d, 0.0, np.inf)
    nodes, pidx = cw.download()
    ids, t, _ = O.traverse(nodes, pidx, tris, rays, nthreads=16)
    return G, cw, rays, ids, t, cw.ray_traverse_compressed(rays)


# 8 warps an SM: the line between k and 2k rays a warp is 8 k SMs (1216 k on 152 SMs)
COUNTS = [1, 2, 31, 33, 100, 1215, 1216, 1217, 2432, 2433, 4865, 9729, 19456, 19457, 38912, 60_000]


@pytest.mark.parametrize("n", COUNTS)
def test_prefixes(scene, n):
    G, cw, rays, ids, t, (cids, ct) = scene
    i, tt = cw.ray_traverse(rays[:n])
    assert np.array_equal(i, ids[:n]) and np.array_equal(tt.view(np.uint32), t[:n].view(np.uint32))
    assert np.array_equal(cw.ray_traverse_miss(rays[:n]), ids[:n] == 0xFFFFFFFF)
    i, tt = cw.ray_traverse_compressed(rays[:n])
    assert np.array_equal(i, cids[:n]) and np.array_equal(tt.view(np.uint32), ct[:n].view(np.uint32))
    i, tt = G.ray_traverse_multi([cw, cw], (np.arange(n) % 2).astype(np.uint32), rays[:n])
    assert np.array_equal(i, ids[:n]) and np.array_equal(tt.view(np.uint32), t[:n].view(np.uint32))
