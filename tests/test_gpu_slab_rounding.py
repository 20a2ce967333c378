"""The slab test keeps the reference's two roundings (a product, then a sum)
per plane: a fused one moves a plane's distance by an ulp, which decides rays
that graze a box.  Rays aimed at triangle vertices meet boxes exactly at their
corners, where the hit is decided by that last bit; ids and t are compared
with the oracle's bit for bit."""
import numpy as np
import pytest

from obvhs_gb300 import scenes as S
from obvhs_gb300 import test_util as T
from obvhs_gb300.params import BvhBuildParams
from oracle import oracle as O

import instances as I

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import obvhs_gb300 as g

    return g


def _rays_at_vertices(tris, n, seed):
    v = tris.reshape(-1, 3)
    rng = np.random.default_rng(seed)
    target = v[rng.integers(0, len(v), size=n)]
    lo, hi = v.min(0), v.max(0)
    o = rng.uniform(lo - (hi - lo), hi + (hi - lo), size=(n, 3)).astype(np.float32)
    return T.make_rays(o, target - o, 0.0, np.inf)


@pytest.mark.parametrize("scene", ["boxes", "soup", "walls"])
def test_rays_at_vertices_match_oracle(G, scene):
    if scene == "boxes":  # corners on a grid: box planes at vertex coordinates
        rng = np.random.default_rng(3)
        c = rng.integers(-40, 40, size=(3000, 1, 3)).astype(np.float32) * np.float32(0.3)
        tris = (c + T.CUBE.reshape(12, 3, 3)[rng.integers(0, 12, size=3000)] * np.float32(0.1)).reshape(-1, 9)
    elif scene == "soup":
        tris = S.scene1(4000)[0]
    else:
        tris = S.scene3_tris(20_000)
    cw = G.build_cwbvh_from_tris(tris, BvhBuildParams.medium_build())
    nodes, pidx = cw.download()
    rays = _rays_at_vertices(tris, 400_000, 5)
    ids, t = cw.ray_traverse(rays)
    oids, ot, _ = O.traverse(nodes, pidx, tris, rays, nthreads=16)
    assert (oids != 0xFFFFFFFF).sum() > len(rays) // 10
    assert np.array_equal(ids, oids)
    assert np.array_equal(t.view(np.uint32), ot.view(np.uint32))
    miss = cw.ray_traverse_miss(rays)
    assert np.array_equal(miss, ids == 0xFFFFFFFF)


def test_rays_at_instance_vertices_match_oracle(G):
    blas_tris = I.instanced_scene(12, seed=21)
    blas = [G.build_cwbvh_from_tris(t, BvhBuildParams.medium_build()) for t in blas_tris]
    tlas = G.build_cwbvh(I.instance_boxes(blas_tris), I.tlas_params(1))
    rays = _rays_at_vertices(np.concatenate(blas_tris), 200_000, 6)
    g, p, orig, t = tlas.ray_traverse_tlas_blas(blas, rays)
    tn, tp = tlas.download()
    ob = [(*b.download(), tr) for b, tr in zip(blas, blas_tris)]
    og, op, oo, ot = O.traverse_tlas(tn, tp, ob, rays, nthreads=16)
    assert np.array_equal(g, og) and np.array_equal(p, op) and np.array_equal(orig, oo)
    assert np.array_equal(t.view(np.uint32), ot.view(np.uint32))
