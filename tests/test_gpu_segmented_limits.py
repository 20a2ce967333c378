"""Segmented builds where one form of their PLOC gives way to another: scenes
around the 2,048 clusters from which a CTA of its own finishes a scene (a batch
of only such scenes has no grid-wide launch), and a scene of 2^24 leaves, from
which a pass counts first and writes after a barrier.  Every tree is the
oracle's, byte for byte."""
import os

import numpy as np
import pytest

from obvhs_gb300.params import BvhBuildParams
from oracle import oracle as O

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 4


@pytest.fixture(scope="module")
def G():
    import obvhs_gb300 as g

    return g


def _tris(n, seed):
    rng = np.random.default_rng(seed)
    c = rng.random((n, 1, 3), dtype=np.float32) * np.float32(100.0)
    return (c + rng.random((n, 3, 3), dtype=np.float32) * np.float32(0.2)).reshape(n, 9)


def _check(G, scenes, p, ctx):
    out = G.build_cwbvh_from_tris_segmented(scenes, p, ctx=ctx)
    for t, cw in zip(scenes, out):
        want = O.build(tris=t, params=p, nthreads=THREADS, keep_intermediate=False)
        nodes, order = cw.download()
        assert nodes.tobytes() == want.cw_nodes.tobytes()
        assert order.tobytes() == want.cw_pidx.tobytes()
    for cw in out:
        cw.free()


@pytest.mark.parametrize("radius,threshold", [(1, 0), (6, 1), (14, 3)])
@pytest.mark.parametrize("sizes", [[2047], [2048], [2049], [2048, 2047, 5], [2049, 1, 2047, 2048, 4097],
                                   [2048, 70_000, 2049, 3, 2047]])
def test_scenes_around_the_hand_over(G, sizes, radius, threshold):
    with G.Context() as ctx:
        scenes = [_tris(n, i) for i, n in enumerate(sizes)]
        for ratio in (0.0, 0.1):
            _check(G, scenes, BvhBuildParams(False, radius, threshold, ratio, 0.0, 0, 3, 3.0), ctx)


def test_scene_of_more_leaves_than_look_back_counts(G):
    with G.Context() as ctx:
        scenes = [_tris(2048, 1), _tris((1 << 24) + 3, 2), _tris(5000, 3)]
        _check(G, scenes, BvhBuildParams(False, 2, 0, 0.0, 0.0, 0, 3, 3.0), ctx)
