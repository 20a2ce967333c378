"""A CWBVH conversion that fails leaves nothing behind: the context's next
call succeeds."""
import numpy as np
import pytest

from obvhs_gb300.params import BvhBuildParams
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_the_next_call_succeeds():
    import obvhs_gb300 as G

    rng = np.random.default_rng(2)
    c = rng.uniform(-5, 5, size=(300, 3)).astype(np.float32)
    boxes = np.concatenate([c, c + np.float32(0.1)], 1)
    nodes, order, md, _ = O.ploc(boxes, None, 6, 0, 1)
    two = nodes.reshape(-1, 32).copy()
    prims = two.view(np.uint32).reshape(-1, 8)[:, 3]
    prims[np.nonzero(prims)[0][7]] = 2  # a leaf of two primitives cannot be converted
    p = BvhBuildParams(False, 6, 1, 0.1, 0.0, 0, 3, 3.0)
    want = O.build(aabbs=boxes, params=p, keep_intermediate=False)
    with G.Context() as ctx:
        b = G.Bvh2.upload(two, order, md, ctx=ctx)
        with pytest.raises(G.ObvhsError):
            G.bvh2_to_cwbvh(b, 3, True)
        b.free()
        cw = G.build_cwbvh(boxes, p, ctx=ctx)
        got, got_order = cw.download()
        cw.free()
        assert got.tobytes() == want.cw_nodes.tobytes() and got_order.tobytes() == want.cw_pidx.tobytes()
