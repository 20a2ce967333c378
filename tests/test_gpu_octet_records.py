"""A level's record passes from the octet that wrote it to all eight lanes of
the octet that reads it: one tree converted over and over, beside a busy second
context, gives the oracle's bytes each time."""
import numpy as np
import pytest

from obvhs_gb300.params import BvhBuildParams
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 5_000, 32_768])
@pytest.mark.parametrize("reinserted", [False, True])
def test_repeated_conversions_agree(n, reinserted):
    import obvhs_gb300 as G

    rng = np.random.default_rng(n)
    c = rng.uniform(-5, 5, size=(n, 3)).astype(np.float32)
    h = np.exp(rng.uniform(-6, 0, size=(n, 3))).astype(np.float32)
    boxes = np.concatenate([c - h, c + h], 1)
    nodes, order, md, _ = O.ploc(boxes, None, 6, 0, 1)
    if reinserted:
        nodes, _ = O.reinsertion(nodes, order, md, 0.2)
    want, want_order = O.bvh2_to_cwbvh(nodes, order, 3, True)[:2]
    p = BvhBuildParams(False, 6, 1, 0.0, 0.0, 0, 3, 3.0)
    with G.Context() as ctx, G.Context() as other:
        b = G.Bvh2.upload(nodes, order, md, ctx=ctx)
        kept = []
        for _ in range(40):
            kept.append(G.build_cwbvh(boxes[: n // 2], p, ctx=other))
            cw = G.bvh2_to_cwbvh(b, 3, True)
            got, got_order = cw.download()
            cw.free()
            assert got.tobytes() == want.tobytes()
            assert got_order.tobytes() == want_order.tobytes()
        for k in kept:
            k.free()
        b.free()


@pytest.mark.parametrize("n", [300, 20_000])
def test_repeated_emission_and_child_order_agree(n):
    """The two work queues, whose items one lane waits for and others read."""
    import obvhs_gb300 as G

    rng = np.random.default_rng(n + 1)
    c = rng.uniform(-5, 5, size=(n, 3)).astype(np.float32)
    h = np.exp(rng.uniform(-6, 0, size=(n, 3))).astype(np.float32)
    boxes = np.concatenate([c - h, c + h], 1)
    nodes, order, md, _ = O.ploc(boxes, None, 6, 0, 1)
    plain, plain_order = O.bvh2_to_cwbvh(nodes, order, 3, False)
    want = O.cwbvh_order_children(plain, plain_order, boxes)
    want = want[0] if isinstance(want, tuple) else want
    with G.Context() as ctx:
        b = G.Bvh2.upload(nodes, order, md, ctx=ctx)
        for _ in range(20):
            cw = G.bvh2_to_cwbvh(b, 3, False)
            assert cw.download()[0].tobytes() == plain.tobytes()
            cw.order_children(boxes)
            assert cw.download()[0].tobytes() == want.tobytes()
            cw.free()
        b.free()
