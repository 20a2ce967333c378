"""Queries through the Python mirror, whose first call has room for a guessed
number of ids: answers just below, at and above the guess, as the oracle's, and
no more of the context's memory than the answer needs."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import obvhs_gb300 as g

    return g


def _tree(n):
    rng = np.random.default_rng(n)
    c = rng.uniform(-5, 5, size=(n, 3)).astype(np.float32)
    boxes = np.concatenate([c - np.float32(0.01), c + np.float32(0.01)], 1)
    nodes, order, md, _ = O.ploc(boxes, None, 6, 0, 1)
    return boxes, nodes, order, md


ALL = np.array([[-100, -100, -100, 100, 100, 100]], np.float32)
NONE = np.array([[50, 50, 50, 51, 51, 51]], np.float32)


@pytest.mark.parametrize("queries", [1, 4])
@pytest.mark.parametrize("over", [-1, 0, 1, 500])
@pytest.mark.parametrize("most", [None, 700])
def test_ids_around_the_guess(G, queries, over, most, monkeypatch):
    from obvhs_gb300 import bvh

    if most:
        monkeypatch.setattr(bvh, "QUERY_IDS_MOST", most)
    guess = min(bvh.QUERY_IDS_EACH * queries + 1024, bvh.QUERY_IDS_MOST)
    n = guess + over  # the last query reaches every leaf, the others none
    boxes, nodes, order, md = _tree(n)
    q = np.concatenate([NONE] * (queries - 1) + [ALL])
    with G.Context() as ctx:
        b = G.Bvh2.upload(nodes, order, md, ctx=ctx)
        cw = G.bvh2_to_cwbvh(b, 3, True)
        cn, cp = cw.download()
        for got, want in ((b.aabb_query(q), O.query(nodes, order, q)),
                          (b.aabb_query(q, boxes), O.query(nodes, order, q, "aabb", boxes)),
                          (cw.aabb_query(q), O.query(cn, cp, q))):
            assert len(got) == queries
            for g, w in zip(got, want):
                assert g.dtype == np.uint32 and np.array_equal(g, w)
        cw.free()
        b.free()


@pytest.mark.parametrize("kind", ["aabb", "point"])
def test_room_for_the_answer_is_enough(G, kind):
    """20,000 queries with few ids in a context of 2 MB: the guess alone would
    be 2.6 MB."""
    boxes, nodes, order, md = _tree(2000)
    rng = np.random.default_rng(1)
    q = boxes[rng.integers(0, len(boxes), 20_000)]
    q = q if kind == "aabb" else np.ascontiguousarray((q[:, :3] + q[:, 3:]) * np.float32(0.5))
    with G.Context(hbm_budget_bytes=2_000_000) as ctx:
        b = G.Bvh2.upload(nodes, order, md, ctx=ctx)
        got = b.aabb_query(q) if kind == "aabb" else b.point_query(q)
        want = O.query(nodes, order, q, kind)
        assert sum(len(w) for w in want) < 100_000
        assert all(np.array_equal(g, w) for g, w in zip(got, want))
        b.free()
