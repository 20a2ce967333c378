"""The eight-lanes-a-node cost pass (trees of 65,536 nodes and fewer) on the
trees where it can go wrong: one to a few nodes, counts around the line to the
other passes, zero areas, equal costs, and each leaf size: CWBVH bytes and
primitive order as the oracle's."""
import numpy as np
import pytest

from obvhs_gb300 import test_util as T
from obvhs_gb300.params import BvhBuildParams
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import obvhs_gb300 as g

    return g


def _boxes(n, kind):
    rng = np.random.default_rng(n + 7)
    c = rng.uniform(-5, 5, size=(n, 3)).astype(np.float32)
    if kind == "points":  # every leaf of zero area: costs tie at zero
        c[: n // 8] = c[0]
        h = np.zeros((n, 3), np.float32)
    elif kind == "grid":  # equal boxes: equal costs everywhere
        c = np.round(c)
        h = np.full((n, 3), 0.5, np.float32)
    else:
        h = np.exp(rng.uniform(-6, 0, size=(n, 3))).astype(np.float32)
    return np.concatenate([c - h, c + h], 1)


# (many equal points make a tree too deep for the oracle's recursion)
CASES = [(n, k) for k in ("spread", "grid") for n in (1, 2, 3, 4, 9, 33, 1000, 32768, 32769)]
CASES += [(n, "points") for n in (1, 2, 3, 4, 9, 33, 1000)]


@pytest.mark.parametrize("n,kind", CASES)
@pytest.mark.parametrize("ratio", [0.0, 0.1])
def test_conversion_matches_oracle(G, n, kind, ratio):
    a = _boxes(n, kind)
    for mp in (1, 3):
        p = BvhBuildParams(False, 6, 1, ratio, 0.0, 0, mp, 3.0)
        ob = O.build(aabbs=a, params=p, keep_intermediate=False)
        nodes, order = G.build_cwbvh(a, p).download()
        assert nodes.tobytes() == ob.cw_nodes.tobytes()
        assert order.tobytes() == ob.cw_pidx.tobytes()


def test_costs_without_a_finite_distribution(G):
    """Boxes of infinite area leave no split: an error, as in the other passes."""
    a = _boxes(50, "spread")
    a[:, 3:] = np.finfo(np.float32).max
    a[:, :3] = -np.finfo(np.float32).max
    with G.Context() as ctx, pytest.raises(G.ObvhsError):
        G.build_cwbvh(a, BvhBuildParams(False, 6, 0, 0.0, 0.0, 0, 3, 3.0), ctx=ctx)


def test_leaf_of_two_primitives_is_an_error(G):
    on, op, md, _ = O.ploc(T.tri_aabbs(T.icosphere(1)), None, 6, 0, 0)
    nodes = on.copy()
    leaf = int(np.nonzero(nodes[:, 12:16].copy().view(np.uint32).ravel())[0][0])
    nodes[leaf, 12:16] = np.array([2], np.uint32).view(np.uint8)
    with G.Context() as ctx:
        b = G.Bvh2.upload(nodes, op, md, ctx=ctx)
        with pytest.raises(G.ObvhsError):
            G.bvh2_to_cwbvh(b, 3, True)
        b.free()
