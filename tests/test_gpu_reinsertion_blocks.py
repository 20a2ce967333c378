"""Reinsertion passes whose candidates one block ranks (512 and fewer, whole
passes in one launch) or many blocks (16,384 and fewer), and the global sort
above, at the sizes where one gives way to the next: the oracle's tree bit for
bit.  Batches: one block per scene sorts above 64M comparisons a launch.
Copies of one box give equal areas and gains, whose order is the candidates'
input order."""
import numpy as np
import pytest

from obvhs_gb300 import scenes as S
from obvhs_gb300.params import BvhBuildParams
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import obvhs_gb300 as g

    return g


def _boxes(n, kind):
    rng = np.random.default_rng(n)
    c = rng.uniform(-10, 10, size=(n, 3)).astype(np.float32)
    if kind == "ties":  # boxes of a few sizes on a coarse grid
        c = np.round(c)
        h = np.repeat(rng.integers(1, 4, size=(n, 1)), 3, 1).astype(np.float32) * np.float32(0.25)
    else:
        h = np.exp(rng.uniform(np.log(0.01), np.log(1.0), size=(n, 3))).astype(np.float32)
    return np.concatenate([c - h, c + h], 1)


def _check(G, boxes, ratio, seq=None, md=None):
    on, op, omd, _ = O.ploc(boxes, None, 6, 0, 0)
    md = md or omd
    want, stats = O.reinsertion(on, op, md, ratio, seq)
    b = G.Bvh2.upload(on, op, md)
    applied = G.ReinsertionOptimizer().run(b, ratio, seq)
    assert applied == int(stats[0])
    assert np.array_equal(b.download()[0], want)


# candidates of a pass: min(2 (floor(len * ratio * seq) + 1), len) - 1, len = 2n - 1
@pytest.mark.parametrize("kind", ["spread", "ties"])
@pytest.mark.parametrize("cand", [1, 2, 31, 511, 512, 513, 1023, 1025, 4096, 16383, 16384, 16385])
def test_candidate_counts(G, cand, kind):
    n = max(4, cand)  # len = 2n - 1 > cand
    ln = 2 * n - 1
    # the first passes search half of `cand` candidates, the last one all nodes but the root
    batch = max(1, (cand + 1) // 2 - 1)
    seq = [(batch + 0.5) / ln, (max(1, batch // 3) + 0.5) / ln, (batch + 0.5) / ln, 1.0 if cand < 2000 else 0.01]
    _check(G, _boxes(n, kind), 1.0, np.array(seq, np.float32))


@pytest.mark.parametrize("n", [2, 3, 5, 256, 257, 8192, 8193])
def test_every_node_a_candidate(G, n):
    _check(G, _boxes(n, "spread"), 1.0)


def test_more_passes_than_one_launch_takes(G):
    _check(G, _boxes(1500, "ties"), 0.05, np.linspace(1.0, 0.02, 75).astype(np.float32))


def test_unclamped_stack(G):
    _check(G, _boxes(1200, "spread"), 0.1, md=300)


@pytest.mark.parametrize("sizes", [[2, 3, 700, 150_000, 30], [300, 90_000, 5_000, 1]])
def test_segmented_candidate_sorts(G, sizes):
    """Scenes whose first passes take the global sort, then a block per scene,
    then the ranking, each equal to the scene built alone."""
    p = BvhBuildParams.medium_build()
    tris = [S.scene2_tris(n, offset=i) for i, n in enumerate(sizes)]
    for cw, t in zip(G.build_cwbvh_from_tris_segmented(tris, p), tris):
        nodes, order = cw.download()
        ob = O.build(tris=t, params=p, keep_intermediate=False)
        assert nodes.tobytes() == ob.cw_nodes.tobytes() and order.tobytes() == ob.cw_pidx.tobytes()
