"""Trees made elsewhere (Bvh2.upload checks nothing): the parent links that the
CWBVH conversion follows (k_parents in obvhs_gb300/csrc/reinsertion.cu).

On the CPU a model of the link table: wherever it calls an array sound, climbs
over the links stay in the array, and the nodes below the root are a tree whose
links agree.  On the GPU: nodes that no tree names are ignored and shared nodes
in node order convert as the oracle converts them; links that lead out of range,
to the root or to a node of two parents in any other order are an error, after
which the context works."""
import numpy as np
import pytest

from oracle import oracle as O

INVALID = 0xFFFFFFFF


def links(first, prims):
    """(parents, odd) as k_parents fills them, in some order of its threads."""
    n = len(first)
    parents, odd = [INVALID] * n, False
    parents[0] = 0
    for i in np.random.default_rng(n).permutation(n):
        if prims[i]:
            continue
        f = first[i]
        if f < n - 1:
            for k in (f, f + 1):
                odd |= parents[k] != INVALID
                parents[k] = int(i)
        odd |= f >= n - 1 or f == 0
    return parents, odd


def random_array(rng, m):
    """A tree of m leaves (node 0 the root, pairs in shuffled places), then
    links of a few nodes replaced and a few nodes of no tree."""
    n = 2 * m - 1
    pairs = 1 + 2 * rng.permutation(m - 1)
    first, prims = np.zeros(n, np.int64), np.ones(n, np.int64)
    open_, at = [0], 0
    while at < m - 1:
        i = open_.pop(rng.integers(len(open_)))
        first[i], prims[i] = pairs[at], 0
        open_ += [int(pairs[at]), int(pairs[at]) + 1]
        at += 1
    extra = int(rng.integers(0, 4))
    first = np.concatenate([first, rng.integers(0, n + 6, extra)])
    prims = np.concatenate([prims, rng.integers(0, 2, extra)])
    for _ in range(int(rng.integers(0, 3))):
        i = int(rng.integers(len(first)))
        first[i] = int(rng.choice([0, rng.integers(len(first)), len(first) - 1, len(first) + 3, INVALID]))
    return first.tolist(), prims.tolist()


def test_sound_links_are_a_tree():
    rng = np.random.default_rng(3)
    sound = 0
    for _ in range(4000):
        first, prims = random_array(rng, int(rng.integers(2, 12)))
        n = len(first)
        parents, odd = links(first, prims)
        assert all(p < n or p == INVALID for p in parents)
        # what the root reaches, each node once
        seen, todo, tree = set(), [0], True
        while todo and tree:
            i = todo.pop()
            tree = i not in seen
            seen.add(i)
            if not prims[i]:
                if first[i] >= n - 1:
                    tree = False
                else:
                    todo += [first[i], first[i] + 1]
        if odd:
            continue
        sound += 1
        assert tree
        for i in seen - {0}:
            assert parents[i] in seen and i - first[parents[i]] in (0, 1)
        # a climb from a leaf outside the tree never enters it
        for i in range(n):
            if prims[i] and i not in seen:
                p, steps = parents[i], 0
                while p != INVALID and steps <= n:
                    assert p not in seen
                    p, steps = parents[p], steps + 1
    assert sound > 300


def _tree(n, reinserted):
    rng = np.random.default_rng(n)
    c = rng.uniform(-5, 5, size=(n, 3)).astype(np.float32)
    h = np.exp(rng.uniform(-6, 0, size=(n, 3))).astype(np.float32)
    nodes, order, md, _ = O.ploc(np.concatenate([c - h, c + h], 1), None, 6, 0, 1)
    if reinserted:
        nodes, _ = O.reinsertion(nodes, order, md, 0.3)
    return nodes.reshape(-1, 32).copy(), np.asarray(order, np.uint32), md


def _word(nodes, col):
    return nodes.view(np.uint32).reshape(len(nodes), 8)[:, col]


PRIMS, FIRST = 3, 7


def _unordered(nodes):
    f, i = _word(nodes, FIRST).astype(np.int64), np.arange(len(nodes))
    return bool(np.any((_word(nodes, PRIMS) == 0) & (f <= i)))


def _convert(G, ctx, nodes, order, md):
    b = G.Bvh2.upload(nodes, order, md, ctx=ctx)
    try:
        cw = G.bvh2_to_cwbvh(b, 3, True)
        out = cw.download()
        cw.free()
        return out
    finally:
        b.free()


SIZES = [3, 40, 3000, 32_768, 40_000]


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("reinserted", [False, True])
@pytest.mark.parametrize("out_of_range", [False, True])
def test_nodes_of_no_tree_are_ignored(n, reinserted, out_of_range):
    import obvhs_gb300 as G

    nodes, order, md = _tree(n, reinserted)
    want = O.bvh2_to_cwbvh(nodes, order, 3, True)
    pad = np.zeros((6, 32), np.uint8)
    ln = len(nodes)
    pad[:, :] = nodes[-1]  # a leaf ...
    # ... an inner node over two of them, and perhaps one whose children are out of range
    _word(pad, PRIMS)[:] = [1, 1, 0, 1, 0 if out_of_range else 1, 1]
    _word(pad, FIRST)[:] = [0, 1, ln + 4, 0, ln + 20 if out_of_range else 1, 2]
    more = np.concatenate([nodes, pad])
    with G.Context() as ctx:
        # links of another tree in the context's scratch
        big = _tree(50_000, True)
        _convert(G, ctx, *big)
        for _ in range(2):
            got = _convert(G, ctx, more, order, md)
            assert got[0].tobytes() == want[0].tobytes()
            assert got[1].tobytes() == want[1].tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [40, 3000, 32_768])
def test_shared_nodes_in_node_order(n):
    import obvhs_gb300 as G

    nodes, order, md = _tree(n, False)
    assert not _unordered(nodes)
    inner = np.nonzero(_word(nodes, PRIMS) == 0)[0]
    a, b = int(inner[len(inner) // 3]), int(inner[len(inner) // 2])
    _word(nodes, FIRST)[a] = _word(nodes, FIRST)[b]  # both name b's children
    room = np.concatenate([order, np.zeros(4 * n, np.uint32)])
    want = O.bvh2_to_cwbvh(nodes, room, 3, True)
    with G.Context() as ctx:
        got = _convert(G, ctx, nodes, order, md)
        assert got[0].tobytes() == want[0].tobytes()
        assert got[1].tobytes() == want[1].tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [40, 3000, 32_768, 40_000])
@pytest.mark.parametrize("reinserted", [False, True])
@pytest.mark.parametrize("link", ["past the end", "all ones", "the last node", "the root"])
def test_bad_links_are_an_error(n, reinserted, link):
    import obvhs_gb300 as G

    nodes, order, md = _tree(n, reinserted)
    good = O.bvh2_to_cwbvh(nodes, order, 3, True)
    bad = nodes.copy()
    inner = np.nonzero(_word(nodes, PRIMS) == 0)[0]
    ln = len(nodes)
    i = int(inner[-3])  # a node near the leaves
    _word(bad, FIRST)[i] = {"past the end": ln + 5, "all ones": INVALID, "the last node": ln - 1, "the root": 0}[link]
    with G.Context() as ctx:
        _convert(G, ctx, nodes, order, md)
        with pytest.raises(G.ObvhsError):
            _convert(G, ctx, bad, order, md)
        got = _convert(G, ctx, nodes, order, md)
        assert got[0].tobytes() == good[0].tobytes()
        assert got[1].tobytes() == good[1].tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [33_000, 65_537, 150_000, 400_000])
def test_trees_in_node_order(n):
    import obvhs_gb300 as G

    nodes, order, md = _tree(n, False)
    assert not _unordered(nodes)
    want = O.bvh2_to_cwbvh(nodes, order, 3, True)
    with G.Context() as ctx:
        for _ in range(3):
            got = _convert(G, ctx, nodes, order, md)
            assert got[0].tobytes() == want[0].tobytes()
            assert got[1].tobytes() == want[1].tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("link", [0, 1, INVALID])
def test_inner_node_alone_is_an_error(link):
    import obvhs_gb300 as G

    nodes = np.zeros((1, 32), np.uint8)
    _word(nodes, FIRST)[0] = link
    with G.Context() as ctx:
        _convert(G, ctx, *_tree(40, False))
        with pytest.raises(G.ObvhsError):
            _convert(G, ctx, nodes, np.zeros(1, np.uint32), 96)
