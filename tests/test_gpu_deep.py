"""Graphs of large diameter (paths, grids, combs, trees): union-find trees that are deep when the labels are
taken.  Every component is known from the construction, so the label is its smallest id."""
import numpy as np
import pytest

from graphine_b200 import gre as G
from graphine_b200 import partition as PT

pytestmark = pytest.mark.gpu


def path(n):
    return n, np.arange(n - 1), np.arange(1, n)


def grid(side):
    i = np.arange(side * side)
    right, down = i[i % side != side - 1], i[i < side * (side - 1)]
    return side * side, np.concatenate([right, down]), np.concatenate([right + 1, down + side])


def comb(spine, tooth):
    s = np.arange(spine)
    t = spine + s[:, None] * tooth + np.arange(tooth)
    u = np.concatenate([s[:-1], s, t[:, :-1].ravel()])
    return spine * (tooth + 1), u, np.concatenate([s[1:], t[:, 0], t[:, 1:].ravel()])


def tree(n, window, rng):
    """Every vertex hangs under one of the `window` before it (0: under any)."""
    i = np.arange(1, n)
    back = rng.integers(0, window, n - 1) if window else (rng.random(n - 1) * i).astype(np.int64)
    return n, np.maximum(0, i - 1 - back), i


def star(n):
    return n, np.zeros(n - 1, int), np.arange(1, n)


def pieces(size, hub, rng):
    """Components of each shape, `size` vertices each, some small ones and a star: arcs and component of each vertex."""
    side = int(size**0.5)
    parts = [path(size), grid(side), comb(side, side - 1), tree(size, 0, rng), tree(size, 8, rng)]
    parts += [path(1 + i % 7) for i in range(50)] + [star(1 + hub)]
    base = np.cumsum([0] + [p[0] for p in parts])
    u = np.concatenate([p[1] + b for p, b in zip(parts, base)])
    v = np.concatenate([p[2] + b for p, b in zip(parts, base)])
    return int(base[-1]), u, v, np.repeat(np.arange(len(parts)), np.diff(base))


def deep_forest(size, ids, directed, seed, hub=0):
    rng = np.random.default_rng(seed)
    n, u, v, comp = pieces(size, hub, rng)
    order = np.arange(n) if ids == "rising" else np.arange(n)[::-1] if ids == "falling" else rng.permutation(n)
    u, v = order[u], order[v]
    if directed:
        turn = rng.random(len(u)) < 0.5  # weakly connected: the direction says nothing
        u, v = np.where(turn, v, u), np.where(turn, u, v)
    else:
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    at = np.argsort(u, kind="stable")
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(u, minlength=n))
    low = np.full(comp.max() + 1, n)
    np.minimum.at(low, comp, order)
    want = np.empty(n, np.uint32)
    want[order] = low[comp]
    return n, off, v[at].astype(np.uint32), want


@pytest.mark.parametrize("reorder", [False, True])
@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("ids", ["rising", "falling", "mixed"])
@pytest.mark.parametrize("size", [900, 200000])
def test_components_of_deep_graphs(size, ids, directed, reorder):
    n, off, col, want = deep_forest(size, ids, directed, size)
    g = G.Graph.from_csr(n, off, col, symmetric=not directed)
    if reorder:
        g.reorder()
    for _ in range(20):  # the threads meet differently every time
        np.testing.assert_array_equal(G.cc(g)[0], want)


@pytest.mark.parametrize("directed,reorder", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("size", [900, 70000])
@pytest.mark.parametrize("hub", [255, 256, 5000])
def test_components_of_deep_graphs_beside_a_hub(hub, size, directed, reorder):
    """On either side of the degree from which first arcs are taken as they are."""
    n, off, col, want = deep_forest(size, "rising", directed, hub, hub)
    g = G.Graph.from_csr(n, off, col, symmetric=not directed)
    if reorder:
        g.reorder()
    for _ in range(5):
        np.testing.assert_array_equal(G.cc(g)[0], want)


# (mixed ids over several parts cut every path everywhere: a round for each cut that a label has to cross)
@pytest.mark.parametrize("directed,reorder", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("parts,size,ids", [(1, 900, "falling"), (1, 40000, "rising"), (1, 40000, "mixed"), (2, 900, "falling"),
                                            (2, 40000, "rising"), (3, 900, "mixed"), (3, 40000, "rising")])
def test_partitioned_components_of_deep_graphs(size, ids, directed, reorder, parts):
    n, off, col, want = deep_forest(size, ids, directed, size)
    g = G.Graph.from_csr(n, off, col, symmetric=not directed)
    if reorder:
        g.reorder()

    def job(part, exchange):
        return [part.cc(exchange)[0] for _ in range(10 if parts == 1 else 2)]

    for labels in PT.run_local(g, parts, job):
        for got in labels:
            np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("arcs", [(1 << 18) - 1, 1 << 18, 600000, (1 << 22) - 1, 1 << 22])
def test_components_of_directed_hubs(arcs):
    """On either side of the sizes between which a directed graph's bins are visited one after the other: two halves,
    each with a hub of large id, rows of every bin, and vertices that no arc meets."""
    rng = np.random.default_rng(arcs)
    n = arcs // 4
    half = n // 2
    u = np.concatenate([np.repeat([half - 1, n - 1], arcs // 8), (rng.random(arcs - 2 * (arcs // 8)) ** 4 * half).astype(np.int64)])
    v = rng.integers(0, half - 20, arcs)
    top = (u >= half) | ((u < half - 1) & (rng.random(arcs) < 0.5))
    u, v = np.where(top & (u < half), u + half, u), np.where(top, v + half, v)
    at = np.argsort(u, kind="stable")
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(u, minlength=n))
    g = G.Graph.from_csr(n, off, v[at].astype(np.uint32))
    want = np.arange(n)
    while True:  # weak components: labels both ways, and along the labels
        low = want.copy()
        np.minimum.at(low, v, want[u])
        np.minimum.at(low, u, low[v])
        low = low[low]
        if (low == want).all():
            break
        want = low
    for _ in range(5):
        np.testing.assert_array_equal(G.cc(g)[0], want.astype(np.uint32))


def weak_labels(n, u, v):
    want = np.arange(n)
    while True:  # labels both ways, and along the labels
        low = want.copy()
        np.minimum.at(low, v, want[u])
        np.minimum.at(low, u, low[v])
        low = low[low]
        if (low == want).all():
            return want.astype(np.uint32)
        want = low


# arcs and vertices around the limits of the forms for rows of about one length: four arcs a vertex, 2^16, 2^21 and 2^22 arcs
@pytest.mark.parametrize("n,arcs", [(3000, 11999), (3000, 12000), (5000, (1 << 16) - 1), (5000, 1 << 16), (16385, 1 << 16), (150000, 450000), (700000, (1 << 21) - 1), (700000, 1 << 21),
                                    (200000, (1 << 22) - 1), (200000, 1 << 22)])
def test_components_of_directed_graphs_without_hubs(n, arcs):
    """Several parts that no arc joins, rows of about one length with some of none; the same graph before and after
    it is relabelled, whose rows are binned anew."""
    rng = np.random.default_rng(arcs)
    part = np.sort(rng.integers(0, 7, n))
    lo, hi = np.searchsorted(part, part), np.searchsorted(part, part, side="right")
    u = rng.integers(0, n, arcs)
    u -= (u % 11 == 0) & (u > 0)
    v = lo[u] + (rng.random(arcs) * (hi - lo)[u]).astype(np.int64)
    mix = rng.permutation(n)
    u, v = mix[u], mix[v]
    at = np.argsort(u, kind="stable")
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(u, minlength=n))
    g = G.Graph.from_csr(n, off, v[at].astype(np.uint32))
    want = weak_labels(n, u, v)
    for _ in range(5):
        np.testing.assert_array_equal(G.cc(g)[0], want)
    g.reorder()
    for _ in range(5):
        np.testing.assert_array_equal(G.cc(g)[0], want)
