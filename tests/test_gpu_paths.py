"""The kernels' own edges: tiles, remainders and the sizes at which a dispatch changes path."""
import numpy as np
import pytest

from graphine_b200 import gre as G

pytestmark = pytest.mark.gpu


def rows_graph(degrees, n, seed):
    """A directed graph in which in-row i has degrees[i] arcs (columns drawn with a seed)."""
    rng = np.random.default_rng(seed)
    dst = np.repeat(np.arange(len(degrees)), degrees)
    src = rng.integers(0, n, len(dst))
    order = np.argsort(src, kind="stable")
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(src, minlength=n))
    return off, dst[order].astype(np.uint32)


def pagerank_ref(n, off, col, iters, base, d=0.85):
    """Power iteration in float64 for the columns of `base` (n x k)."""
    src = np.repeat(np.arange(n), np.diff(off.astype(np.int64)))
    deg = np.diff(off.astype(np.int64))
    x = base.copy()
    for _ in range(iters):
        c = x / np.maximum(deg, 1)[:, None]
        s = np.stack([np.bincount(col, weights=c[src, j], minlength=n) for j in range(x.shape[1])], axis=1)
        x = base + d * s
    return x


# degrees at and around every limit of the schedule lanes 2, CTA from 33, chunks of 64
EDGES = [0, 1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 34, 63, 64, 65, 127, 128, 129, 300, 1024, 1025]


@pytest.mark.parametrize("schedule", ["", "2,32,64,0", "2,32,64,100", "8,512,65536,0"])
@pytest.mark.parametrize("rows", [1, 23, 300, 5000])
def test_rows_of_every_bin_in_one_launch(monkeypatch, schedule, rows):
    """A superstep's bins share a launch: rows at the limits of each bin, from one row to several
    blocks of each; the plain and the batched personalised form (rows of 513-1024 arcs may sit in
    the CTA bin).  Positive sums of at most 1025 terms in float64: 1025 eps relative at most."""
    if schedule:
        monkeypatch.setenv("GRE_ROW_SCHEDULE", schedule)
    degrees = [EDGES[(7 * i + 3) % len(EDGES)] for i in range(rows)]
    n = max(rows, 400)
    off, col = rows_graph(degrees, n, rows)
    g = G.Graph.from_csr(n, off, col)
    ref = pagerank_ref(n, off, col, 6, np.full((n, 1), 0.15))[:, 0]
    pr, _ = G.pagerank(g, G.PR_ITER, 0.85, 6)
    assert np.max(np.abs(pr - ref) / ref) <= 6 * 1025 * 2.3e-16
    if rows <= 300:
        seeds = np.array([0, 5, 399, 17], np.uint32)
        base = np.zeros((n, 4))
        base[seeds, np.arange(4)] = 0.15
        ref = pagerank_ref(n, off, col, 4, base).T
        out, _ = G.ppr(g, seeds, 0.85, 4)
        assert np.max(np.abs(out.reshape(4, n) - ref)) <= 4 * 1025 * 2.3e-16


@pytest.mark.parametrize("reorder", [False, True])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 257, 4000])
def test_components_whatever_the_first_arc(n, reorder):
    """Rows in any order, first arcs to larger ids, a hub with the largest id, isolated vertices, many
    components: labels equal the smallest caller id of each component."""
    rng = np.random.default_rng(n)
    part = rng.integers(0, max(1, n // 40) + 1, n)
    u = rng.integers(0, n, 2 * n)
    v = rng.integers(0, n, 2 * n)
    keep = part[u] == part[v]
    star = np.flatnonzero(part == part[n - 1])[::2]
    u, v = np.concatenate([u[keep], np.full(len(star), n - 1)]), np.concatenate([v[keep], star])
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((rng.random(len(src)), src))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(src, minlength=n))
    g = G.Graph.from_csr(n, off, dst[order].astype(np.uint32), symmetric=True)
    if reorder:
        g.reorder()
    want = np.arange(n)
    while True:
        low = want.copy()
        np.minimum.at(low, src, want[dst])
        if (low == want).all():
            break
        want = low
    np.testing.assert_array_equal(G.cc(g)[0], want.astype(np.uint32))


def bfs_ref(n, off, col, roots):
    level = np.full(n, -1, np.int32)
    level[roots] = 0
    front, d = np.unique(roots), 0
    while len(front):
        d += 1
        heads = np.concatenate([col[int(off[u]):int(off[u + 1])] for u in front] + [np.empty(0, np.uint32)])
        front = np.unique(heads[level[heads] < 0])
        level[front] = d
    return level


def shaped_graph(n, seed, directed):
    """A star with a row at the limit of a queue item, a long path, dense and sparse random parts,
    vertices without arcs, in any id order."""
    rng = np.random.default_rng(seed)
    ids = rng.permutation(n)
    u, v = [], []
    hub = min(n - 1, [127, 128, 129, 1000][seed % 4])
    u += [0] * hub
    v += list(range(1, hub + 1))
    p = n // 3  # a path from the hub's last leaf
    u += list(range(hub, min(n - 1, hub + p)))
    v += list(range(hub + 1, min(n, hub + p + 1)))
    k = 6 * n
    a, b = rng.integers(0, max(1, n // 4), k), rng.integers(0, max(1, n // 2), k)
    u, v = np.concatenate([u, a]).astype(np.int64), np.concatenate([v, b]).astype(np.int64)
    u, v = ids[u], ids[v]
    if not directed:
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    keys = np.unique(u * n + v)
    keys = keys[keys // n != keys % n]
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(keys // n, minlength=n))
    return off, (keys % n).astype(np.uint32), ids


@pytest.mark.parametrize("directed,reorder", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("n", [1, 2, 33, 127, 128, 129, 1100, 5000, 70000])
def test_bfs_shapes(n, directed, reorder):
    """Levels of single and several roots (some twice, some without arcs) equal a plain BFS's."""
    off, col, ids = shaped_graph(n, n, directed)
    g = G.Graph.from_csr(n, off, col, symmetric=not directed)
    if reorder:
        g.reorder()
    roots = np.array([ids[0], ids[n - 1], ids[n // 2], ids[n - 1]], np.uint32)
    lv, _ = G.bfs(g, roots)
    for i, r in enumerate(roots):
        np.testing.assert_array_equal(lv[i * n:(i + 1) * n], bfs_ref(n, off, col, [r]))
    one, st = G.bfs(g, roots[:1])
    np.testing.assert_array_equal(one, lv[:n])
    assert st.active == [int((one == d).sum()) for d in range(1, st.supersteps + 2)]
    many, st = G.bfs_multiroot(g, roots)
    np.testing.assert_array_equal(many, bfs_ref(n, off, col, roots))
    deg = np.diff(off.astype(np.int64))
    assert st.traversed_edges == deg[many >= 0].sum() // (1 if directed else 2)


@pytest.mark.parametrize("n", [300, 4099, 66000])
def test_bfs_directed_sources_only(n):
    """Half of the vertices have out-arcs only: nobody's parent, though they never become visited."""
    rng = np.random.default_rng(n)
    u, v = rng.integers(0, n, 16 * n), rng.integers(0, n // 2, 16 * n)
    keys = np.unique(u * n + v)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(keys // n, minlength=n))
    col = (keys % n).astype(np.uint32)
    g = G.Graph.from_csr(n, off, col)
    for r in (0, n - 1):
        np.testing.assert_array_equal(G.bfs(g, [r])[0], bfs_ref(n, off, col, [r]))


def sssp_ref(n, off, col, w, src):
    inf = np.iinfo(np.int64).max // 2
    d = np.full(n, inf)
    d[src] = 0
    u = np.repeat(np.arange(n), np.diff(off.astype(np.int64)))
    while True:
        new = d.copy()
        np.minimum.at(new, col, d[u] + w)
        if (new == d).all():
            return np.where(d >= inf, 0xFFFFFFFF, d).astype(np.uint32)
        d = new


@pytest.mark.parametrize("wide", ["0", "1000", "1000000000000"], ids=["wide", "mixed", "narrow"])
@pytest.mark.parametrize("binned", ["0", "16"], ids=["loop", "bins"])
@pytest.mark.parametrize("delta", ["", "0", "7", "100000"], ids=["auto", "none", "7", "100000"])
@pytest.mark.parametrize("n,directed", [(2, False), (130, True), (1100, False), (1100, True), (20000, True), (20000, False)])
def test_sssp_shapes(monkeypatch, n, directed, delta, binned, wide):
    """Every form of a pass (classified on the spot, as bits, through the bins) at every kind of bucket:
    distances equal a plain Bellman-Ford's; zero weights, sinks, long paths and unreached vertices."""
    monkeypatch.setenv("GRE_SSSP_WIDE", wide)
    monkeypatch.setenv("GRE_SSSP_BINNED", binned)
    if delta:
        monkeypatch.setenv("GRE_SSSP_DELTA", delta)
    off, col, ids = shaped_graph(n, n, directed)
    rng = np.random.default_rng(n)
    w = rng.integers(0, 256, len(col)).astype(np.uint32)
    w[rng.random(len(col)) < 0.02] = 100000
    g = G.Graph.from_csr(n, off, col, symmetric=not directed)
    g.loadEdgeProperty(w)
    if n == 1100:
        g.reorder()
    srcs = [int(ids[0]), int(ids[n - 1])]
    d, _ = G.sssp(g, srcs)
    for i, s in enumerate(srcs):
        np.testing.assert_array_equal(d[i * n:(i + 1) * n], sssp_ref(n, off, col, w, s))


@pytest.mark.parametrize("iters", [0, 1, 2, 5])
@pytest.mark.parametrize("k", [1, 31, 32, 33, 64, 65, 96, 97, 130])
@pytest.mark.parametrize("reorder", [False, True])
def test_ppr_slices(k, iters, reorder):
    """Slices of 64 and 32 vectors, full and ragged, rows shorter and longer than a warp's width and
    than a chunk; seeds twice, without in-arcs and without out-arcs."""
    degrees = [0, 1, 7, 8, 9, 31, 32, 33, 40, 64, 65, 1023, 1024, 1025, 2100, 0, 3] * 3
    n = 333
    off, col = rows_graph(degrees, n, k)
    g = G.Graph.from_csr(n, off, col)
    if reorder:
        g.reorder()
    seeds = np.random.default_rng(k).integers(0, n, k).astype(np.uint32)
    seeds[: min(3, k)] = [0, 332, 14][: min(3, k)]
    base = np.zeros((n, k))
    base[seeds, np.arange(k)] = 0.15
    ref = pagerank_ref(n, off, col, iters, base).T
    out, _ = G.ppr(g, seeds, 0.85, iters)
    # sums of at most 2100 positive terms below 1, a division and a product a superstep
    assert np.max(np.abs(out.reshape(k, n) - ref)) <= (iters + 1) * 2100 * 2.3e-16


def bc_ref(n, off, col, srcs):
    """Brandes in float64 with the framework's directions: levels over the out-arcs, path counts and
    dependencies both pulled over the in-arcs (as the reference's plugins do)."""
    u = np.repeat(np.arange(n), np.diff(off.astype(np.int64)))
    bc = np.zeros(n)
    for s in srcs:
        lev = bfs_ref(n, off, col, [s])
        sigma, dep = np.zeros(n), np.zeros(n)
        sigma[s] = 1.0
        top = lev.max()
        for d in range(1, top + 1):
            on = (lev[u] == d - 1) & (lev[col] == d)
            sigma += np.bincount(col[on], weights=sigma[u[on]], minlength=n)
        for d in range(top - 1, -1, -1):
            on = (lev[u] == d + 1) & (lev[col] == d)
            dep += np.bincount(col[on], weights=(1 + dep[u[on]]) / sigma[u[on]], minlength=n) * np.where(lev == d, sigma, 0)
        dep[s] = 0
        bc += dep
    return bc


def deep_graph(path, hub, extra, directed, seed):
    """A path that ends in a vertex with `hub` arcs to (and, some of them, from) leaves with random arcs
    between them, then a second path; `extra` vertices without arcs; in any id order.  Returns the
    vertices in that sequence too."""
    rng = np.random.default_rng(seed)
    n = path + 1 + hub + path + extra
    ids = rng.permutation(n)
    leaves = np.arange(path + 1, path + 1 + hub)
    u = [np.arange(path), np.full(hub, path), rng.choice(leaves, hub // 2, False), rng.choice(leaves, 3 * hub), np.arange(path + hub, 2 * path + hub)]
    v = [np.arange(1, path + 1), leaves, np.full(hub // 2, path), rng.choice(leaves, 3 * hub), np.arange(path + hub + 1, 2 * path + hub + 1)]
    u, v = ids[np.concatenate(u)], ids[np.concatenate(v)]
    if not directed:
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    keys = np.unique(u.astype(np.int64) * n + v)
    keys = keys[keys // n != keys % n]
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(keys // n, minlength=n))
    return n, off, (keys % n).astype(np.uint32), ids


# (path, leaves, vertices without arcs): around the head and the tail pieces of a long row, levels
# within one group of bit planes, two and three, and within and beyond the first pool of levels
DEEP = [(1, 3, 0), (3, 512, 1), (14, 513, 2), (15, 1025, 0), (40, 2500, 7), (150, 700, 300), (2100, 90, 0)]


def word_sources(n, ids, k, seed):
    srcs = np.random.default_rng(seed).integers(0, n, k).astype(np.uint32)
    first = [ids[0], ids[n // 2], ids[0]]  # the first path's end, one of the leaves; one twice
    srcs[: min(3, k)] = first[: min(3, k)]
    return srcs


@pytest.mark.parametrize("directed,reorder", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("k", [1, 2, 63, 64, 65])
@pytest.mark.parametrize("shape", DEEP)
def test_word_bfs_shapes(shape, directed, reorder, k):
    """The 64-source level loop: more levels than the first planes hold, rows that go on as tails,
    sources without in-arcs, without out-arcs and twice."""
    n, off, col, ids = deep_graph(*shape, directed, k)
    g = G.Graph.from_csr(n, off, col, symmetric=not directed)
    if reorder:
        g.reorder()
    srcs = word_sources(n, ids, k, n + k)
    lv, st = G.msbfs(g, srcs)
    lv = lv.reshape(k, n)
    deg = np.diff(off.astype(np.int64))
    arcs = sum(deg[row >= 0].sum() for row in lv)
    check = range(k) if shape[0] < 100 else (0, k // 2, k - 1)
    for i in check:
        np.testing.assert_array_equal(lv[i], bfs_ref(n, off, col, [int(srcs[i])]))
    assert st.traversed_edges == (arcs if directed else arcs // 2)
    assert st.supersteps == lv.max()


@pytest.mark.parametrize("directed,reorder", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("k", [1, 3, 65])
@pytest.mark.parametrize("shape", DEEP)
def test_batched_betweenness_shapes(shape, directed, reorder, k):
    """Batched betweenness where the levels outgrow the pool, rows are longer and shorter than a chunk and
    sources coincide: equal to one source at a time, and to Brandes in float64."""
    n, off, col, ids = deep_graph(*shape, directed, k)
    g = G.Graph.from_csr(n, off, col, symmetric=not directed)
    if reorder:
        g.reorder()
    srcs = word_sources(n, ids, k, n + k)
    got, _ = G.bc(g, srcs, batched=True)
    np.testing.assert_array_equal(got, G.bc(g, srcs, batched=True)[0])
    if shape[0] < 100 or k == 1:
        np.testing.assert_array_equal(got, G.bc(g, srcs, batched=False)[0])
    if k <= 3 and shape[0] < 1000:
        # positive terms only, so that every sum, product and division costs at most half an ulp of what it
        # adds to; no more than n sums and two roundings a level follow one another, on either side
        np.testing.assert_allclose(got, bc_ref(n, off, col, srcs), rtol=2 * 3 * n * 1.2e-16, atol=0)


@pytest.mark.parametrize("schedule", ["", "2,32,64,0", "2,32,64,100", "8,512,65536,0"])
@pytest.mark.parametrize("tol,limits", [(0.0, [0, 1, 3, 4, 6, 31, 32, 33, 70]), (1e-3, [5, 28, 200]), (1e-14, [400])])
def test_weighted_solve_stops_where_it_converges(monkeypatch, schedule, tol, limits):
    """The solve looks at every fourth iteration's change: ranks and the number of iterations equal a plain
    loop's for limits around the launches' groups, and the gradients those of the formulas, over rows at the
    limits of every bin."""
    if schedule:
        monkeypatch.setenv("GRE_ROW_SCHEDULE", schedule)
    n, d = 400, 0.85
    off, col = rows_graph(EDGES * 3, n, 5)
    rng = np.random.default_rng(6)
    w, c = np.exp(rng.standard_normal(len(col))), rng.standard_normal(n)
    src = np.repeat(np.arange(n), np.diff(off.astype(np.int64)))
    s = np.bincount(src, weights=w, minlength=n)
    p = w / s[src]
    g = G.Graph.from_csr(n, off, col)
    g.set_weights_f64(w)

    def solve(base, to, frm, limit):
        x, it = base.copy(), 0
        while it < limit:
            y = base + d * np.bincount(to, weights=p * x[frm], minlength=n)
            change = np.abs(y - x).max()
            x, it = y, it + 1
            if it % 4 == 0 and change <= tol:
                break
        return x, it

    for limit in limits:
        ref, it = solve(np.full(n, 1 - d), col, src, limit)
        r, st, _ = G.pagerank_weighted(g, d, tol=tol, max_iters=limit)
        # sums of at most 1025 positive terms below the result, a product and a sum an iteration
        bound = 1100 * 2.3e-16 / (1 - d)

        def same_end(got, ref, largest):
            # a tolerance below the roundings themselves is met when they settle, not at a given iteration
            assert got == ref if not 0 < tol < bound * largest else got % 4 == 0 and got < limit

        same_end(st.supersteps, it, ref.max())
        np.testing.assert_allclose(r, ref, rtol=bound, atol=0)
        lam, gp, gw, st, _ = G.pagerank_adjoint(g, ref, c, d, tol=tol, max_iters=limit)
        ref_lam, it = solve(c, src, col, limit)
        scale = np.abs(c).max() / (1 - d)  # of every partial sum
        same_end(st.supersteps, it, scale)
        pl = np.bincount(src, weights=p * ref_lam[col], minlength=n)
        np.testing.assert_allclose(lam, ref_lam, rtol=0, atol=bound * scale)
        np.testing.assert_allclose(gp, (1 - d) * ref_lam, rtol=0, atol=bound * scale)
        f = (d * ref / np.where(s > 0, s, 1))[src]
        np.testing.assert_allclose(gw, f * (ref_lam[col] - pl[src]), rtol=0, atol=4 * bound * scale * f.max())
