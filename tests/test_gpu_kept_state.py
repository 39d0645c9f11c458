"""State that a graph keeps from one call to the next, where something changes in between."""
import numpy as np
import pytest

from graphine_b200 import gre as G

pytestmark = pytest.mark.gpu


def dense_part(n, directed, seed):
    """Random arcs within every second third of the ids (two levels reach all of it, found by pulling), the other
    vertices without arcs or, on a directed graph, with out-arcs only."""
    rng = np.random.default_rng(seed)
    on = np.flatnonzero(np.arange(n) // 3 % 2)
    u, v = rng.choice(on, 12 * n), rng.choice(on, 12 * n)
    if directed:
        off_ids = np.setdiff1d(np.arange(n), on)
        u, v = np.concatenate([u, off_ids]), np.concatenate([v, rng.choice(on, len(off_ids))])
    else:
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    keys = np.unique(u.astype(np.int64) * n + v)
    keys = keys[keys // n != keys % n]
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(keys // n, minlength=n))
    return off, (keys % n).astype(np.uint32), on


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("n", [100, 5000])
def test_batched_betweenness_after_relabelling(n, directed):
    """The frontier words kept for the batched betweenness are those of the ids that searched last."""
    off, col, on = dense_part(n, directed, n)
    srcs = np.random.default_rng(1).choice(on, 70).astype(np.uint32)
    g = G.Graph.from_csr(n, off, col, symmetric=not directed)
    before, _ = G.bc(g, srcs, batched=True)
    np.testing.assert_array_equal(before, G.bc(g, srcs, batched=False)[0])
    g.reorder()
    after, _ = G.bc(g, srcs, batched=True)
    np.testing.assert_array_equal(after, G.bc(g, srcs, batched=False)[0])
    fresh = G.Graph.from_csr(n, off, col, symmetric=not directed)
    fresh.reorder()
    np.testing.assert_array_equal(after, G.bc(fresh, srcs, batched=True)[0])


@pytest.mark.parametrize("n", [200, 3000, 40000])
def test_supersteps_that_start_early_read_the_last_values(n):
    """A superstep's blocks are on the chip before the one before has ended, and their caches may hold the buffer's
    older values: long runs of short supersteps give the same bits every time, and the ranks of a float64 loop."""
    rng = np.random.default_rng(n)
    u, v = rng.integers(0, n, 8 * n), (rng.integers(0, n, 8 * n) * rng.random(8 * n)).astype(np.int64)
    order = np.argsort(u, kind="stable")
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(u, minlength=n))
    col, deg = v[order].astype(np.uint32), np.maximum(np.bincount(u, minlength=n), 1)
    g = G.Graph.from_csr(n, off, col)
    iters, d = 120, 0.85
    x = np.full(n, 1 - d)
    for _ in range(iters):
        x = (1 - d) + d * np.bincount(col, weights=(x / deg)[u[order]], minlength=n)
    first, _ = G.pagerank(g, G.PR_ITER, d, iters)
    # sums of positive terms, a product, a quotient and a sum a superstep; errors shrink by d from one to the next
    longest = np.bincount(col, minlength=n).max()
    np.testing.assert_allclose(first, x, rtol=2 * (longest + 3) * 1.2e-16 / (1 - d), atol=0)
    for _ in range(30):
        np.testing.assert_array_equal(G.pagerank(g, G.PR_ITER, d, iters)[0], first)
    w = np.ones(len(col))
    g.set_weights_f64(w)
    weighted, _, _ = G.pagerank_weighted(g, d, tol=0.0, max_iters=iters)
    np.testing.assert_allclose(weighted, x, rtol=2 * (longest + 3) * 1.2e-16 / (1 - d), atol=0)
    for _ in range(30):
        np.testing.assert_array_equal(G.pagerank_weighted(g, d, tol=0.0, max_iters=iters)[0], weighted)


@pytest.mark.parametrize("depth,groups", [(15, 0), (16, 1), (255, 1), (256, 2), (300, 2)])
def test_word_bfs_takes_room_for_the_levels_it_meets(depth, groups):
    """Levels as bit planes, 32 bytes a vertex for every four: a search takes those that its levels need."""
    import torch

    n = 1 << 20
    off = np.minimum(np.arange(n + 1), depth).astype(np.uint64)  # a path of `depth` arcs, the rest without arcs
    g = G.Graph.from_csr(n, off, np.arange(1, depth + 1, dtype=np.uint32))
    out = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    G.msbfs(g, [depth, depth - 2], out=out)
    free = torch.cuda.mem_get_info()[0]
    G.msbfs(g, [0, 1], out=out)
    taken = free - torch.cuda.mem_get_info()[0]
    assert taken <= groups * (32 * n + (2 << 20)), f"{taken / n:.1f} bytes a vertex"
    want = np.full((2, n), -1)
    want[0, : depth + 1] = np.arange(depth + 1)
    want[1, 1 : depth + 1] = np.arange(depth)
    np.testing.assert_array_equal(out.cpu().numpy().reshape(2, n), want)


@pytest.mark.parametrize("scale,edgefactor,want", [(8, 4, (4, 4096)), (13, 16, (8, 512)), (16, 16, (8, 512))])
def test_row_schedules_below_the_tuned_sizes(monkeypatch, scale, edgefactor, want):
    """Short chains from 2^16 arcs on; with GRE_TUNE=0 the default schedule at every size."""
    assert G.Graph.rmat(scale, edgefactor, 5, True).row_schedule()[:2] == want
    monkeypatch.setenv("GRE_TUNE", "0")
    assert G.Graph.rmat(scale, edgefactor, 5, True).row_schedule() == (4, 4096, 65536, 0)


@pytest.mark.parametrize("n", [50, 3000, 45000])
@pytest.mark.parametrize("k", [65, 128, 193, 232, 300])
def test_personalised_slices_side_by_side(n, k):
    """Slices of 64 vectors run side by side on a small graph, as many as fit, then the rest: every vector has the
    bits that it has in a call of its slice alone."""
    rng = np.random.default_rng(n)
    u, v = rng.integers(0, n, 9 * n), (rng.integers(0, n, 9 * n) * rng.random(9 * n) ** 4).astype(np.int64)
    at = np.argsort(u, kind="stable")
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(u, minlength=n))
    g = G.Graph.from_csr(n, off, v[at].astype(np.uint32))
    if n == 3000:
        g.reorder()
    seeds = rng.integers(0, n, k).astype(np.uint32)
    seeds[-1] = seeds[0]
    out = G.ppr(g, seeds, 0.85, 3)[0].reshape(k, n)
    for j in range(0, k, 64):
        np.testing.assert_array_equal(out[j : j + 64].reshape(-1), G.ppr(g, seeds[j : j + 64], 0.85, 3)[0])
