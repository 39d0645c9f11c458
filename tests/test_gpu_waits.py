"""The level loops' bounded waits, and several handles at work at once."""
import threading

import numpy as np
import pytest

from graphine_b200 import gre as G

pytestmark = pytest.mark.gpu


def rmat(scale, seed, directed=False, reorder=False):
    n, off, col = G.rmat_host(scale, 16, seed, not directed)
    g = G.Graph.from_csr(n, off, col, symmetric=not directed)
    if reorder:
        g.reorder()
    g.set_weights_hash(5)
    return g, G.sample_sources(off, 64, 1)


@pytest.mark.parametrize("threads", [2, 4])
def test_handles_of_several_threads(threads):
    """Every handle has its stream, and every level loop asks for all SMs at once: calls from several host threads
    give what each gives alone."""
    jobs = []
    for t in range(threads):
        g, srcs = rmat(13 + t % 3, 40 + t, reorder=t % 2 == 1)
        jobs.append((g, srcs, [
            lambda g=g, s=srcs: G.bfs(g, s[:4])[0],
            lambda g=g, s=srcs: G.sssp(g, s[:2])[0],
            lambda g=g, s=srcs: G.msbfs(g, s)[0],
            lambda g=g, s=srcs: G.bfs_multiroot(g, s[:3])[0],
            lambda g=g, s=srcs: G.bc(g, s, batched=True)[0],
            lambda g=g: G.pagerank(g, G.PR_ITER, 0.85, 10)[0],
            lambda g=g: G.cc(g)[0],
        ]))
    want = [[call() for call in calls] for _, _, calls in jobs]
    errors, start = [], threading.Barrier(threads)

    def work(t):
        try:
            start.wait()
            for turn in range(8):
                for i in range(len(jobs[t][2])):
                    k = (i + t + turn) % len(jobs[t][2])
                    np.testing.assert_array_equal(jobs[t][2][k](), want[t][k])
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    pool = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
    for p in pool:
        p.start()
    for p in pool:
        p.join()
    if errors:
        raise errors[0]


def test_many_roots_within_the_wait_budget(monkeypatch):
    """Two million roots, most of them twice: taking them is no longer than a level (budget 2 ms, default 2000)."""
    n = 1 << 21
    off = np.minimum(np.arange(n + 1), n - 1).astype(np.uint64)  # a path along the ids, directed
    g = G.Graph.from_csr(n, off, np.arange(1, n, dtype=np.uint32))
    roots = np.concatenate([np.arange(1, n, 2), np.arange(n)[::-1]]).astype(np.uint32)
    monkeypatch.setenv("GRE_GRID_WAIT_MS", "2")
    level, _ = G.bfs_multiroot(g, roots)
    np.testing.assert_array_equal(level, 0)


def test_long_row_of_another_component_within_the_wait_budget(monkeypatch):
    """A search that turns bottom-up looks at every row not reached, among them a star's: one warp is at it for some
    40 ms, twice the budget, and says so."""
    leaves, n1, ef = 4000000, 1 << 17, 32
    rng = np.random.default_rng(3)
    u, v = rng.integers(0, n1, n1 * ef), rng.integers(0, n1, n1 * ef)
    n, hub = n1 + leaves + 1, n1
    star = np.arange(hub + 1, n)
    u, v = np.concatenate([u, v, np.full(leaves, hub), star]), np.concatenate([v, u, star, np.full(leaves, hub)])
    at = np.argsort(u, kind="stable")
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(u, minlength=n))
    col = v[at].astype(np.uint32)
    g = G.Graph.from_csr(n, off, col, symmetric=True)
    want, _ = G.bfs(g, [0])
    front, level, d = np.array([0]), np.full(n, -1), 0
    level[0] = 0
    while len(front):
        d += 1
        on = np.zeros(n, bool)
        on[front] = True
        heads = v[on[u]]
        front = np.unique(heads[level[heads] < 0])
        level[front] = d
    np.testing.assert_array_equal(want, level)
    monkeypatch.setenv("GRE_GRID_WAIT_MS", "20")
    for _ in range(3):
        np.testing.assert_array_equal(G.bfs(g, [0])[0], level)


CALLS = {
    "bfs": lambda g, s: G.bfs(g, s[:2]),
    "bfs_multiroot": lambda g, s: G.bfs_multiroot(g, s[:9]),
    "sssp": lambda g, s: G.sssp(g, s[:2]),
    "msbfs": lambda g, s: G.msbfs(g, s),
    "bc": lambda g, s: G.bc(g, s, batched=True),
    "bc looped": lambda g, s: G.bc(g, s[:2], batched=False),
}


@pytest.mark.parametrize("reorder", [False, True])
@pytest.mark.parametrize("call", CALLS)
def test_a_wait_that_runs_out_leaves_the_handle_usable(monkeypatch, call, reorder):
    """A budget of nothing: every wait gives up at once, the call ends with the status, and the next calls on the same
    handle (that one, and those that share its scratch) give what they gave before."""
    g, srcs = rmat(14, 32, reorder=reorder)
    want = {name: f(g, srcs)[0] for name, f in CALLS.items()}
    monkeypatch.setenv("GRE_GRID_WAIT_MS", "0")
    for _ in range(2):
        with pytest.raises(G.GreError) as e:
            CALLS[call](g, srcs)
        assert e.value.status == G.GRE_TIMEOUT
        assert "grid barrier" in str(e.value)
    monkeypatch.delenv("GRE_GRID_WAIT_MS")
    for name in [call, *CALLS]:
        np.testing.assert_array_equal(CALLS[name](g, srcs)[0], want[name])


@pytest.mark.parametrize("directed,reorder", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("k", [1, 64])
def test_counts_of_the_level_loops_are_those_of_the_levels(k, directed, reorder):
    """Pairs found a level, supersteps and traversed edges of the 64-source BFS and of a search from several roots,
    from the levels themselves."""
    n, off, col = G.rmat_host(13, 16, 31, not directed)
    g = G.Graph.from_csr(n, off, col, symmetric=not directed)
    if reorder:
        g.reorder()
    srcs = G.sample_sources(off, k, 4)
    deg = np.diff(off.astype(np.int64))
    for levels, st in (G.msbfs(g, srcs), G.bfs_multiroot(g, srcs)):
        rows = levels.reshape(-1, n)
        # the level after the deepest is looked at too, and empty
        assert list(st.active) == [int((rows == d).sum()) for d in range(1, rows.max() + 2)]
        assert st.supersteps == rows.max()
        assert st.traversed_edges == sum(deg[row >= 0].sum() for row in rows) // (1 if directed else 2)
