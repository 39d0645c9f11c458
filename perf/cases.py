"""The calls that a user of this framework makes, as measured cases.

Each case is one call (or one forward and backward pair) of the Python interface on a graph the
program already holds: PageRank, BFS, SSSP, connected components and betweenness in their plain
forms, and the batched and differentiable forms beside them.  Graphs are RMAT
(a/b/c = .57/.19/.19), either made by the framework's own generator (`gen: "rmat"`, a power of two
vertices) or handed over as a CSR of any size (`gen: "list"`).  Sizes are those of the stated
configurations, the tests and the benchmark: RMAT-16 directed PageRank, RMAT-20 batches and
gradients, RMAT-22 BFS / SSSP / CC, and beyond (RMAT-24: the ranks alone are larger than L2).
Results stay in device tensors, as the benchmark's.
"""
import math

import numpy as np
import torch

from graphine_b200 import gre

DAMPING = 0.85


def listed():
    return [
        # one interactive query on a small graph: launches and latency are all there is
        dict(name="bfs_small", algo="bfs", gen="list", n=4000, ef=8, directed=False, reorder=False, k=1),
        # the stated PageRank configuration: RMAT-16, directed, 20 supersteps
        dict(name="pagerank_s16_directed", algo="pagerank", gen="rmat", n=1 << 16, ef=16, directed=True, reorder=False, iters=20),
        # ranking a graph whose ranks exceed L2
        dict(name="pagerank_s24", algo="pagerank", gen="rmat", n=1 << 24, ef=16, directed=False, reorder=True, iters=20),
        # the stated BFS configuration: RMAT-22, 16 sources one after the other
        dict(name="bfs_s22_16src", algo="bfs", gen="rmat", n=1 << 22, ef=16, directed=False, reorder=True, k=16),
        # shortest paths over a directed list of arcs with a weight each, as read from a file, ragged size
        dict(name="sssp_60k_directed", algo="sssp", gen="list", n=60000, ef=12, directed=True, reorder=False, k=1),
        # the stated SSSP configuration (RMAT-22, weights of the undirected edge), four of its sources
        dict(name="sssp_s22_4src", algo="sssp", gen="rmat", n=1 << 22, ef=16, directed=False, reorder=True, k=4),
        # the stated components configuration
        dict(name="cc_s22", algo="cc", gen="rmat", n=1 << 22, ef=16, directed=False, reorder=True),
        # one word of the stated batched betweenness (RMAT-20)
        dict(name="bc_s20_64src", algo="bc", gen="rmat", n=1 << 20, ef=16, directed=False, reorder=True, k=64),
        # the stated batched BFS
        dict(name="msbfs_s20_64src", algo="msbfs", gen="rmat", n=1 << 20, ef=16, directed=False, reorder=True, k=64),
        # the stated batch of personalisation vectors
        dict(name="ppr_s20_128", algo="ppr", gen="rmat", n=1 << 20, ef=16, directed=False, reorder=True, k=128, iters=20),
        # the stated differentiation: weighted PageRank to convergence, then its gradients
        dict(name="pagerank_grad_s20", algo="grad", gen="rmat", n=1 << 20, ef=16, directed=False, reorder=True),
        # the stated batch of uneven graphs, one BFS in each, over their union
        dict(name="batch_bfs_32graphs", algo="batch", gen="rmat", n=1 << 18, ef=16, directed=False, reorder=False, k=32),
    ]


def draw(rng):
    def log_size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    algo = rng.choice(["bfs", "pagerank", "sssp", "cc", "bc", "msbfs", "ppr", "grad", "batch"])
    if algo == "batch":
        return dict(algo=algo, gen="rmat", n=1 << rng.randint(13, 18), ef=rng.randint(6, 20), directed=False, reorder=False,
                    k=rng.randint(3, 40))
    hi = {"bfs": 2000000, "pagerank": 2000000, "sssp": 2000000, "cc": 2000000, "bc": 250000, "msbfs": 500000, "ppr": 100000,
          "grad": 120000}[algo]
    c = dict(algo=algo, gen="list", n=log_size(3000, hi), ef=rng.randint(4, 20), directed=rng.random() < 0.35,
             reorder=rng.random() < 0.6)
    if algo in ("bfs", "sssp"):
        c["k"] = rng.randint(1, 8)
    if algo in ("bc", "msbfs"):
        c["k"] = rng.randint(2, 130)
    if algo == "ppr":
        c["k"] = rng.randint(2, 200)
    if algo in ("pagerank", "ppr"):
        c["iters"] = rng.randint(5, 40)
    return c


# ----------------------------------------------------------------------------------------------
# graphs
# ----------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _arcs_of(keys, n):
    """CSR of sorted, distinct arc keys u * n + v."""
    u = torch.div(keys, n, rounding_mode="floor")
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.bincount(u, minlength=n).cumsum(0)
    return off, (keys - u * n).to(torch.int32)


def _distinct(u, v, n, directed):
    keep = u != v
    u, v = u[keep], v[keep]
    keys = u * n + v
    if not directed:
        keys = torch.cat([keys, v * n + u])
    return torch.unique(keys)


def _list_keys(case, seed):
    """An RMAT-like list of arcs over any number of vertices."""
    n, gen = case["n"], _generator(seed)
    m = n * case["ef"]
    u = torch.zeros(m, dtype=torch.int64, device="cuda")
    v = torch.zeros_like(u)
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(m, generator=gen, device="cuda")
        ub = r >= 0.76
        vb = ((r >= 0.57) & ~ub) | (r >= 0.95)
        u = u * 2 + ub
        v = v * 2 + vb
    ids = torch.randperm(n, generator=gen, device="cuda")
    return _distinct(ids[u % n], ids[v % n], n, case["directed"])


def _signed(x):
    x &= (1 << 64) - 1
    return x - (1 << 64) if x >> 63 else x


def _mix_int(x):
    x = (x + 0x9E3779B97F4A7C15) & ((1 << 64) - 1)
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & ((1 << 64) - 1)
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & ((1 << 64) - 1)
    return x ^ (x >> 31)


def _mix(x):
    """SplitMix64 of int64 tensors (the bits of uint64)."""
    def shr(y, k):
        return (y >> k) & ((1 << (64 - k)) - 1)

    x = x + _signed(0x9E3779B97F4A7C15)
    x = (x ^ shr(x, 30)) * _signed(0xBF58476D1CE4E5B9)
    x = (x ^ shr(x, 27)) * _signed(0x94D049BB133111EB)
    return x ^ shr(x, 31)


def _rmat_keys(n, ef, seed, directed, device="cuda"):
    """The arcs of the framework's seeded generator, restated for the 64-bit reference results."""
    scale, mask = n.bit_length() - 1, n - 1
    thr = [int(0.57 * 2.0**32), int((0.57 + 0.19) * 2.0**32), int((0.57 + 0.19 + 0.19) * 2.0**32)]
    shift = scale // 2 + 1
    mul = [_mix_int(seed ^ (0xA5A5 + k)) | 1 for k in range(3)]
    add = [_mix_int(seed ^ (0x5A5A + k)) for k in range(3)]

    def permute(x):
        for k in range(3):
            x = (x * _signed(mul[k])) & mask
            x = x ^ (x >> shift)
            x = (x + _signed(add[k])) & mask
        return x

    us, vs, step = [], [], 1 << 26
    for e0 in range(0, n * ef, step):
        e = torch.arange(e0, min(e0 + step, n * ef), dtype=torch.int64, device=device)
        base = _mix(_mix(e) ^ _signed(seed))
        u, v = torch.zeros_like(e), torch.zeros_like(e)
        for lev in range(0, scale, 2):
            h = _mix(base + lev)
            for t in range(2):
                if lev + t >= scale:
                    break
                r = (h >> (32 * t)) & 0xFFFFFFFF
                ub = r >= thr[1]
                vb = ((r >= thr[0]) & ~ub) | (r >= thr[2])
                u = u * 2 + ub
                v = v * 2 + vb
        us.append(permute(u).to(torch.int32))
        vs.append(permute(v).to(torch.int32))
    return _distinct(torch.cat(us).to(torch.int64), torch.cat(vs).to(torch.int64), n, directed)


def _csr(case, seed):
    """(off, col) of the case's graph without the framework."""
    n = case["n"]
    if case["gen"] == "rmat":
        return _arcs_of(_rmat_keys(n, case["ef"], seed, case["directed"]), n)
    return _arcs_of(_list_keys(case, seed), n)


def _graph(case, seed):
    if case["gen"] == "rmat":
        return gre.Graph.rmat(case["n"].bit_length() - 1, case["ef"], seed=seed, symmetric=not case["directed"], reorder=case["reorder"])
    off, col = _csr(case, seed)
    torch.cuda.synchronize()
    g = gre.Graph.from_csr(case["n"], off, col, symmetric=not case["directed"])
    if case["reorder"]:
        g.reorder()
    return g


def _sample(degree, k, seed):
    """k seeded vertices that have arcs."""
    cand = torch.nonzero(degree > 0).reshape(-1)
    pick = torch.randint(0, cand.numel(), (k,), generator=_generator(seed + 7), device="cuda")
    return cand[pick]


def _batch_scales(case):
    """Uneven scales up to the case's own, the same for every seed (the results' length is)."""
    top = case["n"].bit_length() - 1
    return [int(s) for s in np.random.RandomState(case["k"]).randint(max(8, top - 6), top + 1, case["k"])]


def _topology(case, seed):
    """Gradients are taken again and again on one topology with other weights: its seed is its own
    (the weight gradient has an entry an arc)."""
    return 20 if case["algo"] == "grad" else seed


def _degree(g):
    d = torch.empty(g.n, dtype=torch.int32, device="cuda")
    g.getOutdegree(out=d)
    return d


# ----------------------------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------------------------
def prepare(case, seed):
    algo, dev = case["algo"], "cuda"
    if algo == "batch":
        parts = [gre.Graph.rmat(s, case["ef"], seed=seed * 1000 + i, symmetric=True) for i, s in enumerate(_batch_scales(case))]
        union, offs = gre.Graph.union(parts)
        roots = [int(offs[i]) + int(_sample(_degree(p), 1, seed + i)) for i, p in enumerate(parts)]
        for p in parts:
            p.free()
        return dict(case=case, g=union, srcs=np.asarray(roots, np.uint32), out=torch.empty(union.n, dtype=torch.int32, device=dev))
    g = _graph(case, _topology(case, seed))
    n, s = g.n, dict(case=case)
    s["g"] = g
    if algo in ("bfs", "sssp", "bc", "msbfs", "ppr"):
        s["srcs"] = _sample(_degree(g), case["k"], seed).cpu().numpy().astype(np.uint32)
    if algo in ("bfs", "msbfs", "sssp"):
        s["out"] = torch.empty(case["k"] * n, dtype=torch.int32, device=dev)
    if algo == "cc":
        s["out"] = torch.empty(n, dtype=torch.int32, device=dev)
    if algo in ("pagerank", "bc"):
        s["out"] = torch.empty(n, dtype=torch.float64, device=dev)
    if algo == "ppr":
        s["out"] = torch.empty(case["k"] * n, dtype=torch.float64, device=dev)
    if algo == "sssp":
        if case["directed"]:
            g.loadEdgeProperty(torch.randint(1, 256, (g.m,), dtype=torch.int32, generator=_generator(seed + 3), device=dev))
        else:
            g.set_weights_hash(seed + 3)
    if algo == "grad":
        w, s["c"] = _weights(g.n, g.m, seed)
        g.set_weights_f64(w)
        s["r"], s["lam"], s["gp"] = (torch.empty(n, dtype=torch.float64, device=dev) for _ in range(3))
        s["gw"] = torch.empty(g.m, dtype=torch.float64, device=dev)
    return s


def _weights(n, m, seed):
    """Log-normal arc weights and the gradient of a linear loss."""
    gen = _generator(seed + 5)
    w = torch.exp(torch.randn(m, dtype=torch.float64, generator=gen, device="cuda"))
    return w, torch.randn(n, dtype=torch.float64, generator=gen, device="cuda")


def run(s):
    case, g = s["case"], s["g"]
    algo = case["algo"]
    if algo == "pagerank":
        return gre.pagerank(g, gre.PR_ITER, DAMPING, case["iters"], out=s["out"])[0]
    if algo == "bfs":
        return gre.bfs(g, s["srcs"], out=s["out"])[0]
    if algo == "msbfs":
        return gre.msbfs(g, s["srcs"], out=s["out"])[0]
    if algo == "sssp":
        return gre.sssp(g, s["srcs"], out=s["out"])[0]
    if algo == "cc":
        return gre.cc(g, out=s["out"])[0]
    if algo == "bc":
        return gre.bc(g, s["srcs"], batched=True, out=s["out"])[0]
    if algo == "ppr":
        return gre.ppr(g, s["srcs"], DAMPING, case["iters"], out=s["out"])[0]
    if algo == "batch":
        return gre.bfs_multiroot(g, s["srcs"], out=s["out"])[0]
    r = gre.pagerank_weighted(g, DAMPING, out=s["r"])[0]
    lam, gp, gw = gre.pagerank_adjoint(g, r, s["c"], DAMPING, lam=s["lam"], grad_pers=s["gp"], grad_w=s["gw"])[:3]
    return dict(rank=r, adjoint=lam, grad_pers=gp, grad_w=gw)


def work(case):
    """Bytes and FP64 operations of a pass: the topology once (once a superstep where ranks are
    iterated, since it does not fit on the chip), each input once, each output once."""
    n, m = case["n"], case["n"] * case["ef"] * (1 if case["directed"] else 2)
    algo, k, it = case["algo"], case.get("k", 1), case.get("iters", 1)
    if algo == "pagerank":
        return dict(bytes=it * (8 * (n + 1) + 4 * m + 20 * n), flops=it * (m + 3 * n))
    if algo == "bfs":  # per source: an arc that finds it, the offsets and the level of each vertex
        return dict(bytes=k * (8 * (n + 1) + 4 * n + 4 * n), flops=0)
    if algo == "msbfs":
        return dict(bytes=-(-k // 64) * (8 * (n + 1) + 4 * m) + 4 * n * k, flops=0)
    if algo == "sssp":
        return dict(bytes=k * (8 * (n + 1) + 8 * m + 4 * n), flops=0)
    if algo == "cc":
        return dict(bytes=8 * (n + 1) + 4 * n + 4 * n, flops=0)
    if algo == "bc":  # two sweeps of the topology a word of 64, path counts and dependencies written once
        return dict(bytes=-(-k // 64) * 2 * (8 * (n + 1) + 4 * m) + 16 * n * k + 8 * n, flops=4 * m * k)
    if algo == "ppr":
        return dict(bytes=it * (-(-k // 128) * (8 * (n + 1) + 4 * m) + 16 * n * k), flops=it * k * (m + 3 * n))
    if algo == "batch":
        nn = k * n // 4
        return dict(bytes=8 * nn + 8 * nn, flops=0)
    it = 300  # supersteps of the two solves together, to 1e-14
    return dict(bytes=it * (8 * (n + 1) + 12 * m + 16 * n) + 28 * m, flops=it * 2 * m)


# ----------------------------------------------------------------------------------------------
# 64-bit results without the framework
# ----------------------------------------------------------------------------------------------
def _rows(off, col):
    u = torch.repeat_interleave(torch.arange(off.numel() - 1, device=off.device), off[1:] - off[:-1])
    return u, col.to(torch.int64)


def _matrix(off, col, values):
    n = off.numel() - 1
    return torch.sparse_csr_tensor(off.to(torch.int32), col.to(torch.int32), values, (n, n), check_invariants=False)


def _transposed(off, col, values):
    n = off.numel() - 1
    u, v = _rows(off, col)
    keys, order = torch.sort(v * n + u)
    roff, rcol = _arcs_of(keys, n)
    return _matrix(roff, rcol, values[order])


def exact(case, seed):
    algo = case["algo"]
    if algo not in ("pagerank", "ppr", "bc", "grad"):
        return None  # levels, distances and labels are whole numbers
    off, col = _csr(case, _topology(case, seed))
    n, m = case["n"], col.numel()
    deg = off[1:] - off[:-1]
    ones = torch.ones(m, dtype=torch.float64, device="cuda")
    if algo in ("pagerank", "ppr"):
        pull = _matrix(off, col, ones) if not case["directed"] else _transposed(off, col, ones)
        inv = torch.where(deg > 0, 1.0 / deg.clamp(min=1).double(), torch.zeros((), dtype=torch.float64, device="cuda"))
    tele = 1.0 - DAMPING
    if algo == "pagerank":
        x = torch.full((n, 1), tele, dtype=torch.float64, device="cuda")
        for _ in range(case["iters"]):
            x = tele + DAMPING * (pull @ (x * inv[:, None]))
        return x.reshape(-1)
    if algo == "ppr":
        base = torch.zeros(n, case["k"], dtype=torch.float64, device="cuda")
        base[_sample(deg, case["k"], seed), torch.arange(case["k"], device="cuda")] = tele
        x = base
        for _ in range(case["iters"]):
            x = base + DAMPING * (pull @ (x * inv[:, None]))
        return x.t().contiguous().reshape(-1)
    if algo == "grad":
        w, c = _weights(n, m, seed)
        u, v = _rows(off, col)
        s = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, u, w)
        p = w / s[u]
        fwd, bwd = _transposed(off, col, p), _matrix(off, col, p)
        r = torch.full((n, 1), tele, dtype=torch.float64, device="cuda")
        lam = c[:, None]
        for _ in range(300):
            r = tele + DAMPING * (fwd @ r)
            lam = c[:, None] + DAMPING * (bwd @ lam)
        pl = (bwd @ lam).reshape(-1)
        r, lam = r.reshape(-1), lam.reshape(-1)
        return dict(rank=r, adjoint=lam, grad_pers=tele * lam, grad_w=DAMPING * (r / s)[u] * (lam[v] - pl[u]))
    out = torch.zeros(n, dtype=torch.float64, device="cuda")
    srcs = _sample(deg, case["k"], seed)
    push = _matrix(off, col, ones)
    pull = push if not case["directed"] else _transposed(off, col, ones)
    for j in range(0, case["k"], 64):
        out += _brandes(pull, srcs[j:j + 64], n)
    return out


def _brandes(pull, srcs, n):
    """Dependencies of a block of sources.  The framework's backward pass pulls over the in-arcs as its
    forward pass does (the reference's plugins)."""
    k = srcs.numel()
    cols = torch.arange(k, device="cuda")
    level = torch.full((n, k), -1, dtype=torch.int32, device="cuda")
    sigma = torch.zeros(n, k, dtype=torch.float64, device="cuda")
    level[srcs, cols] = 0
    sigma[srcs, cols] = 1.0
    d = 0
    while True:
        got = pull @ torch.where(level == d, sigma, 0.0)
        new = (got > 0) & (level < 0)
        if not bool(new.any()):
            break
        d += 1
        level[new] = d
        sigma = torch.where(new, got, sigma)
    dep = torch.zeros_like(sigma)
    for e in range(d - 1, -1, -1):
        got = pull @ torch.where(level == e + 1, (1.0 + dep) / sigma.clamp(min=1.0), 0.0)
        dep = torch.where(level == e, sigma * got, dep)
    dep[srcs, cols] = 0.0
    return dep.sum(1)
