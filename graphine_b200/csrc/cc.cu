// Connected components fast path: lock-free union-find with min-id hooking.
//
// The reference ConnectedComponents plugin (Kernels/CC.hpp:33-67, run<InOut>) propagates the
// minimum global vid across every arc until no label changes; the fixed point labels each
// vertex with the minimum vid of its (weakly) connected component.  Union-find reaches the
// same labels directly: every arc {u, v} unites the two trees, and a root is only ever linked
// under a smaller root (atomicCAS on the larger root's parent), so the root of each tree is
// the smallest stored id it contains.  A final pass writes find(v) for every v.  (Jayanti & Tarjan
// style concurrent union-find as used by ECL-CC, Jaiganesh & Burtscher 2018.)  On a relabelled
// graph the stored ids put the hubs first, so that nearly every link is a vertex under the
// first hub, each on its own word; the smallest caller id of each tree is then found by one pass
// over the vertices.  (Linked by caller ids instead, the root of the giant tree changes whenever a
// smaller id joins, and links and path writes meet on few words: RMAT-22 the first pass 1084 us.)
//
// Arcs are visited through the degree bins of the CSR (rows.cuh): groups of 1..32 lanes per
// row, a CTA per long row, CTA chunks for hubs, so the column reads stay coalesced.  A directed
// graph's arcs are all visited (their union is the weakly connected components).
//
// On a symmetric graph the arcs are visited the Afforest way (Sutton, Ben-Nun and Bar 2018):
// the first two arcs of every row, then the rest of the rows outside the largest component
// only; on RMAT most rows belong to it (RMAT-26: 7.8 -> 3.6 ms).
//
// Byte model: 8(n+1) offsets + 12 per visited arc (column + two parent probes, mostly L2)
// + 8n init/final labels (+ n/4 for the skip bits and their reads).
#include <algorithm>
#include <cstdlib>
#include <vector>

#include "gre_internal.cuh"
#include "rows.cuh"
#include "uf.cuh"

namespace gre {

struct HookArcs {
  const uint32_t* __restrict__ col;
  uint32_t* parent;
  // Afforest's second pass: rows flagged in `skip` (null: none) are left out and the first `sampled` arcs of
  // the others were already united.  Plain loads: the launch before writes the flags
  const uint32_t* skip = nullptr;
  const uint64_t* __restrict__ off = nullptr;
  uint32_t sampled = 0;
  __device__ __forceinline__ bool skips(uint32_t u) const { return skip && ((skip[u >> 5] >> (u & 31u)) & 1u); }
  __device__ __forceinline__ double operator()(uint32_t u, uint64_t a) const {
    if (sampled && a < __ldg(off + u) + sampled) return 0.0;
    uf_union(parent, nullptr, u, __ldg(col + a));
    return 0.0;
  }
};

// Afforest (Sutton, Ben-Nun and Bar 2018), first pass: every vertex is united with its first k
// neighbours (relabelled rows list the hubs first, which joins most of a giant component).  The
// first arc, where it leads to a smaller id, needs no union: it is the vertex's parent from the
// start (ids fall along it, so no cycle), written with plain stores; most of the second arcs then
// find both ends in one tree.  RMAT-22: 252 us with unions for both
// arcs, 64 us (29 + 35) so; the whole call 1240 -> 215 us with it, the links by stored id and k_uf_least.
// On a graph without hubs (`joined` given: a bit per vertex) only a parent whose own first arc goes up is taken: rising
// ids along a path or a tree would hang every vertex under the one before, and the unions that follow walk
// those chains (10^6 vertices, rising ids, the call with chains / so: path 499 / 236 us, random tree 1172 / 231, comb
// 379 / 136, grid 614 / 293; ids at random: the same).
__global__ void k_uf_first(uint64_t n, const uint64_t* __restrict__ off, const uint32_t* __restrict__ col,
                           uint32_t* __restrict__ parent, uint32_t* __restrict__ joined) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ull; base < n; base += stride) {
    const uint64_t u = base + (threadIdx.x & 31u);
    bool in = false;
    if (u < n) {
      const uint64_t a0 = off[u];
      const uint32_t v = a0 < off[u + 1] ? __ldg(col + a0) : (uint32_t)u;
      in = v < u;
      if (in && joined) {
        const uint64_t b0 = off[v];
        in = b0 == off[v + 1] || __ldg(col + b0) >= v;
      }
      parent[u] = in ? v : (uint32_t)u;
    }
    if (joined) {
      const uint32_t word = __ballot_sync(0xffffffffu, in);
      if ((threadIdx.x & 31u) == 0) joined[base >> 5] = word;
    }
  }
}
// The first k arcs of every row as unions; `all`: no first arc is a parent yet.
__global__ void k_uf_sample(uint64_t n, const uint64_t* __restrict__ off, const uint32_t* __restrict__ col, uint32_t k,
                            uint32_t* parent, const uint32_t* __restrict__ joined, bool all) {
  for (uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; u < n; u += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t a0 = off[u], a1 = off[u + 1];
    for (uint64_t a = a0; a < a1 && a < a0 + k; ++a) {
      const uint32_t v = __ldg(col + a);
      if (a == a0 && !all && (joined ? (__ldg(joined + (u >> 5)) >> (u & 31u)) & 1u : v < u)) continue;
      uf_union(parent, nullptr, (uint32_t)u, v);
    }
  }
}

// The most frequent root among those of kSample evenly spaced vertices (the smallest of equals), found
// by one CTA: the host is not asked.
constexpr uint32_t kSample = 256;
__global__ void __launch_bounds__(kSample) k_uf_mode(uint64_t n, uint64_t stride, uint32_t* parent, uint32_t* __restrict__ best) {
  __shared__ uint32_t root[kSample];
  __shared__ unsigned long long top;
  const uint32_t ns = (uint32_t)((n + stride - 1) / stride < kSample ? (n + stride - 1) / stride : kSample);
  const uint32_t t = threadIdx.x;
  if (t == 0) top = 0;
  if (t < ns) root[t] = uf_find(parent, (uint32_t)(t * stride));
  __syncthreads();
  if (t < ns) {
    uint32_t same = 0;
    for (uint32_t i = 0; i < ns; ++i) same += root[i] == root[t];
    atomicMax(&top, (unsigned long long)same << 32 | (0xffffffffu - root[t]));
  }
  __syncthreads();
  if (t == 0) *best = 0xffffffffu - (uint32_t)top;
}

// parent[v] = root of v; skip bit of every vertex in the tree of *best; counts[0] += arcs sampled,
// counts[1] += arcs the second pass still visits (byte model)
__global__ void k_uf_compress_skip(uint64_t n, uint32_t* parent, const uint64_t* __restrict__ off, const uint32_t* __restrict__ best,
                                   uint32_t k, uint32_t* __restrict__ skip, unsigned long long* __restrict__ counts) {
  const uint32_t b = *best;
  unsigned long long sampled = 0, rest = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ull; base < n; base += stride) {
    const uint64_t v = base + (threadIdx.x & 31u);
    bool in = false;
    if (v < n) {
      const uint32_t r = uf_find(parent, (uint32_t)v);
      parent[v] = r;
      in = r == b;
      const uint64_t d = off[v + 1] - off[v];
      sampled += d < k ? d : k;
      if (!in && d > k) rest += d - k;
    }
    const uint32_t word = __ballot_sync(0xffffffffu, in);
    if ((threadIdx.x & 31u) == 0) skip[base >> 5] = word;
  }
  for (int o = 16; o > 0; o >>= 1) {
    sampled += __shfl_xor_sync(0xffffffffu, sampled, o);
    rest += __shfl_xor_sync(0xffffffffu, rest, o);
  }
  if ((threadIdx.x & 31u) == 0) {
    if (sampled) atomicAdd(counts, sampled);
    if (rest) atomicAdd(counts + 1, rest);
  }
}

// root[v] = root of v, and the roots of an evenly spaced sample of vertices.  parent[v] is set to it too, but
// a find that passes through v may leave an inner vertex there after that: only root[] is to be relied on.
__global__ void k_uf_compress(uint64_t n, uint32_t* parent, uint32_t* __restrict__ root, uint64_t stride,
                              uint32_t* __restrict__ sample, uint32_t nsample) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t r = uf_find(parent, (uint32_t)v);
    parent[v] = r;
    root[v] = r;
    if (v % stride == 0 && v / stride < nsample) sample[v / stride] = r;
  }
}

// skip bit of every vertex already in the largest component c; counts[0] += arcs sampled,
// counts[1] += arcs the second pass still visits (byte model)
__global__ void k_uf_skipbits(uint64_t n, const uint32_t* __restrict__ root, const uint64_t* __restrict__ off, uint32_t c,
                              uint32_t k, uint32_t* __restrict__ skip, unsigned long long* __restrict__ counts) {
  const uint64_t nwords = (n + 31) >> 5;
  unsigned long long sampled = 0, rest = 0;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwords; w += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t bits = 0;
    for (uint32_t b = 0; b < 32 && (w << 5) + b < n; ++b) {
      const uint64_t v = (w << 5) + b;
      const uint64_t d = off[v + 1] - off[v];
      const bool in_c = root[v] == c;
      bits |= (uint32_t)in_c << b;
      sampled += d < k ? d : k;
      if (!in_c && d > k) rest += d - k;
    }
    skip[w] = bits;
  }
  for (int o = 16; o > 0; o >>= 1) {
    sampled += __shfl_xor_sync(0xffffffffu, sampled, o);
    rest += __shfl_xor_sync(0xffffffffu, rest, o);
  }
  if ((threadIdx.x & 31u) == 0) {
    if (sampled) atomicAdd(counts, sampled);
    if (rest) atomicAdd(counts + 1, rest);
  }
}
struct NoFinish {
  __device__ __forceinline__ void operator()(uint32_t, double) const {}
};

__global__ void k_uf_init(uint64_t n, uint32_t* __restrict__ parent) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
    parent[v] = (uint32_t)v;
}

__global__ void k_uf_flatten(uint64_t n, uint32_t* parent, uint32_t* __restrict__ label) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
    label[v] = uf_find(parent, (uint32_t)v);
}

// Relabelled graphs: least[r] = smallest caller id in the tree of root r (least starts as a copy of perm)
// and label[caller id of v] = root of v.  The root is written to the label, not to parent[v]: another
// thread's uf_find that passes through v may store an inner vertex to parent[v] after it, and on deep trees did.
// A warp keeps the smallest id of the tree of its first lane
// from step to step and hands it on when that tree changes: nearly all warps meet the giant tree's
// word, which serves one request a clock, reads too (looked at every step: RMAT-22 42 us, so 23).
__device__ __forceinline__ void uf_lower(uint32_t* least, uint32_t r, uint32_t id) {
  if (id < __ldcg(least + r)) atomicMin(least + r, id);
}
__global__ void k_uf_least(uint64_t n, uint32_t* parent, const uint32_t* __restrict__ perm, uint32_t* least,
                           uint32_t* __restrict__ label) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const bool lead = (threadIdx.x & 31u) == 0;
  uint32_t tree = 0xffffffffu, low = 0xffffffffu;  // the warp's
  for (uint64_t base = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ull; base < n; base += stride) {
    const uint64_t v = base + (threadIdx.x & 31u);
    uint32_t r = 0xffffffffu, id = 0xffffffffu;
    if (v < n) {
      r = uf_find(parent, (uint32_t)v);
      id = __ldg(perm + v);
      label[id] = r;
    }
    const uint32_t first = __shfl_sync(0xffffffffu, r, 0);  // lane 0 holds a vertex
    if (first != tree) {
      if (lead && tree != 0xffffffffu) uf_lower(least, tree, low);
      tree = first;
      low = 0xffffffffu;
    }
    const uint32_t step = __reduce_min_sync(0xffffffffu, r == first ? id : 0xffffffffu);
    low = step < low ? step : low;
    if (v < n && r != first) uf_lower(least, r, id);
  }
  if (lead && tree != 0xffffffffu) uf_lower(least, tree, low);
}
__global__ void k_uf_label(uint64_t n, const uint32_t* __restrict__ least, uint32_t* __restrict__ label) {
  for (uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; u < n; u += (uint64_t)gridDim.x * blockDim.x)
    label[u] = __ldg(least + label[u]);
}

uint32_t uf_most_frequent(std::vector<uint32_t>& hs, uint32_t ns) {
  std::sort(hs.begin(), hs.begin() + ns);
  uint32_t best = hs[0], run = 0, best_run = 0;
  for (uint32_t i = 0; i < ns; ++i) {
    run = (i && hs[i] == hs[i - 1]) ? run + 1 : 1;
    if (run > best_run) {
      best_run = run;
      best = hs[i];
    }
  }
  return best;
}

}  // namespace gre

using namespace gre;

extern "C" {

int gre_cc(gre_graph g, uint32_t* label, gre_stats* st) {
  if (!g || !label) return GRE_NULL;
  GRE_CHECK(use_graph(g));
  stats_reset(st);
  const uint64_t n = g->n;
  GRE_CHECK(ensure_bins(g, false));
  uint32_t *dlabel, *parent, *least = nullptr;
  double* partial;
  void* p;
  GRE_CHECK(prepare_output(g, label, n, WS_OUTBUF, &dlabel));
  GRE_CHECK(g->ws.get(WS_A, sizeof(uint32_t) * n, &p));
  parent = (uint32_t*)p;
  GRE_CHECK(g->ws.get(WS_B, sizeof(double) * (g->bins_out.n_partials + 1), &p));
  partial = (double*)p;
  if (g->perm) {
    GRE_CHECK(g->ws.get(WS_PERM_OUT, sizeof(uint32_t) * n, &p));
    least = (uint32_t*)p;
  }
  constexpr uint32_t kSampled = 2;
  constexpr uint64_t kHubArcs = 256;  // largest degree of a graph with hubs
  // Blocks of a bin an SM: one wave strides over the rows, so that those of small ids are linked and flattened before the
  // rest start (directed grid of 10^6 vertices, 16 / 8 blocks: rising ids 234 / 173 us; ids at random 244 / 284)
  constexpr int kWave = 8;
  uint32_t *skip = nullptr, *best = nullptr;
  unsigned long long* counts = nullptr;
  if (g->symmetric()) {
    GRE_CHECK(g->ws.get(WS_C, sizeof(uint32_t) * ((n + 31) >> 5), &p));
    skip = (uint32_t*)p;
    GRE_CHECK(g->ws.get(WS_COUNTERS, 3 * sizeof(unsigned long long), &p));
    counts = (unsigned long long*)p;
    best = (uint32_t*)(counts + 2);
  }
  // Directed graphs: what is linked first decides how deep the trees get.  Us, one launch of all bins / the form chosen:
  //  * few arcs, no hubs: short rows in the order of their ids, and what they have beyond four arcs after all of them.
  //    10^6 vertices, trees with parents at most 10 ids back 476 / 141, relabelled 900 / 576, 50 back 314 / 139; grids and
  //    paths the same; any id before 80 / 95, with ids at random 330 / 650; 2M
  //    vertices of two random arcs 213 / 308;
  //  * rows of about one length: four arcs a lane instead of the eight that suit a sum, since a lane's unions follow each
  //    other, and bin by bin.  30000 vertices of 40 arcs 425 / 105, relabelled 401 / 137, 300000 of 8 216 / 111, 3000 of 40 115 /
  //    66; 24000 arcs 48 / 60; 12M arcs 199 / 255;
  //  * hubs that do not have the smallest ids: their CTAs link the loose vertices of half the graph and the root changes
  //    under all of them, unless the short rows went first.  RMAT-16, 0.95M arcs 306 / 135, RMAT-18, 1.5M 545 / 230; about
  //    equal at 0.25M (97 / 92) and 4M (290 / 292); RMAT-20 at 6M 434 / 604.  A relabelled graph's hubs are the roots
  //    (RMAT-18: 128 / 275).
  const bool directed = !g->symmetric(), hubs = g->max_outdeg >= kHubArcs, untuned = g->m < (1ull << 22);
  const bool few = directed && !hubs && g->m < 4 * n && g->m < (1ull << 21);
  const bool even = directed && !hubs && !few && g->m >= (1ull << 16) && untuned;
  const bool loose = directed && hubs && !g->perm && g->m >= (1ull << 18) && untuned;
  const DegreeBins* bins = &g->bins_out;
  if (even && bins->sched.lane_arcs > RowSchedule().lane_arcs && !getenv("GRE_ROW_SCHEDULE")) {
    if (!g->bins_cc.ready) GRE_CHECK(build_bins(g, g->bins_cc, g->off, g->col, RowSchedule()));
    bins = &g->bins_cc;
  }
  RunTimer timer(g);
  if (g->symmetric()) {
    // Afforest: unite the first arcs of every row, find the largest component from a sample,
    // then unite the remaining arcs of the vertices outside it only.  Undirected edges appear
    // in both rows, so an edge between the largest component and another vertex is seen from
    // the other side.
    GRE_CUDA(cudaMemsetAsync(counts, 0, 2 * sizeof(unsigned long long), g->stream));
    uint32_t* joined = g->max_outdeg < kHubArcs ? skip : nullptr;  // the skip flags' words are free until the compression
    k_uf_first<<<grid_for(n, 256), 256, 0, g->stream>>>(n, g->off, g->col, parent, joined);
    k_uf_sample<<<grid_for(n, 256), 256, 0, g->stream>>>(n, g->off, g->col, kSampled, parent, joined, false);
    k_uf_mode<<<1, kSample, 0, g->stream>>>(n, n > kSample ? n / kSample : 1, parent, best);
    k_uf_compress_skip<<<grid_for(n, 256), 256, 0, g->stream>>>(n, parent, g->off, best, kSampled, skip, counts);
    HookArcs rest{g->col, parent, skip, g->off, kSampled};
    GRE_CHECK(rows::reduce_rows(g->bins_out, g->off, rest, NoFinish{}, partial, g->stream, kWave));
  } else {
    k_uf_init<<<grid_for(n, 256), 256, 0, g->stream>>>(n, parent);
    HookArcs arcs{g->col, parent};
    if (few) {
      constexpr uint32_t kFew = 4;
      k_uf_sample<<<grid_for(n, 256), 256, 0, g->stream>>>(n, g->off, g->col, kFew, parent, nullptr, true);
      arcs.off = g->off;
      arcs.sampled = kFew;
      if (g->max_outdeg > kFew) GRE_CHECK(rows::reduce_rows(*bins, g->off, arcs, NoFinish{}, partial, g->stream, kWave));
    } else if (even || loose) {
      GRE_CHECK(rows::visit_rows_apart(*bins, g->off, arcs, NoFinish{}, partial, g->stream, kWave));
    } else {
      GRE_CHECK(rows::reduce_rows(*bins, g->off, arcs, NoFinish{}, partial, g->stream, kWave));
    }
  }
  if (g->perm) {
    GRE_CUDA(cudaMemcpyAsync(least, g->perm, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, g->stream));
    k_uf_least<<<grid_for(n, 256), 256, 0, g->stream>>>(n, parent, g->perm, least, dlabel);
    k_uf_label<<<grid_for(n, 256), 256, 0, g->stream>>>(n, least, dlabel);
  } else {
    k_uf_flatten<<<grid_for(n, 256), 256, 0, g->stream>>>(n, parent, dlabel);
  }
  GRE_LAUNCH_CHECK();
  GRE_CHECK(finish_output(g, label, dlabel, n));
  GRE_CHECK(timer.stop(st));
  if (st) {
    uint64_t visited = g->m;
    if (g->symmetric()) {  // arcs the two Afforest passes visited
      unsigned long long h[2] = {0, 0};
      GRE_CUDA(cudaMemcpy(h, counts, sizeof h, cudaMemcpyDeviceToHost));
      visited = h[0] + h[1];
    }
    st->supersteps = 1;
    st->arcs_traversed = visited;
    st->traversed_edges = g->symmetric() ? g->m / 2 : g->m;
    st->algo_bytes = 8 * (n + 1) + 12 * visited + 8 * n + (g->symmetric() ? n / 4 : 0);
  }
  return GRE_SUCCESS;
}

}  // extern "C"
