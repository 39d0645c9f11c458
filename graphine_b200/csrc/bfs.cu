// BFS fast paths.
//
// The reference BFS (Kernels/BFS.hpp:34-72 on Engine.hpp's superstep) expands every frontier
// vertex over its arcs, claims unvisited neighbours first-writer-wins under a lock and makes
// them the next frontier; levels are the superstep of discovery.  Here:
//
//  * gre_bfs / gre_bfs_multiroot: direction-optimising BFS (Beamer, Asanovic, Patterson 2012), the
//    level loop inside one cooperative kernel (bfs_persist.cu).  Switch rule: to bottom-up when the
//    frontier's arcs exceed (unvisited arcs)/15, back to top-down when the frontier holds fewer
//    than n/18 vertices.
//  * the step kernels of the searches whose level loop stays on the host: the partitioned one (an
//    exchange a level, partition.cu) and gre_bfs_noalloc (noalloc.cu).  Top-down steps expand a
//    frontier queue edge-balanced: one thread per frontier arc, the owning vertex found by binary
//    search in the exclusive scan of frontier degrees; a visited bitmap (n/8 bytes, L2-resident)
//    filters claims, atomicOr claims a vertex.  Bottom-up steps give each unvisited vertex one
//    thread that scans its in-arcs for a parent in the frontier bitmap and stops at the first; a
//    warp covers 32 consecutive vertices, so the next-frontier word is one __ballot_sync and needs
//    no atomics.
//  * gre_msbfs: 64 sources per uint64 word, the level loop in msbfs.cu.
//
// Byte model, top-down level: 16 F (queue + offsets) + 8 A (column + visited probe) + 8 N;
// bottom-up level: 16 U (offsets + level of unvisited) + 4.125 A (column + frontier bit) + 4 N
// + n/8 (bitmap).  F frontier, A arcs scanned, U unvisited vertices scanned, N newly visited.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstdlib>

#include "bfs_persist.cuh"
#include "gre_internal.cuh"
#include "msbfs.cuh"

namespace gre {

template <class T>
static int ws_array(gre_graph g, int slot, uint64_t count, T** p) {
  void* v = nullptr;
  GRE_CHECK(g->ws.get(slot, sizeof(T) * (count ? count : 1), &v));
  *p = (T*)v;
  return GRE_SUCCESS;
}

struct BfsCounters {
  unsigned long long next_count;  // vertices discovered in this level
  unsigned long long next_arcs;   // sum of their (out) degrees
  unsigned long long scanned;     // arcs scanned in this level
  unsigned long long pad;
};

__global__ void k_bfs_seed(const uint32_t* __restrict__ roots, uint32_t nroots, int32_t* __restrict__ level,
                           uint32_t* __restrict__ vis, uint32_t* __restrict__ queue, const uint64_t* __restrict__ off,
                           BfsCounters* __restrict__ c) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  uint32_t q = 0;
  unsigned long long arcs = 0;
  for (uint32_t i = 0; i < nroots; ++i) {
    const uint32_t r = roots[i];
    if (vis[r >> 5] & (1u << (r & 31u))) continue;
    vis[r >> 5] |= 1u << (r & 31u);
    level[r] = 0;
    queue[q++] = r;
    arcs += off[r + 1] - off[r];
  }
  c->next_count = q;
  c->next_arcs = arcs;
}

__global__ void k_frontier_degrees(const uint32_t* __restrict__ queue, uint64_t nq, const uint64_t* __restrict__ off,
                                   uint64_t* __restrict__ deg) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nq; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t u = queue[i];
    deg[i] = off[u + 1] - off[u];
  }
}

// One thread per frontier arc; prefix = exclusive scan of frontier degrees.
__global__ void __launch_bounds__(256) k_td_expand(const uint32_t* __restrict__ queue, uint64_t nq, const uint64_t* __restrict__ prefix,
                                                   uint64_t total, const uint64_t* __restrict__ off, const uint32_t* __restrict__ col,
                                                   uint32_t* __restrict__ vis, int32_t* __restrict__ level, int32_t next_level,
                                                   uint32_t* __restrict__ next_queue, BfsCounters* __restrict__ c) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  // iterate warp-uniformly so warp_append sees all 32 lanes
  for (uint64_t base = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ull; base < total; base += stride) {
    const uint64_t t = base + (threadIdx.x & 31u);
    bool claim = false;
    uint32_t v = 0;
    unsigned long long dv = 0;
    if (t < total) {
      // largest i with prefix[i] <= t
      uint64_t lo = 0, hi = nq;
      while (hi - lo > 1) {
        const uint64_t mid = (lo + hi) >> 1;
        if (prefix[mid] <= t) lo = mid;
        else hi = mid;
      }
      const uint32_t u = queue[lo];
      v = __ldg(col + off[u] + (t - prefix[lo]));
      const uint32_t bit = 1u << (v & 31u);
      if (!(vis[v >> 5] & bit)) {
        const uint32_t old = atomicOr(vis + (v >> 5), bit);
        if (!(old & bit)) {
          claim = true;
          level[v] = next_level;
          dv = off[v + 1] - off[v];
        }
      }
    }
    const uint32_t pos = warp_append((uint32_t*)&c->pad, claim);  // slot counter lives in pad
    if (claim) next_queue[pos] = v;
    unsigned long long s = dv;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31u) == 0 && s) atomicAdd(&c->next_arcs, s);
  }
}

__global__ void k_queue_to_bits(const uint32_t* __restrict__ queue, uint64_t nq, uint32_t* __restrict__ bits) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nq; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = queue[i];
    atomicOr(bits + (v >> 5), 1u << (v & 31u));
  }
}

// Bottom-up level over in-arcs (roff/rcol); warp = one 32-vertex bitmap word.
__global__ void __launch_bounds__(256) k_bu_step(uint64_t n, const uint64_t* __restrict__ roff, const uint32_t* __restrict__ rcol,
                                                 const uint64_t* __restrict__ off, const uint32_t* __restrict__ front,
                                                 uint32_t* __restrict__ next, uint32_t* __restrict__ vis, int32_t* __restrict__ level,
                                                 int32_t next_level, BfsCounters* __restrict__ c) {
  const uint64_t nwords = (n + 31) >> 5;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long found_arcs = 0, scanned = 0, found_n = 0;
  for (uint64_t w = warp; w < nwords; w += nwarps) {
    const uint32_t vw = vis[w];
    if (vw == 0xffffffffu) {
      if (lane == 0) next[w] = 0;
      continue;
    }
    const uint64_t v = (w << 5) + lane;
    bool found = false;
    if (v < n && !((vw >> lane) & 1u)) {
      const uint64_t a1 = roff[v + 1];
      for (uint64_t a = roff[v]; a < a1; ++a) {
        const uint32_t u = __ldg(rcol + a);
        ++scanned;
        if ((__ldg(front + (u >> 5)) >> (u & 31u)) & 1u) {
          found = true;
          break;
        }
      }
      if (found) {
        level[v] = next_level;
        found_arcs += off[v + 1] - off[v];
        ++found_n;
      }
    }
    const uint32_t ball = __ballot_sync(0xffffffffu, found);
    if (lane == 0) {
      next[w] = ball;
      if (ball) vis[w] = vw | ball;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    found_arcs += __shfl_xor_sync(0xffffffffu, found_arcs, o);
    scanned += __shfl_xor_sync(0xffffffffu, scanned, o);
    found_n += __shfl_xor_sync(0xffffffffu, found_n, o);
  }
  if (lane == 0) {
    if (found_n) atomicAdd(&c->next_count, found_n);
    if (found_arcs) atomicAdd(&c->next_arcs, found_arcs);
    if (scanned) atomicAdd(&c->scanned, scanned);
  }
}

// bitmap -> queue (order within a warp's 32 words is by vertex id)
__global__ void k_bits_to_queue(uint64_t n, const uint32_t* __restrict__ bits, uint32_t* __restrict__ queue,
                                unsigned long long* __restrict__ count) {
  const uint64_t nwords = (n + 31) >> 5;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = tid - lane; base < nwords; base += nthreads) {
    const uint64_t w = base + lane;
    const uint32_t word = (w < nwords) ? bits[w] : 0u;
    const uint32_t cnt = __popc(word);
    uint32_t incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (uint32_t)o) incl += t;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    unsigned long long pos = 0;
    if (lane == 31 && total) pos = atomicAdd(count, (unsigned long long)total);
    pos = __shfl_sync(0xffffffffu, pos, 31) + incl - cnt;
    uint32_t x = word;
    while (x) {
      const uint32_t b = __ffs(x) - 1;
      x &= x - 1;
      queue[pos++] = (uint32_t)(w << 5) + b;
    }
  }
}

}  // namespace gre

using namespace gre;

extern "C" {

int gre_bfs(gre_graph g, const uint32_t* srcs, uint32_t nsrc, int32_t* levels, gre_stats* st) {
  if (!g || !levels || (nsrc && !srcs)) return GRE_NULL;
  GRE_CHECK(use_graph(g));
  stats_reset(st);
  const uint64_t n = g->n;
  std::vector<uint32_t> hs(nsrc);
  if (nsrc) GRE_CUDA(cudaMemcpy(hs.data(), srcs, sizeof(uint32_t) * nsrc, cudaMemcpyDefault));
  GRE_CHECK(map_ids(g, &hs, "gre_bfs"));
  int32_t* dl;
  GRE_CHECK(prepare_output(g, levels, (uint64_t)nsrc * n, WS_OUTBUF, &dl));
  RunTimer timer(g);
  uint64_t arcs = 0;
  if (nsrc) {
    BfsPlan plan;
    GRE_CHECK(plan.prepare(g, nsrc, true, st && nsrc == 1));
    for (uint32_t i = 0; i < nsrc; ++i) GRE_CHECK(plan.search(i, nullptr, 1, hs[i], dl + (uint64_t)i * n));
    GRE_CHECK(plan.collect(st, &arcs));
  }
  GRE_CHECK(finish_output(g, levels, dl, (uint64_t)nsrc * n));
  GRE_CHECK(timer.stop(st));
  if (st) st->traversed_edges = g->symmetric() ? arcs / 2 : arcs;
  return GRE_SUCCESS;
}

int gre_bfs_multiroot(gre_graph g, const uint32_t* roots, uint32_t nroots, int32_t* level, gre_stats* st) {
  if (!g || !level || (nroots && !roots)) return GRE_NULL;
  GRE_CHECK(use_graph(g));
  stats_reset(st);
  const uint64_t n = g->n;
  std::vector<uint32_t> hs(nroots);
  if (nroots) GRE_CUDA(cudaMemcpy(hs.data(), roots, sizeof(uint32_t) * nroots, cudaMemcpyDefault));
  GRE_CHECK(map_ids(g, &hs, "gre_bfs_multiroot"));
  int32_t* dl;
  uint32_t* droot;
  GRE_CHECK(prepare_output(g, level, n, WS_OUTBUF, &dl));
  GRE_CHECK(ws_array(g, WS_H, nroots ? nroots : 1, &droot));
  RunTimer timer(g);
  if (nroots) GRE_CUDA(cudaMemcpyAsync(droot, hs.data(), sizeof(uint32_t) * nroots, cudaMemcpyHostToDevice, g->stream));
  BfsPlan plan;
  uint64_t arcs = 0;
  GRE_CHECK(plan.prepare(g, 1, true, st != nullptr));
  GRE_CHECK(plan.search(0, droot, nroots, 0, dl));
  GRE_CHECK(plan.collect(st, &arcs));
  GRE_CHECK(finish_output(g, level, dl, n));
  GRE_CHECK(timer.stop(st));
  if (st) st->traversed_edges = g->symmetric() ? arcs / 2 : arcs;
  return GRE_SUCCESS;
}

int gre_msbfs(gre_graph g, const uint32_t* srcs, uint32_t nsrc, int32_t* levels, gre_stats* st) {
  if (!g || !levels || (nsrc && !srcs)) return GRE_NULL;
  GRE_CHECK(use_graph(g));
  stats_reset(st);
  const uint64_t n = g->n;
  std::vector<uint32_t> hs(nsrc);
  if (nsrc) GRE_CUDA(cudaMemcpy(hs.data(), srcs, sizeof(uint32_t) * nsrc, cudaMemcpyDefault));
  GRE_CHECK(map_ids(g, &hs, "gre_msbfs"));
  int32_t* dl;
  uint32_t* dsrc;
  unsigned long long* reached;
  GRE_CHECK(prepare_output(g, levels, (uint64_t)nsrc * n, WS_OUTBUF, &dl));
  GRE_CHECK(ws_array(g, WS_I, nsrc, &dsrc));
  GRE_CHECK(ws_array(g, WS_COUNTERS, 8, &reached));
  RunTimer timer(g);
  uint32_t max_levels = 0;
  MsBfs word;
  unsigned long long arcs = 0;
  if (nsrc) {
    GRE_CHECK(word.prepare(g, false));
    GRE_CUDA(cudaMemsetAsync(reached, 0, sizeof *reached, g->stream));
    GRE_CUDA(cudaMemcpyAsync(dsrc, hs.data(), sizeof(uint32_t) * nsrc, cudaMemcpyHostToDevice, g->stream));
    for (uint32_t j0 = 0; j0 < nsrc; j0 += 64) {
      const uint32_t k = std::min<uint32_t>(64, nsrc - j0);
      GRE_CHECK(word.run(dsrc + j0, k, st && nsrc <= 64));
      GRE_CHECK(word.write_levels(k, dl + (uint64_t)j0 * n, reached));
      max_levels = std::max(max_levels, word.levels);
    }
    GRE_CUDA(cudaMemcpyAsync(&arcs, reached, sizeof arcs, cudaMemcpyDeviceToHost, g->stream));
    GRE_CUDA(cudaStreamSynchronize(g->stream));
  }
  GRE_CHECK(finish_output(g, levels, dl, (uint64_t)nsrc * n));
  GRE_CHECK(timer.stop(st));
  if (st) {
    for (unsigned long long f : word.found) stats_record(st, f);
    st->supersteps = max_levels;
    st->arcs_traversed = word.scanned;
    st->traversed_edges = g->symmetric() ? arcs / 2 : arcs;
    st->algo_bytes = word.bytes;
  }
  return GRE_SUCCESS;
}

}  // extern "C"
