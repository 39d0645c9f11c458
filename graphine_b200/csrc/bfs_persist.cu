// Direction-optimising BFS (Beamer, Asanovic, Patterson 2012) as one cooperative launch a search.
//
// A level of a search takes a few microseconds; driven from the host it cost two or three counter
// reads and up to six launches, so the host's round trips bounded every search (RMAT-22: 470 us a
// source, kernels about half of it; 4000 vertices: 300 us, kernels 60).  Here the level loop runs in
// the kernel: the blocks meet at a grid barrier a level and read the direction off the same
// counters.  Searches of one call follow each other on the stream without the host.
//
// State: one bit a vertex (visited), in two buffers.
//   * top-down: the frontier is a queue of items (vertex, 128-arc piece of its row), so that a hub
//     is spread over the grid; a warp lays the arcs of up to 32 items side by side and its lanes
//     take 32 at a time, four steps in flight.  A new vertex is claimed by atomicOr on its bit and
//     appended as items.
//   * bottom-up: a warp takes 128 vertices; the unvisited ones look for a visited in-neighbour.
//     A vertex found by neither direction so far can have in-neighbours on the last level only
//     (an earlier one would have found it), so the visited bits serve as the frontier and none is
//     kept; what is found goes to the other buffer.  Back to top-down, the queue is the difference
//     of the two buffers.
// Vertices without any arc count as visited from the start (RMAT: about half of all): their words
// are skipped.  (Those with out-arcs only are not marked: they are nobody's parent until a search
// starts there.)  Levels go straight to the caller's order (perm), so nothing is reordered after.
//
// Measured against the host-driven loop: RMAT-22, 16 sources one after the other, 7470 -> 2540 us;
// 32 graphs of 2^12..2^18 vertices in one union 550 -> 204 us; 4000 vertices 294 -> 103 us; a grid of 1000 x 1000
// 98 -> 14.4 ms.  A barrier is 1.5 us; most of a small level is the chain of dependent loads (queue, offsets, column,
// bit, claim).
#include <algorithm>
#include <vector>

#include "bfs_persist.cuh"
#include "grid_sync.cuh"
#include "item_queue.cuh"

namespace gre {

constexpr int kBfsThreads = 512;

// Back from bottom-up to top-down below n/18 frontier vertices; not yet, for two levels, when the vertices
// not found so far hold less than 1/32 of the arcs: with so little left to look at a bottom-up step is
// 4-5 us, the way back (queue from the bits, one barrier more, a top-down step) 10-16 us, and most searches
// end there (RMAT-22, a frontier of 65473: 15.8 us).  RMAT-22, 16 sources 2610 -> 2540 us; eight over 20000 vertices
// 537 -> 484, over 200000 748 -> 680, over 1.5M 964 -> 906.  At RMAT-25 the bits themselves are 4 MB a step:
// 7490 -> 7640 us for eight, so graphs above 2^23 vertices go back at once.
constexpr uint64_t kFewLeft = 32;
constexpr uint32_t kLate = 2;
constexpr uint64_t kLateVertices = 1ull << 23;

struct BfsSlot {  // the frontier of one level
  unsigned long long nf, mf;      // vertices, their out-arcs
  unsigned long long scanned;     // arcs looked at by the bottom-up step that found it
  unsigned int nitems, pad;
};

struct BfsCtl {
  GridBar bar;
  BfsSlot slot[3];  // level d: slot d % 3; the next one is filled, the one after cleared
  unsigned long long arcs_td, arcs_bu, bytes, reached_arcs;
  unsigned int levels, pad;
};

struct BfsRun {
  uint64_t n, m, nwords;  // nwords: a multiple of 4
  const uint64_t* __restrict__ off;
  const uint32_t* __restrict__ col;
  const uint64_t* __restrict__ roff;
  const uint32_t* __restrict__ rcol;
  const uint32_t* __restrict__ arc_bits;
  const uint32_t* __restrict__ perm;
  const uint32_t* __restrict__ roots;  // null: the one root is `root`
  uint32_t nroots, root;
  uint32_t* vis0;
  uint32_t* vis1;
  uint2* q0;
  uint2* q1;
  int32_t* level;
  unsigned long long* rec;  // vertices of every level from the second (null: not recorded)
  uint32_t nrec;
  BfsCtl* ctl;
  long long wait_ns;
};

// Bit per vertex: it has arcs, in or out.  Bits past n are 0.
__global__ void k_arc_bits(uint64_t n, uint64_t nwords, const uint64_t* __restrict__ off, const uint64_t* __restrict__ roff,
                           uint32_t* __restrict__ bits) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ull; base < nwords * 32; base += stride) {
    const uint64_t v = base + (threadIdx.x & 31u);
    const uint32_t w = __ballot_sync(0xffffffffu, v < n && (roff[v + 1] > roff[v] || off[v + 1] > off[v]));
    if ((threadIdx.x & 31u) == 0) bits[base >> 5] = w;
  }
}

struct BfsStage {
  unsigned long long nf, mf, scanned;  // this level's slot
  unsigned int nitems;
  ItemStage<kBfsThreads> items;
  BlockSums<3> sums;
};
using BfsAppend = ItemAppend<kBfsThreads, uint2>;

__device__ __forceinline__ void add_found(BfsStage& st, BfsSlot* s, unsigned long long nf, unsigned long long mf,
                                          unsigned long long scanned) {
  st.sums.add({nf, mf, scanned}, {&s->nf, &s->mf, &s->scanned});
}

__device__ __forceinline__ void top_down(const BfsRun& R, const uint2* queue, uint32_t nitems, uint32_t* vis, int32_t next_level,
                                         uint2* out, BfsSlot* s, BfsStage& st, uint32_t gwarp, uint32_t nwarps) {
  constexpr int U = 4;
  BfsAppend append(st.items, &s->nitems, out);
  const uint32_t lane = lane_id();
  // few items: one a warp, so that all warps share the arcs
  const uint32_t per = min(32u, max(1u, (nitems + nwarps - 1) / nwarps));
  unsigned long long nf = 0, mf = 0;
  for (uint64_t base = (uint64_t)gwarp * per; base < nitems; base += (uint64_t)nwarps * per) {
    uint64_t a0 = 0;
    uint32_t len = 0;
    if (lane < per && base + lane < nitems) {
      const uint2 it = __ldcg(queue + base + lane);
      a0 = R.off[it.x] + (uint64_t)it.y * kPiece;
      len = (uint32_t)min((uint64_t)kPiece, R.off[it.x + 1] - a0);
    }
    const ItemSpan span(a0, len);
    for (uint32_t t = 0; t < span.total; t += 32 * U) {
      uint32_t u[U];
      bool want[U];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const uint32_t pos = t + 32 * k + lane;
        const uint64_t arc = span.arc_of(pos, span.owner(pos));
        want[k] = pos < span.total;
        u[k] = want[k] ? __ldg(R.col + arc) : 0u;
      }
#pragma unroll
      for (int k = 0; k < U; ++k) want[k] = want[k] && !((vis[u[k] >> 5] >> (u[k] & 31u)) & 1u);
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (want[k]) want[k] = !((atomicOr(vis + (u[k] >> 5), 1u << (u[k] & 31u)) >> (u[k] & 31u)) & 1u);
      uint32_t nit[U];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        nit[k] = 0;
        if (want[k]) {
          R.level[R.perm ? __ldg(R.perm + u[k]) : u[k]] = next_level;
          const uint64_t d = R.off[u[k] + 1] - R.off[u[k]];
          nit[k] = items_of(d);
          mf += d;
          ++nf;
        }
      }
      append.push(u, nit);
    }
  }
  append.finish();
  add_found(st, s, nf, mf, 0);
}

__device__ __forceinline__ bool bit_of(const uint32_t* bits, uint32_t u) { return (bits[u >> 5] >> (u & 31u)) & 1u; }

// A warp's 128 vertices are looked at side by side: the first in-arc of each (on a relabelled graph
// the hub, which mostly ends it), then two arcs a round of those still open, so that the loads of
// four rows a lane are in flight together.  What is open after kRounds is a long row: the warp scans
// it 64 arcs at a time (one lane alone held its block for 40 us and more, RMAT-18 batch).
__device__ __forceinline__ void bottom_up(const BfsRun& R, const uint32_t* cur, uint32_t* next, int32_t next_level, BfsSlot* s,
                                          BfsStage& st, uint32_t gwarp, uint32_t nwarps) {
  constexpr int kRounds = 8;
  const uint32_t lane = lane_id();
  unsigned long long nf = 0, mf = 0, scanned = 0;
  for (uint64_t wb = (uint64_t)gwarp * 4; wb < R.nwords; wb += (uint64_t)nwarps * 4) {
    const uint4 raw = *(const uint4*)(cur + wb);
    if ((raw.x & raw.y & raw.z & raw.w) == 0xffffffffu) {
      if (lane == 0) *(uint4*)(next + wb) = raw;
      continue;
    }
    const uint32_t vw[4] = {raw.x, raw.y, raw.z, raw.w};
    uint64_t a[4];
    uint32_t len[4], c[4];  // arcs left from a
    bool open[4], got[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t v = ((wb + j) << 5) + lane;
      open[j] = !((vw[j] >> lane) & 1u);
      a[j] = 0;
      len[j] = 0;
      if (open[j]) {
        a[j] = R.roff[v];
        len[j] = (uint32_t)(R.roff[v + 1] - a[j]);
        open[j] = len[j] != 0;
      }
      got[j] = false;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j] = open[j] ? __ldg(R.rcol + a[j]) : 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (open[j]) {
        ++scanned;
        ++a[j];
        --len[j];
        got[j] = bit_of(cur, c[j]);
        open[j] = !got[j] && len[j] != 0;
      }
    for (int r = 0; r < kRounds && (open[0] || open[1] || open[2] || open[3]); ++r) {
      uint32_t x[4], y[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[j] = open[j] ? __ldg(R.rcol + a[j]) : 0u;
        y[j] = open[j] && len[j] > 1 ? __ldg(R.rcol + a[j] + 1) : x[j];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (open[j]) {
          got[j] = bit_of(cur, x[j]) || bit_of(cur, y[j]);
          const uint32_t k = len[j] > 1 ? 2 : 1;
          scanned += k;
          a[j] += k;
          len[j] -= k;
          open[j] = !got[j] && len[j] != 0;
        }
    }
    uint32_t ball[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      for (uint32_t left = __ballot_sync(0xffffffffu, open[j]); left; left &= left - 1) {
        const int src = __ffs(left) - 1;
        const uint64_t b = __shfl_sync(0xffffffffu, a[j], src);
        const uint32_t n = __shfl_sync(0xffffffffu, len[j], src);
        bool hit = false;
        for (uint32_t i = 0; i < n && !hit; i += 64) {
          if ((i & 0xffffu) == 0 && i && lane == 0) grid_beat(&R.ctl->bar);  // every 0.7 ms
          const uint32_t p = i + lane, q = p + 32;
          const uint32_t x = p < n ? __ldg(R.rcol + b + p) : 0u, y = q < n ? __ldg(R.rcol + b + q) : 0u;
          scanned += (p < n) + (q < n);
          hit = __any_sync(0xffffffffu, (p < n && bit_of(cur, x)) || (q < n && bit_of(cur, y)));
        }
        if (lane == (uint32_t)src) got[j] = hit;
      }
      ball[j] = __ballot_sync(0xffffffffu, got[j]);
      if (got[j]) {
        const uint64_t v = ((wb + j) << 5) + lane;
        R.level[R.perm ? __ldg(R.perm + v) : v] = next_level;
        mf += R.off[v + 1] - R.off[v];
        ++nf;
      }
    }
    if (lane == 0) *(uint4*)(next + wb) = make_uint4(vw[0] | ball[0], vw[1] | ball[1], vw[2] | ball[2], vw[3] | ball[3]);
  }
  add_found(st, s, nf, mf, scanned);
}

// The vertices set in `now` and not in `before`, as items.
__device__ __forceinline__ void bits_to_items(const BfsRun& R, const uint32_t* now, const uint32_t* before, uint2* queue,
                                              unsigned int* count, BfsStage& st, uint32_t gwarp, uint32_t nwarps) {
  BfsAppend append(st.items, count, queue);
  const uint64_t chunks = bit_chunks(R.nwords);
  for (uint64_t ch = gwarp; ch < chunks; ch += nwarps) {
    const uint64_t num = chunk_word(ch, chunks);
    for_bits<1>(num, num < R.nwords ? now[num] & ~before[num] : 0u, [&](const bool (&valid)[1], const uint32_t (&v)[1]) {
      const uint32_t nit[1] = {valid[0] ? items_of(R.off[v[0] + 1] - R.off[v[0]]) : 0u};
      append.push(v, nit);
    });
  }
  append.finish();
}

__global__ void __launch_bounds__(kBfsThreads, 2) k_bfs_persist(const __grid_constant__ BfsRun R) {
  __shared__ BfsStage st;
  const uint32_t lane = lane_id();
  const uint32_t gwarp = (blockIdx.x * kBfsThreads + threadIdx.x) >> 5, nwarps = gridDim.x * (kBfsThreads / 32);
  const uint64_t gtid = blockIdx.x * (uint64_t)kBfsThreads + threadIdx.x, nthreads = (uint64_t)gridDim.x * kBfsThreads;
  BfsCtl* c = R.ctl;
  unsigned int target = 0;
  const bool first = blockIdx.x == 0 && threadIdx.x == 0;
  for (uint64_t v = gtid; v < R.n; v += nthreads) R.level[v] = -1;
  for (uint64_t w = gtid; w < R.nwords; w += nthreads) R.vis0[w] = ~R.arc_bits[w];
  if (!grid_barrier(&c->bar, target, R.wait_ns)) return;
  // the roots, each once, over all blocks (one block took 10 ms for two million while the others waited)
  if ((uint64_t)blockIdx.x * kBfsThreads < R.nroots) {
    unsigned long long nf = 0, mf = 0;
    BfsAppend append(st.items, &c->slot[0].nitems, R.q0);
    for (uint64_t base = (uint64_t)blockIdx.x * kBfsThreads; base < R.nroots; base += nthreads) {
      const uint64_t i = base + threadIdx.x;
      uint32_t rv[1] = {0}, nit[1] = {0};
      if (i < R.nroots) {
        const uint32_t r = rv[0] = R.roots ? R.roots[i] : R.root;
        // a root without arcs has its bit already: its level says whether it was seen
        int32_t* lv = R.level + (R.perm ? R.perm[r] : r);
        if (atomicExch(lv, 0) == -1) {
          atomicOr(R.vis0 + (r >> 5), 1u << (r & 31u));
          const uint64_t d = R.off[r + 1] - R.off[r];
          nit[0] = items_of(d);
          mf += d;
          ++nf;
        }
      }
      append.push(rv, nit);
    }
    append.finish();
    add_found(st, &c->slot[0], nf, mf, 0);
  }
  uint32_t* cur = R.vis0;
  uint32_t* other = R.vis1;
  long long mu = (long long)R.m;
  unsigned long long visited = 0;
  bool bu = false;
  uint32_t d = 0, late = 0;
  for (;; ++d) {
    BfsSlot* s = &c->slot[d % 3];
    BfsSlot* sn = &c->slot[(d + 1) % 3];
    if (!grid_barrier(&c->bar, target, R.wait_ns, [&] {
          st.nf = __ldcg(&s->nf);
          st.mf = __ldcg(&s->mf);
          st.nitems = __ldcg(&s->nitems);
          st.scanned = __ldcg(&s->scanned);
        }))
      return;
    const unsigned long long nf = st.nf, mf = st.mf;
    if (first) {
      const unsigned long long sc = st.scanned;
      c->reached_arcs += mf;
      c->arcs_bu += sc;
      c->bytes += bu ? sc * 4 + sc / 8 + 4 * nf : 8 * nf;
      if (R.rec && d > 0 && d - 1 < R.nrec) R.rec[d - 1] = nf;
      BfsSlot* sz = &c->slot[(d + 2) % 3];  // last read a level ago
      sz->nf = sz->mf = sz->scanned = 0;
      sz->nitems = 0;
    }
    if (nf == 0) break;
    mu -= (long long)mf;
    visited += nf;
    uint2* queue = (d & 1) ? R.q1 : R.q0;
    if (!bu && (double)mf > (double)mu / 15.0 && nf > 64) {
      bu = true;
    } else if (bu && nf < R.n / 18 && (R.n > kLateVertices || mu > (long long)(R.m / kFewLeft) || ++late > kLate)) {
      bits_to_items(R, cur, other, queue, &s->nitems, st, gwarp, nwarps);
      if (!grid_barrier(&c->bar, target, R.wait_ns, [&] { st.nitems = __ldcg(&s->nitems); })) return;
      bu = false;
      late = 0;
    }
    if (bu) {
      if (first) c->bytes += 16 * (R.n - visited) + R.n / 8;
      bottom_up(R, cur, other, (int32_t)d + 1, sn, st, gwarp, nwarps);
      uint32_t* t = cur;
      cur = other;
      other = t;
    } else {
      if (first) {
        c->arcs_td += mf;
        c->bytes += 16 * nf + 8 * mf;
      }
      top_down(R, queue, st.nitems, cur, (int32_t)d + 1, (d & 1) ? R.q0 : R.q1, sn, st, gwarp, nwarps);
    }
  }
  if (first) c->levels = d;
}

template <class T>
static int ws_array(gre_graph g, int slot, uint64_t count, T** p) {
  void* v = nullptr;
  GRE_CHECK(g->ws.get(slot, sizeof(T) * (count ? count : 1), &v));
  *p = (T*)v;
  return GRE_SUCCESS;
}

static int ensure_arc_bits(gre_graph g, uint64_t nwords) {
  if (g->arc_bits) return GRE_SUCCESS;
  GRE_CUDA(cudaMalloc(&g->arc_bits, sizeof(uint32_t) * nwords));
  k_arc_bits<<<grid_for(nwords * 32, 256), 256, 0, g->stream>>>(g->n, nwords, g->off, g->roff, g->arc_bits);
  GRE_LAUNCH_CHECK();
  return GRE_SUCCESS;
}

int BfsPlan::prepare(gre_graph graph, uint32_t nsearch, bool caller_order, bool record) {
  g = graph;
  const uint64_t n = g->n, nwords = ((n + 127) >> 7) << 2;
  GRE_CHECK(ensure_arc_bits(g, nwords));
  uint32_t* vis;
  uint2 *q0, *q1;
  BfsCtl* c;
  const uint64_t cap = n + g->m / kPiece + 1;
  GRE_CHECK(ws_array(g, WS_A, 2 * nwords, &vis));
  GRE_CHECK(ws_array(g, WS_B, cap, &q0));
  GRE_CHECK(ws_array(g, WS_C, cap, &q1));
  unsigned char* mem;  // the control blocks, then the recorded counts
  GRE_CHECK(ws_array(g, WS_D, sizeof(BfsCtl) * nsearch + sizeof(unsigned long long) * GRE_MAX_RECORDED_SUPERSTEPS, &mem));
  c = (BfsCtl*)mem;
  rec = record ? (unsigned long long*)(c + nsearch) : nullptr;
  GRE_CUDA(cudaMemsetAsync(c, 0, sizeof(BfsCtl) * nsearch, g->stream));
  ctl = c;
  searches = nsearch;
  static int per_sm = 0;
  if (!per_sm) {
    int b = 0;
    GRE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_bfs_persist, kBfsThreads, 0));
    per_sm = b > 0 ? b : 1;
  }
  // a small graph's levels are barriers more than work: fewer blocks, cheaper barriers
  grid = (int)std::min<uint64_t>((uint64_t)num_sms() * per_sm, std::max<uint64_t>(1, std::max(n, g->m / 4) / kBfsThreads));
  run.reset(new BfsRun());
  BfsRun& R = *run;
  R.n = n;
  R.m = g->m;
  R.nwords = nwords;
  R.off = g->off;
  R.col = g->col;
  R.roff = g->roff;
  R.rcol = g->rcol;
  R.arc_bits = g->arc_bits;
  R.perm = caller_order ? g->perm : nullptr;
  R.vis0 = vis;
  R.vis1 = vis + nwords;
  R.q0 = q0;
  R.q1 = q1;
  R.rec = rec;
  R.nrec = GRE_MAX_RECORDED_SUPERSTEPS;
  R.wait_ns = grid_wait_ns();
  return GRE_SUCCESS;
}

int BfsPlan::search(uint32_t i, const uint32_t* droots, uint32_t nroots, uint32_t root, int32_t* level) {
  BfsRun& R = *run;
  R.roots = droots;
  R.nroots = nroots;
  R.root = root;
  R.level = level;
  R.ctl = (BfsCtl*)ctl + i;
  void* args[] = {&R};
  GRE_CUDA(cudaLaunchCooperativeKernel((const void*)k_bfs_persist, dim3(grid), dim3(kBfsThreads), args, 0, g->stream));
  launch_count_add(1);
  return GRE_SUCCESS;
}

int BfsPlan::collect(gre_stats* st, uint64_t* reached_arcs) {
  // one read for the control blocks and the first recorded counts
  constexpr uint32_t kFirst = 64;
  std::vector<BfsCtl> h(searches + (rec ? (sizeof(unsigned long long) * kFirst + sizeof(BfsCtl) - 1) / sizeof(BfsCtl) : 0));
  GRE_CUDA(cudaMemcpyAsync(h.data(), ctl, sizeof(BfsCtl) * searches + (rec ? sizeof(unsigned long long) * kFirst : 0),
                           cudaMemcpyDeviceToHost, g->stream));
  GRE_CUDA(cudaStreamSynchronize(g->stream));
  *reached_arcs = 0;
  for (uint32_t i = 0; i < searches; ++i) {
    const BfsCtl& c = h[i];
    if (c.bar.err) {
      set_error("gre_bfs: a grid barrier wait of the level loop ran out (%lld ms budget)", (long long)(run->wait_ns / 1000000ll));
      return GRE_TIMEOUT;
    }
    *reached_arcs += c.reached_arcs;
    if (!st) continue;
    st->supersteps += c.levels ? c.levels - 1 : 0;  // getSuperstepCount: the empty level is not counted
    st->arcs_traversed += c.arcs_td + c.arcs_bu;
    st->algo_bytes += c.bytes;
  }
  if (rec && st) {
    const uint32_t k = std::min<uint32_t>(h[searches - 1].levels, GRE_MAX_RECORDED_SUPERSTEPS);
    const unsigned long long* a = (const unsigned long long*)(h.data() + searches);
    std::vector<unsigned long long> all;
    if (k > kFirst) {
      all.resize(k);
      GRE_CUDA(cudaMemcpy(all.data(), rec, sizeof(unsigned long long) * k, cudaMemcpyDeviceToHost));
      a = all.data();
    }
    for (uint32_t i = 0; i < k; ++i) stats_record(st, a[i]);
  }
  return GRE_SUCCESS;
}

BfsPlan::BfsPlan() = default;
BfsPlan::~BfsPlan() = default;

// One search from device roots, levels by internal id, waited for.
int bfs_levels(gre_graph g, const uint32_t* droots, uint32_t nroots, int32_t* level, gre_stats* st) {
  BfsPlan p;
  uint64_t arcs = 0;
  GRE_CHECK(p.prepare(g, 1, false, false));
  GRE_CHECK(p.search(0, droots, nroots, 0, level));
  return p.collect(st, &arcs);
}

}  // namespace gre
