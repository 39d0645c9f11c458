// The 64-sources-per-word BFS: the level loop of a word in one cooperative kernel.
//
// A level of RMAT-20 is 20-150 us of work.  The loop before this one gave a hub's row to one warp in
// either direction (the second level's pull: 1350 us, 1 warp of 9000 busy at its end; the first level's
// push from 64 sources: 480 us), passed every vertex's word once more a level to commit it and wrote
// the 64 rows of levels in every level's pass.  Here
//   * push: the frontier is a queue of items (vertex, 128-arc piece of its row), the arcs of up to 32
//     items side by side on a warp; new bits gather in acc by atomicOr and a pass over the vertices
//     commits them;
//   * pull: rows by degree bin, long to short, L lanes a row; a row's owner commits it at once.  A row
//     of more than kHead arcs whose wanted sources are not all found in the first kHead goes on as tail
//     items of kTail arcs spread over the grid, committed after a second barrier;
//   * the levels are bit planes (bit b of the level of (v, source j) is bit j of plane b of v: 32 bytes a
//     vertex for levels below 16), which one pass at the end turns into the 64 rows in the caller's order.
// The pull looks for live sources only (those with a vertex on the current level): no other can reach a
// vertex on the next.  Both directions give the same words; the arcs counted are the same on every run
// (a tail item counts its arcs whether or not another one finds its sources first).
//
// 64 sources: RMAT-20 2.71 -> 0.57 ms, RMAT-22 9.5 -> 1.7, RMAT-24 28.3 -> 5.3 (with no level rows: 2.5 -> 0.4
// ms of the batched betweenness at RMAT-20).
//
// Words that one phase writes and the next reads go through plain loads (the barrier's fences order
// them), never the read-only path.  Barriers have a bounded wait (grid_sync.cuh): GRE_TIMEOUT.
#include "msbfs.cuh"

#include <algorithm>

#include "grid_sync.cuh"
#include "item_queue.cuh"

namespace gre {

namespace {

using u64 = unsigned long long;

constexpr int kMsThreads = 512;
constexpr uint32_t kHead = 512, kTail = 512;  // multiples of 128
constexpr uint32_t kPlanes = 4;               // bit planes of a group: levels below 16 need one, below 256 two, ...
constexpr uint32_t kDeepGroups = 7;           // groups after the first (levels below 2^32)

struct MsSlot {  // the frontier of one level
  u64 nf, bits, mf;  // vertices, (vertex, source) pairs, out-arcs of the vertices
  u64 scanned;       // arcs the pull that found it looked at
  u64 live;          // sources with a vertex on it
  unsigned int nitems, ntails;
};

struct MsCtl {
  GridBar bar;
  MsSlot slot[3];  // level d: slot d % 3; the next one is filled, the one after cleared
  u64 frontiers;     // vertices of all levels
  u64 push_levels, push_list, push_arcs, pull_levels, pull_scanned;
  unsigned int levels, d, queued, done;
};

struct MsRun {
  uint64_t n, m;
  const uint64_t* __restrict__ off;
  const uint32_t* __restrict__ col;
  const uint64_t* __restrict__ roff;
  const uint32_t* __restrict__ rcol;
  const uint32_t* __restrict__ rows;  // degree bins of the in-arcs
  uint64_t bin_start[DegreeBins::NB], bin_count[DegreeBins::NB];
  const uint32_t* __restrict__ srcs;
  uint32_t k;
  u64* seen;
  u64* acc;
  u64* front;   // frontier words of level d at (d & ring) * n
  uint32_t ring;
  u64* planes;  // null: none.  [n][4]: planes 0..3
  u64* deep[kDeepGroups];  // planes 4..7, 8..11, ..: [n][4] each
  uint2* q0;
  uint2* q1;
  uint32_t limit;  // levels from this one on wait for more space
  u64* rec;
  uint32_t nrec;
  MsCtl* ctl;
  long long wait_ns;
};

struct MsStage {
  u64 nf, bits, mf, scanned, live;
  unsigned int nitems, ntails;
  u64 any;
  ItemStage<kMsThreads> items;
  BlockSums<4> sums;
};
using MsAppend = ItemAppend<kMsThreads, uint2>;

__device__ __forceinline__ u64 warp_or(u64 x) {
  const unsigned int lo = __reduce_or_sync(0xffffffffu, (unsigned int)x), hi = __reduce_or_sync(0xffffffffu, (unsigned int)(x >> 32));
  return ((u64)hi << 32) | lo;
}

// What a thread found in a phase.
struct MsFound {
  u64 nf = 0, bits = 0, mf = 0, scanned = 0, any = 0;
  __device__ __forceinline__ void add_to(MsSlot* s, MsStage& st) {
    if (threadIdx.x == 0) st.any = 0;
    __syncthreads();
    const u64 w = warp_or(any);
    if (lane_id() == 0 && w) atomicOr(&st.any, w);
    st.sums.add({nf, bits, mf, scanned}, {&s->nf, &s->bits, &s->mf, &s->scanned});
    if (threadIdx.x == 0 && st.any) atomicOr(&s->live, st.any);
    __syncthreads();
  }
};

// New sources nb of vertex v at `level`.
__device__ __forceinline__ uint64_t commit(const MsRun& R, u64* next, uint64_t v, u64 nb, uint32_t level, MsFound& f) {
  next[v] = nb;
  if (!nb) return 0;
  R.seen[v] |= nb;
  if (R.planes) {
    for (uint32_t x = level & (16u - 1u); x; x &= x - 1) R.planes[v * 4 + __ffs(x) - 1] |= nb;
    for (uint32_t x = level >> kPlanes; x; x &= x - 1) {
      const uint32_t b = __ffs(x) - 1;
      R.deep[b / kPlanes][v * 4 + b % kPlanes] |= nb;
    }
  }
  const uint64_t deg = R.off[v + 1] - R.off[v];
  ++f.nf;
  f.bits += __popcll(nb);
  f.mf += deg;
  f.any |= nb;
  return deg;
}

__device__ __forceinline__ void push_items(const MsRun& R, const uint2* queue, uint32_t nitems, const u64* cur, uint32_t gwarp,
                                           uint32_t nwarps) {
  constexpr int U = 4;
  const uint32_t lane = lane_id();
  const uint32_t per = min(32u, max(1u, (nitems + nwarps - 1) / nwarps));
  for (uint64_t base = (uint64_t)gwarp * per; base < nitems; base += (uint64_t)nwarps * per) {
    uint64_t a0 = 0;
    uint32_t len = 0;
    u64 word = 0;
    if (lane < per && base + lane < nitems) {
      const uint2 it = __ldcg(queue + base + lane);
      a0 = R.off[it.x] + (uint64_t)it.y * kPiece;
      len = (uint32_t)min((uint64_t)kPiece, R.off[it.x + 1] - a0);
      word = cur[it.x];
    }
    const ItemSpan span(a0, len);
    for (uint32_t t = 0; t < span.total; t += 32 * U) {
      uint32_t v[U];
      u64 fu[U];
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const uint32_t pos = t + 32 * j + lane, own = span.owner(pos);
        const uint64_t arc = span.arc_of(pos, own);
        fu[j] = __shfl_sync(0xffffffffu, word, own);
        if (pos >= span.total) fu[j] = 0;
        v[j] = fu[j] ? __ldg(R.col + arc) : 0u;
      }
#pragma unroll
      for (int j = 0; j < U; ++j)
        if (fu[j]) fu[j] &= ~R.seen[v[j]];
#pragma unroll
      for (int j = 0; j < U; ++j)
        if (fu[j] && (__ldcg(R.acc + v[j]) & fu[j]) != fu[j]) atomicOr(R.acc + v[j], fu[j]);
    }
  }
}

// acc into the next frontier, and its items.
__device__ __forceinline__ void push_commit(const MsRun& R, u64* next, uint32_t level, uint2* out, MsSlot* sn, MsStage& st,
                                            uint32_t gwarp, uint32_t nwarps) {
  constexpr int U = 4;
  MsAppend append(st.items, &sn->nitems, out);
  MsFound f;
  for (uint64_t base = (uint64_t)gwarp * 32 * U; base < R.n; base += (uint64_t)nwarps * 32 * U) {
    u64 nb[U];
    uint32_t v[U], nit[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const uint64_t w = base + 32 * j + lane_id();
      nb[j] = w < R.n ? __ldcg(R.acc + w) : 0;
    }
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const uint64_t w = base + 32 * j + lane_id();
      v[j] = (uint32_t)w;
      nit[j] = 0;
      if (w < R.n) {
        if (nb[j]) R.acc[w] = 0;
        nit[j] = items_of(commit(R, next, w, nb[j], level, f));
      }
    }
    append.push(v, nit);
  }
  append.finish();
  f.add_to(sn, st);
}

// The frontier's items from its words.
__device__ __forceinline__ void words_to_items(const MsRun& R, const u64* cur, uint2* queue, unsigned int* count, MsStage& st,
                                               uint32_t gwarp, uint32_t nwarps) {
  MsAppend append(st.items, count, queue);
  for (uint64_t base = (uint64_t)gwarp * 32; base < R.n; base += (uint64_t)nwarps * 32) {
    const uint64_t w = base + lane_id();
    const uint32_t v[1] = {(uint32_t)w};
    const uint32_t nit[1] = {w < R.n && cur[w] ? items_of(R.off[w + 1] - R.off[w]) : 0u};
    append.push(v, nit);
  }
  append.finish();
}

// The rows of one bin, L lanes each; `task` is the warp's place in the bin's sequence, and comes
// back as its place in what follows.
template <int L>
__device__ __forceinline__ void pull_lanes(const MsRun& R, int bin, uint64_t& task, uint32_t nwarps, u64 live, const u64* cur,
                                           u64* next, uint32_t level, MsFound& f) {
  constexpr uint32_t G = 32 / L;
  const uint32_t lane = lane_id(), lig = lane % L;
  const uint64_t count = R.bin_count[bin], tasks = (count + G - 1) / G;
  const uint32_t* rows = R.rows + R.bin_start[bin];
  for (; task < tasks; task += nwarps) {
    const uint64_t i = task * G + lane / L;
    u64 got = 0, want = 0;
    uint64_t v = 0;
    if (i < count) {
      v = __ldg(rows + i);
      want = live & ~R.seen[v];
      if (want) {
        uint64_t a = R.roff[v] + lig;
        const uint64_t a1 = R.roff[v + 1];
        if (L == 1 && a < a1) {  // the hub of a relabelled graph: mostly ends it once it is on the frontier
          got = cur[__ldg(R.rcol + a)];
          ++f.scanned;
          a = (got & want) == want ? a1 : a + 1;
        }
        for (; a < a1; a += 4 * L) {
          uint32_t u[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) u[j] = a + j * L < a1 ? __ldg(R.rcol + a + j * L) : 0xffffffffu;
          u64 x[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] = u[j] != 0xffffffffu ? cur[u[j]] : 0;
#pragma unroll
          for (int j = 0; j < 4; ++j) f.scanned += u[j] != 0xffffffffu;
          got |= (x[0] | x[1]) | (x[2] | x[3]);
          if (L == 1 && (got & want) == want) break;
        }
      }
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) got |= __shfl_xor_sync(0xffffffffu, got, o);
    if (i < count && lig == 0) commit(R, next, v, got & want, level, f);
  }
  task -= tasks;
}

// Arcs [a, a1) by the warp until `want` is found; scanned counts per lane.
__device__ __forceinline__ u64 warp_gather(const MsRun& R, uint64_t a, uint64_t a1, u64 want, const u64* cur, u64& scanned) {
  const uint32_t lane = lane_id();
  u64 got = 0;
  if (a + lane < a1) {
    got = cur[__ldg(R.rcol + a + lane)];
    ++scanned;
  }
  got = warp_or(got);
  for (a += 32; a < a1 && (got & want) != want; a += 128) {
    uint32_t u[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) u[j] = a + 32 * j + lane < a1 ? __ldg(R.rcol + a + 32 * j + lane) : 0xffffffffu;
    u64 x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = u[j] != 0xffffffffu ? cur[u[j]] : 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) scanned += u[j] != 0xffffffffu;
    got = warp_or(got | (x[0] | x[1]) | (x[2] | x[3]));
  }
  return got;
}

// A warp a row, long rows first; what is left of a row after its first kHead arcs becomes tail items.
__device__ __forceinline__ void pull_long(const MsRun& R, uint64_t& task, uint32_t nwarps, u64 live, const u64* cur, u64* next,
                                          uint32_t level, uint2* tails, unsigned int* ntails, MsFound& f) {
  const uint32_t lane = lane_id();
  const uint64_t count = R.bin_count[5] + R.bin_count[6] + R.bin_count[7];
  const uint32_t* rows = R.rows + R.bin_start[5];
  for (; task < count; task += nwarps) {
    const uint64_t v = __ldg(rows + count - 1 - task);
    const u64 want = live & ~R.seen[v];
    if (!want) {
      if (lane == 0) next[v] = 0;
      continue;
    }
    const uint64_t a0 = R.roff[v], a1 = R.roff[v + 1];
    const u64 got = warp_gather(R, a0, min(a1, a0 + kHead), want, cur, f.scanned) & want;
    if (got != want && a1 - a0 > kHead) {
      const uint32_t pieces = (uint32_t)((a1 - a0 - kHead + kTail - 1) / kTail);
      uint32_t at = 0;
      if (lane == 0) {
        R.acc[v] = got;
        at = atomicAdd(ntails, pieces);
      }
      at = __shfl_sync(0xffffffffu, at, 0);
      for (uint32_t i = lane; i < pieces; i += 32) tails[at + i] = make_uint2((uint32_t)v, i);
    } else if (lane == 0) {
      commit(R, next, v, got, level, f);
    }
  }
  task -= count;
}

__device__ __forceinline__ void pull_tails(const MsRun& R, const uint2* tails, uint32_t ntails, u64 live, const u64* cur,
                                           uint32_t gwarp, uint32_t nwarps, MsFound& f) {
  const uint32_t lane = lane_id();
  for (uint64_t i = gwarp; i < ntails; i += nwarps) {
    const uint2 it = __ldcg(tails + i);
    const uint64_t a = R.roff[it.x] + kHead + (uint64_t)it.y * kTail, a1 = min(R.roff[it.x + 1], a + kTail);
    if (lane == 0) f.scanned += a1 - a;
    const u64 want = live & ~R.seen[it.x] & ~__ldcg(R.acc + it.x);
    u64 looked = 0;
    const u64 got = __shfl_sync(0xffffffffu, want, 0) ? warp_gather(R, a, a1, __shfl_sync(0xffffffffu, want, 0), cur, looked) & want : 0;
    if (lane == 0 && got) atomicOr(R.acc + it.x, got);
  }
}

__global__ void __launch_bounds__(kMsThreads, 2) k_msbfs(const __grid_constant__ MsRun R) {
  __shared__ MsStage st;
  const uint32_t gwarp = (blockIdx.x * kMsThreads + threadIdx.x) >> 5, nwarps = gridDim.x * (kMsThreads / 32);
  const uint64_t gtid = blockIdx.x * (uint64_t)kMsThreads + threadIdx.x, nthreads = (uint64_t)gridDim.x * kMsThreads;
  MsCtl* c = R.ctl;
  unsigned int target = 0;
  const bool first = blockIdx.x == 0 && threadIdx.x == 0;
  uint32_t d = c->d;  // above 0: a launch that goes on
  bool queued = d == 0 || c->queued, resumed = d != 0;
  if (d == 0) {
    for (uint64_t v = gtid; v < R.n; v += nthreads) {
      R.seen[v] = 0;
      R.acc[v] = 0;
      R.front[v] = 0;
      if (R.planes) {
        R.front[R.n + v] = 0;
        *(ulonglong2*)(R.planes + v * 4) = make_ulonglong2(0, 0);
        *(ulonglong2*)(R.planes + v * 4 + 2) = make_ulonglong2(0, 0);
      }
    }
    if (!grid_barrier(&c->bar, target, R.wait_ns)) return;
    if (blockIdx.x == 0) {  // the sources; a vertex that is several joins the queue once
      MsAppend append(st.items, &c->slot[0].nitems, R.q0);
      MsFound f;
      uint32_t v[1] = {0}, nit[1] = {0};
      if (threadIdx.x < R.k) {
        v[0] = R.srcs[threadIdx.x];
        const u64 bit = 1ull << threadIdx.x;
        atomicOr(R.seen + v[0], bit);
        ++f.bits;
        f.any = bit;
        if (atomicOr(R.front + v[0], bit) == 0) {
          const uint64_t deg = R.off[v[0] + 1] - R.off[v[0]];
          nit[0] = items_of(deg);
          f.mf += deg;
          ++f.nf;
        }
      }
      append.push(v, nit);
      append.finish();
      f.add_to(&c->slot[0], st);
    }
  }
  for (;; ++d) {
    MsSlot* s = &c->slot[d % 3];
    MsSlot* sn = &c->slot[(d + 1) % 3];
    if (!grid_barrier(&c->bar, target, R.wait_ns, [&] {
          st.nf = __ldcg(&s->nf);
          st.bits = __ldcg(&s->bits);
          st.mf = __ldcg(&s->mf);
          st.scanned = __ldcg(&s->scanned);
          st.live = __ldcg(&s->live);
          st.nitems = __ldcg(&s->nitems);
        }))
      return;
    const u64 live = st.live;
    const bool push = st.mf * 14 < R.m;
    if (first && !resumed) {
      c->pull_scanned += st.scanned;
      c->frontiers += st.nf;
      if (d > 0 && d - 1 < R.nrec) R.rec[d - 1] = st.bits;
      MsSlot* sz = &c->slot[(d + 2) % 3];  // last read a level ago
      sz->nf = sz->bits = sz->mf = sz->scanned = sz->live = 0;
      sz->nitems = sz->ntails = 0;
    }
    resumed = false;
    if (st.bits == 0) break;
    if (d + 1 >= R.limit && !(R.planes && st.mf == 0)) {  // the host makes room (for planes: if anything can follow)
      if (first) {
        c->d = d;
        c->queued = queued;
      }
      return;
    }
    const u64* cur = R.front + (d & R.ring) * R.n;
    u64* next = R.front + ((d + 1) & R.ring) * R.n;
    uint2* queue = (d & 1) ? R.q1 : R.q0;
    if (push) {
      if (first) {
        ++c->push_levels;
        c->push_list += st.nf;
        c->push_arcs += st.mf;
      }
      if (!queued) {
        words_to_items(R, cur, queue, &s->nitems, st, gwarp, nwarps);
        if (!grid_barrier(&c->bar, target, R.wait_ns, [&] { st.nitems = __ldcg(&s->nitems); })) return;
      }
      push_items(R, queue, st.nitems, cur, gwarp, nwarps);
      if (!grid_barrier(&c->bar, target, R.wait_ns)) return;
      push_commit(R, next, d + 1, (d & 1) ? R.q0 : R.q1, sn, st, gwarp, nwarps);
      queued = true;
    } else {
      if (first) ++c->pull_levels;
      // two levels share the words of level 0: a source without in-arcs is in no bin
      if (R.planes && d == 1 && blockIdx.x == 0 && threadIdx.x < R.k) {
        const uint32_t v = R.srcs[threadIdx.x];
        if (R.roff[v + 1] == R.roff[v]) next[v] = 0;
      }
      MsFound f;
      uint64_t task = gwarp;
      pull_long(R, task, nwarps, live, cur, next, d + 1, queue, &s->ntails, f);
      pull_lanes<16>(R, 4, task, nwarps, live, cur, next, d + 1, f);
      pull_lanes<8>(R, 3, task, nwarps, live, cur, next, d + 1, f);
      pull_lanes<4>(R, 2, task, nwarps, live, cur, next, d + 1, f);
      pull_lanes<2>(R, 1, task, nwarps, live, cur, next, d + 1, f);
      pull_lanes<1>(R, 0, task, nwarps, live, cur, next, d + 1, f);
      if (R.bin_count[5] + R.bin_count[6] + R.bin_count[7]) {
        if (!grid_barrier(&c->bar, target, R.wait_ns, [&] { st.ntails = __ldcg(&s->ntails); })) return;
        const uint32_t ntails = st.ntails;
        if (ntails) {
          pull_tails(R, queue, ntails, live, cur, gwarp, nwarps, f);
          if (!grid_barrier(&c->bar, target, R.wait_ns)) return;
          for (uint64_t i = gtid; i < ntails; i += nthreads) {
            const uint2 it = __ldcg(queue + i);
            if (it.y) continue;
            const u64 nb = __ldcg(R.acc + it.x);
            R.acc[it.x] = 0;
            commit(R, next, it.x, nb, d + 1, f);
          }
        }
      }
      f.add_to(sn, st);
      queued = false;
    }
  }
  if (first) {
    c->levels = d - 1;
    c->done = 1;
  }
}

struct MsDeep {
  const u64* group[kDeepGroups];
};

// The planes of 32 vertices a warp, in the caller's order, as one row of 32 levels a source.
template <bool DEEP>
__global__ void __launch_bounds__(256) k_ms_levels(uint64_t n, uint32_t k, uint32_t nplanes, const u64* __restrict__ seen,
                                                   const u64* __restrict__ planes, const __grid_constant__ MsDeep deep,
                                                   const uint32_t* __restrict__ iperm, const uint64_t* __restrict__ off,
                                                   int32_t* __restrict__ out, u64* __restrict__ reached) {
  u64 arcs = 0;
  for (uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; u < n; u += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t v = iperm ? __ldg(iperm + u) : u;
    const u64 s = seen[v];
    const ulonglong2 p01 = *(const ulonglong2*)(planes + v * 4), p23 = *(const ulonglong2*)(planes + v * 4 + 2);
    arcs += (u64)__popcll(s) * (off[v + 1] - off[v]);
#pragma unroll 8
    for (uint32_t j = 0; j < k; ++j) {
      uint32_t x = (uint32_t)((p01.x >> j) & 1ull) | (uint32_t)((p01.y >> j) & 1ull) << 1 | (uint32_t)((p23.x >> j) & 1ull) << 2 |
                   (uint32_t)((p23.y >> j) & 1ull) << 3;
      if constexpr (DEEP)
        for (uint32_t e = 0; e + kPlanes < nplanes; ++e)
          x |= (uint32_t)((deep.group[e / kPlanes][v * 4 + e % kPlanes] >> j) & 1ull) << (e + kPlanes);
      out[(uint64_t)j * n + u] = (s >> j) & 1ull ? (int32_t)x : -1;
    }
  }
  for (int o = 16; o > 0; o >>= 1) arcs += __shfl_xor_sync(0xffffffffu, arcs, o);
  if (lane_id() == 0 && arcs) atomicAdd(reached, arcs);
}

template <class T>
int ws_array(gre_graph g, int slot, uint64_t count, T** p) {
  void* v = nullptr;
  GRE_CHECK(g->ws.get(slot, sizeof(T) * (count ? count : 1), &v));
  *p = (T*)v;
  return GRE_SUCCESS;
}

// Frontier words of at least `levels` levels.  Rows without in-arcs are in no bin, so no pull writes
// their words: all start at zero.
int pool_levels(gre_graph g, uint64_t levels) {
  if (g->bc_fpool_levels >= levels) return GRE_SUCCESS;
  const uint64_t want = std::max<uint64_t>(levels, std::max<uint64_t>(32, 2 * g->bc_fpool_levels)), n = g->n;
  uint64_t* p = nullptr;
  GRE_CUDA(cudaMalloc(&p, sizeof(uint64_t) * n * want));
  if (g->bc_fpool) {
    GRE_CUDA(cudaMemcpyAsync(p, g->bc_fpool, sizeof(uint64_t) * n * g->bc_fpool_levels, cudaMemcpyDeviceToDevice, g->stream));
    GRE_CUDA(cudaStreamSynchronize(g->stream));
    cudaFree(g->bc_fpool);
  }
  GRE_CUDA(cudaMemsetAsync(p + n * g->bc_fpool_levels, 0, sizeof(uint64_t) * n * (want - g->bc_fpool_levels), g->stream));
  g->bc_fpool = p;
  g->bc_fpool_levels = want;
  return GRE_SUCCESS;
}

}  // namespace

int MsBfs::prepare(gre_graph graph, bool keep_levels) {
  g = graph;
  keep_ = keep_levels;
  const uint64_t n = g->n, cap = n + g->m / kPiece + 1;
  GRE_CHECK(ensure_bins(g, true));
  GRE_CHECK(ws_array(g, WS_A, n, &seen));
  GRE_CHECK(ws_array(g, WS_E, n, &acc_));
  GRE_CHECK(ws_array(g, WS_B, cap, &q0_));
  GRE_CHECK(ws_array(g, WS_C, cap, &q1_));
  GRE_CHECK(ws_array(g, WS_H, sizeof(MsCtl) + sizeof(u64) * GRE_MAX_RECORDED_SUPERSTEPS, &ctl_));
  if (keep_) {
    GRE_CHECK(pool_levels(g, 32));
  } else {
    GRE_CHECK(ws_array(g, WS_F, 2 * n, &front_));
    GRE_CHECK(ws_array(g, WS_D, 4 * n, &planes_));
  }
  static int per_sm = 0;
  if (!per_sm) {
    int b = 0;
    GRE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_msbfs, kMsThreads, 0));
    per_sm = b > 0 ? b : 1;
  }
  // a small graph's levels are barriers more than work: fewer blocks, cheaper barriers
  grid_ = (int)std::min<uint64_t>((uint64_t)num_sms() * per_sm, std::max<uint64_t>(1, std::max(n, g->m / 4) / kMsThreads));
  return GRE_SUCCESS;
}

int MsBfs::run(const uint32_t* dsrcs, uint32_t k, bool record) {
  const uint64_t n = g->n;
  MsCtl* ctl = (MsCtl*)ctl_;
  MsRun R{};
  R.n = n;
  R.m = g->m;
  R.off = g->off;
  R.col = g->col;
  R.roff = g->roff;
  R.rcol = g->rcol;
  R.rows = g->bins_in.rows;
  for (int b = 0; b < DegreeBins::NB; ++b) {
    R.bin_start[b] = g->bins_in.start[b];
    R.bin_count[b] = g->bins_in.count[b];
  }
  R.srcs = dsrcs;
  R.k = k;
  R.seen = seen;
  R.acc = acc_;
  R.planes = planes_;
  R.q0 = q0_;
  R.q1 = q1_;
  R.rec = (u64*)(ctl + 1);
  R.nrec = GRE_MAX_RECORDED_SUPERSTEPS;
  R.ctl = ctl;
  R.wait_ns = grid_wait_ns();
  R.ring = keep_ ? 0xffffffffu : 1u;
  R.limit = keep_ ? 0 : 1u << kPlanes;
  ngroups_ = 0;
  GRE_CUDA(cudaMemsetAsync(ctl, 0, sizeof(MsCtl), g->stream));
  MsCtl h;
  do {
    R.front = keep_ ? (u64*)g->bc_fpool : front_;
    if (keep_) R.limit = (uint32_t)std::min<uint64_t>(g->bc_fpool_levels, 0xffffffffu);
    for (uint32_t e = 0; e < ngroups_; ++e) R.deep[e] = deep_[e];
    void* args[] = {&R};
    GRE_CUDA(cudaLaunchCooperativeKernel((const void*)k_msbfs, dim3(grid_), dim3(kMsThreads), args, 0, g->stream));
    launch_count_add(1);
    GRE_CUDA(cudaMemcpyAsync(&h, ctl, sizeof h, cudaMemcpyDeviceToHost, g->stream));
    GRE_CUDA(cudaStreamSynchronize(g->stream));
    if (h.bar.err) {
      set_error("64-source BFS: a grid barrier wait of the level loop ran out (%lld ms budget)", (long long)(R.wait_ns / 1000000ll));
      return GRE_TIMEOUT;
    }
    if (h.done) break;
    // more levels than there is room for
    if (keep_) {
      GRE_CHECK(pool_levels(g, g->bc_fpool_levels + 1));
    } else {
      // a group more: all that levels up to n could need would be 192 bytes a vertex at 2^26 vertices
      constexpr int slots[kDeepGroups] = {WS_G, WS_J, WS_K, WS_L, WS_M, WS_N, WS_PERM_IN};
      u64** p = &deep_[ngroups_];
      GRE_CHECK(ws_array(g, slots[ngroups_], kPlanes * n, p));
      GRE_CUDA(cudaMemsetAsync(*p, 0, sizeof(u64) * kPlanes * n, g->stream));
      ++ngroups_;
      const uint32_t bits = kPlanes * (ngroups_ + 1);
      R.limit = bits < 32 ? 1u << bits : 0xffffffffu;
    }
    GRE_CUDA(cudaMemsetAsync(&ctl->bar, 0, sizeof(GridBar), g->stream));
  } while (true);
  levels = h.levels;
  frontier_vertices = h.frontiers;
  scanned += h.push_arcs + h.pull_scanned;
  bytes += 16 * h.push_list + 12 * h.push_arcs + 32 * n * h.push_levels + 24 * n * h.pull_levels + 12 * h.pull_scanned;
  if (record) {
    found.resize(std::min<uint32_t>(h.levels + 1, GRE_MAX_RECORDED_SUPERSTEPS));
    GRE_CUDA(cudaMemcpyAsync(found.data(), ctl + 1, sizeof(u64) * found.size(), cudaMemcpyDeviceToHost, g->stream));
    GRE_CUDA(cudaStreamSynchronize(g->stream));
  }
  return GRE_SUCCESS;
}

int MsBfs::write_levels(uint32_t k, int32_t* out, unsigned long long* reached) {
  const uint64_t n = g->n;
  uint32_t nplanes = kPlanes;
  while (nplanes < 32 && (levels >> nplanes)) ++nplanes;
  auto kernel = nplanes > kPlanes ? k_ms_levels<true> : k_ms_levels<false>;
  MsDeep deep{};
  for (uint32_t e = 0; e < ngroups_; ++e) deep.group[e] = deep_[e];
  kernel<<<grid_for(n, 256, 8), 256, 0, g->stream>>>(n, k, nplanes, seen, planes_, deep, g->iperm, g->off, out, reached);
  GRE_LAUNCH_CHECK();
  return GRE_SUCCESS;
}

}  // namespace gre
