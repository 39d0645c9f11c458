// SSSP fast path: near-far frontier relaxation with uint32 weights.
//
// Same fixed point as the reference SSSP plugin (Kernels/SSSP.hpp:55-89: scatter last[u]+w,
// combine = min, every improved vertex re-activated): shortest-path distances are unique, so
// the result is bit-exact whatever the relaxation order.  Differences from the reference's
// superstep, chosen for the GPU:
//   * near-far ordering (Davidson et al., IPDPS 2014): improved vertices below a moving limit
//     form the next frontier, the others wait in a far set until the limit (raised by a bucket
//     width delta, or to the smallest waiting distance + delta) passes them; with the light/heavy
//     split of delta-stepping (Meyer and Sanders 2003) only arcs lighter than delta are relaxed
//     inside a bucket and a settled bucket's heavy arcs once.  On RMAT this relaxes each arc
//     about 1.1 times instead of about 2.2 for a plain Bellman-Ford frontier (delta = 0);
//   * the superstep loop runs in one cooperative kernel (sssp_loop.cu): frontiers are queues of
//     128-arc items, so hubs do not serialise a warp, and sets (near, bucket, far) are bitmaps;
//   * passes over a large share of the graph go through the degree bins (below), where an
//     improvement is a fire-and-forget atomic min on the distance plus a bit in a changed bitmap: no
//     thread waits for an atomic's reply (hub heads receive thousands per superstep);
//   * the distance of a frontier vertex is read when its arcs are relaxed (not a copy taken at the
//     start of the superstep), which can only lower the values sent;
//   * vertices without out-arcs are never queued (they have nothing to relax).
//
// Byte model per superstep: 16 F (queue + offsets) + 12 A (column + weight + dist probe)
// + 8 N (queue append + bitmap), F frontier, A arcs relaxed, N improved vertices.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstdlib>

#include "gre_internal.cuh"
#include "rows.cuh"
#include "sssp_loop.cuh"

namespace gre {

template <class T>
static int ws_array(gre_graph g, int slot, uint64_t count, T** p) {
  void* v = nullptr;
  GRE_CHECK(g->ws.get(slot, sizeof(T) * (count ? count : 1), &v));
  *p = (T*)v;
  return GRE_SUCCESS;
}


// Light/heavy split of each row for bucket width delta (warp per row, stable within a class).
__global__ void k_split_light_heavy(uint64_t n, const uint64_t* __restrict__ off, const uint32_t* __restrict__ col,
                                    const uint32_t* __restrict__ w, uint32_t delta, uint32_t* __restrict__ ocol,
                                    uint32_t* __restrict__ ow, uint64_t* __restrict__ lsplit) {
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t below = (1u << lane) - 1u;
  for (uint64_t v = warp; v < n; v += nwarps) {
    const uint64_t a0 = off[v], a1 = off[v + 1];
    uint64_t nlight = 0;
    for (uint64_t b = a0; b < a1; b += 32) {
      const bool light = b + lane < a1 && w[b + lane] < delta;
      nlight += __popc(__ballot_sync(0xffffffffu, light));
    }
    uint64_t lc = a0, hc = a0 + nlight;
    for (uint64_t b = a0; b < a1; b += 32) {
      const bool in = b + lane < a1;
      const uint32_t x = in ? w[b + lane] : 0u;
      const bool light = in && x < delta;
      const uint32_t lm = __ballot_sync(0xffffffffu, light);
      const uint32_t hm = __ballot_sync(0xffffffffu, in && !light);
      if (in) {
        const uint64_t dst = light ? lc + __popc(lm & below) : hc + __popc(hm & below);
        ocol[dst] = col[b + lane];
        ow[dst] = x;
      }
      lc += __popc(lm);
      hc += __popc(hm);
    }
    if (lane == 0) lsplit[v] = a0 + nlight;
  }
}

// Edge-balanced expansion in tiles of kTile consecutive frontier arcs (the partitioned path, whose
// offers are exchanged between the supersteps).  k_tile_starts records,
// for every tile, the frontier index owning its first arc (each frontier vertex writes the
// tiles that begin inside its arc range, so every entry is written exactly once).  A CTA then
// stages the owners of its tile (at most kTile + 1 of them, since queued vertices have at least
// one out-arc) in shared memory and each thread finds the owner of its arc there: the per-arc
// search touches shared memory only, and the column and weight reads of one vertex coalesce.
// Queue appends are gathered per tile in shared memory and reserved with one global atomic per
// tile, so the queue counters are not a point of contention.
constexpr int kTileThreads = 256;
constexpr int kTileItems = 8;
constexpr uint64_t kTile = (uint64_t)kTileThreads * kTileItems;
static_assert(kTileItems == 8, "owner scan packs 8 uint16 per thread");

struct MaxOp {
  __device__ __forceinline__ uint32_t operator()(uint32_t a, uint32_t b) const { return a > b ? a : b; }
};

__global__ void k_tile_starts(const uint64_t* __restrict__ prefix, uint64_t nq, uint32_t* __restrict__ start) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nq; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t p0 = prefix[i], p1 = prefix[i + 1];
    if (p1 == p0) continue;
    for (uint64_t t = (p0 + kTile - 1) / kTile; t <= (p1 - 1) / kTile; ++t) start[t] = (uint32_t)i;
  }
}

// Offer forms: an arc to head x offering nd.  A head in `own` is relaxed in place (its distance
// probed, lowered by atomic min, its pending bit set when it has out-arcs); another head is
// probed against known[x] (when given) and the offer array, and offered by atomic min with its
// bit in `touched`.  probe() returns the value nd must beat; commit() applies an offer that does.
struct OfferArc {
  uint64_t lx;
  bool mine;
  __device__ __forceinline__ uint32_t probe(const OwnHeads& o, const uint32_t* known, const uint32_t* offers, uint32_t x,
                                            uint32_t nd) {
    lx = (uint64_t)x - o.lo;
    mine = lx < o.len;
    if (mine) return __ldcg(o.dist + lx);
    if (known && nd >= __ldcg(known + x)) return 0u;
    return __ldcg(offers + x);
  }
  __device__ __forceinline__ void commit(const OwnHeads& o, uint32_t* offers, uint32_t* touched, uint32_t x, uint32_t nd) const {
    if (mine) {
      atomicMin(o.dist + lx, nd);
      if (o.outdeg[lx]) atomicOr(o.pend + (lx >> 5), 1u << (lx & 31u));
    } else {
      atomicMin(offers + x, nd);
      if (touched) atomicOr(touched + (x >> 5), 1u << (x & 31u));
    }
  }
};

// The partitioned path's relaxation: the owners' distances come from srcdist and `dist` is a separate
// offer array; an improved entry sets its bit in `changed` when that bitmap is given.
__global__ void __launch_bounds__(kTileThreads) k_sssp_relax(const uint32_t* __restrict__ queue, uint64_t nq,
                                                             const uint64_t* __restrict__ prefix, uint64_t total, const uint32_t* __restrict__ start,
                                                             const uint64_t* __restrict__ base, const uint32_t* __restrict__ col,
                                                             const uint32_t* __restrict__ w, const uint32_t* __restrict__ srcdist,
                                                             uint32_t* __restrict__ dist, uint32_t* __restrict__ changed,
                                                             uint32_t* __restrict__ error, const uint32_t* __restrict__ known,
                                                             const OwnHeads own) {
  using OwnerScan = cub::BlockScan<uint32_t, kTileThreads>;
  __shared__ uint64_t s_arc[kTile + 1];                // arc index at tile position s_rel[j]
  __shared__ uint32_t s_du[kTile + 1];                 // distance of owner j
  __shared__ uint16_t s_rel[kTile + 1];                // first tile position of owner j
  __shared__ __align__(16) uint16_t s_own[kTile];      // owner of each tile position
  __shared__ typename OwnerScan::TempStorage s_scan;
  const uint64_t ntiles = (total + kTile - 1) / kTile;
  for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const uint64_t t0 = tile * kTile;
    const uint32_t len = (uint32_t)(total - t0 < kTile ? total - t0 : kTile);
    const uint64_t lo = start[tile];
    const uint64_t hi = tile + 1 < ntiles ? start[tile + 1] : nq - 1;
    const uint64_t cnt = hi - lo + 1;
    if (cnt > kTile + 1) {  // cannot happen while every queued vertex has an out-arc; uniform
      if (threadIdx.x == 0) atomicOr(error, 1u);
      continue;
    }
    *(uint4*)(s_own + threadIdx.x * kTileItems) = make_uint4(0, 0, 0, 0);
    for (uint64_t j = threadIdx.x; j < cnt; j += kTileThreads) {
      const uint32_t u = queue[lo + j];
      const uint64_t p = prefix[lo + j];
      const uint64_t r = p > t0 ? p - t0 : 0;
      s_rel[j] = (uint16_t)r;
      s_arc[j] = base[u] + (t0 + r - p);
      s_du[j] = __ldcg(srcdist + u);
    }
    __syncthreads();
    // owner of every tile position: mark where each owner's arcs begin, then a running maximum
    // (owners begin at strictly increasing positions, every queued vertex having an out-arc)
    for (uint32_t j = 1 + threadIdx.x; j < cnt; j += kTileThreads)
      if (s_rel[j] < len) s_own[s_rel[j]] = (uint16_t)j;
    __syncthreads();
    {
      uint32_t own[kTileItems];
      const uint4 raw = *(const uint4*)(s_own + threadIdx.x * kTileItems);
      const uint32_t wds[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        own[2 * k] = wds[k] & 0xffffu;
        own[2 * k + 1] = wds[k] >> 16;
      }
      OwnerScan(s_scan).InclusiveScan(own, own, MaxOp());
      *(uint4*)(s_own + threadIdx.x * kTileItems) =
          make_uint4(own[0] | own[1] << 16, own[2] | own[3] << 16, own[4] | own[5] << 16, own[6] | own[7] << 16);
    }
    __syncthreads();
    // the thread's kTileItems arcs in rounds of independent loads (column and weight, then the
    // head's distance); an improvement is a fire-and-forget atomic min plus a bit in `changed`,
    // so no thread waits for an atomic's reply (hub heads receive many of them)
    uint32_t du[kTileItems], v[kTileItems], wt[kTileItems], dv[kTileItems];
#pragma unroll
    for (int k = 0; k < kTileItems; ++k) {
      const uint32_t t = (uint32_t)k * kTileThreads + threadIdx.x;
      const uint32_t a = s_own[t];
      const uint64_t arc = s_arc[a] + (t - s_rel[a]);
      du[k] = s_du[a];
      const bool ok = t < len;
      v[k] = ok ? __ldg(col + arc) : 0u;
      wt[k] = ok ? __ldg(w + arc) : 0u;
    }
    OfferArc oa[kTileItems];
#pragma unroll
    for (int k = 0; k < kTileItems; ++k) {
      const bool ok = (uint32_t)k * kTileThreads + threadIdx.x < len;
      dv[k] = ok ? oa[k].probe(own, known, dist, v[k], du[k] + wt[k]) : 0u;
    }
#pragma unroll
    for (int k = 0; k < kTileItems; ++k) {
      const uint32_t nd = du[k] + wt[k];
      if (nd < dv[k]) oa[k].commit(own, dist, changed, v[k], nd);
    }
    __syncthreads();
  }
}

// Large frontiers relaxed through the degree bins of the CSR instead of arc tiles: every bin's
// rows are scanned in order, and a row whose vertex is in the frontier bitmap relaxes its light
// ([off, lend)) or heavy ([lend, off+1)) arcs with 1..32 lanes (bins 0-5), a CTA (bin 6) or a CTA
// per 65536-arc chunk (bin 7).  No queue scan, no tile staging and no block barriers: the
// relaxations of a large frontier stream like the PageRank pull.  Same improvements (atomic min
// and a changed bit) as the tile kernel.
struct RelaxRange {
  const uint32_t* __restrict__ front;  // frontier bitmap
  const uint64_t* __restrict__ off;
  const uint64_t* __restrict__ lend;
  const uint32_t* __restrict__ col;
  const uint32_t* __restrict__ w;
  uint32_t* __restrict__ dist;
  uint32_t* __restrict__ changed;
  unsigned long long* __restrict__ arcs;  // arcs relaxed (statistics)
  bool heavy;
  const uint32_t* __restrict__ srcdist;  // OFFER form: the rows' own distances (dist holds offers)
  const uint32_t* __restrict__ known;    // OFFER form: upper bounds of the heads' distances (may be null)
  OwnHeads oh;                           // OFFER form: heads relaxed in place
  __device__ __forceinline__ bool in(uint32_t v) const { return (__ldg(front + (v >> 5)) >> (v & 31u)) & 1u; }
  __device__ __forceinline__ void range(uint32_t v, uint64_t* lo, uint64_t* hi) const {
    *lo = heavy ? lend[v] : off[v];
    *hi = heavy ? off[v + 1] : lend[v];
  }
  // arcs a, a + step, ... < hi offered du + w; four column/weight loads, then four distance
  // probes in flight per lane.  OFFER: dist is a separate offer array, probed and committed as
  // OfferArc says.
  template <bool OFFER>
  __device__ __forceinline__ uint32_t own(uint32_t v) const { return __ldcg((OFFER ? srcdist : dist) + v); }
  template <bool OFFER>
  __device__ __forceinline__ void relax(uint32_t du, uint64_t a, uint64_t hi, uint64_t step) const {
    for (; a + 3 * step < hi; a += 4 * step) {
      uint32_t x[4], nd[4], dv[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        x[k] = __ldg(col + a + k * step);
        nd[k] = du + __ldg(w + a + k * step);
      }
      if (OFFER) {
        OfferArc oa[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) dv[k] = oa[k].probe(oh, known, dist, x[k], nd[k]);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (nd[k] < dv[k]) oa[k].commit(oh, dist, changed, x[k], nd[k]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) dv[k] = __ldcg(dist + x[k]);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (nd[k] < dv[k]) {
            atomicMin(dist + x[k], nd[k]);
            if (changed) atomicOr(changed + (x[k] >> 5), 1u << (x[k] & 31u));
          }
      }
    }
    for (; a < hi; a += step) {
      const uint32_t x = __ldg(col + a);
      const uint32_t nd = du + __ldg(w + a);
      if (OFFER) {
        OfferArc oa;
        if (nd < oa.probe(oh, known, dist, x, nd)) oa.commit(oh, dist, changed, x, nd);
      } else if (nd < __ldcg(dist + x)) {
        atomicMin(dist + x, nd);
        if (changed) atomicOr(changed + (x >> 5), 1u << (x & 31u));
      }
    }
  }
};

// Rows of one bin (G lanes each) of block `part` of `nparts`.
template <int G, bool OFFER>
__device__ __forceinline__ void relax_lanes(const uint32_t* __restrict__ rows, uint64_t count, uint32_t part, uint32_t nparts,
                                            const RelaxRange& R, unsigned long long* arcs) {
  const uint32_t lig = threadIdx.x % G;
  for (uint64_t i = (uint64_t)part * (256 / G) + threadIdx.x / G; i < count; i += (uint64_t)nparts * (256 / G)) {
    const uint32_t v = rows[i];
    if (!R.in(v)) continue;
    uint64_t lo, hi;
    R.range(v, &lo, &hi);
    if (lo >= hi) continue;
    if (lig == 0) *arcs += hi - lo;
    R.template relax<OFFER>(R.template own<OFFER>(v), lo + lig, hi, G);
  }
}

// All bins in one launch, the longest rows first (rows::k_rows_all's plan): one after the other each
// bin's own tail of 15-25 us added up (RMAT-22, four sources: 10.1 -> 8.2 ms).
template <bool OFFER>
__global__ void __launch_bounds__(256) k_relax_all(const __grid_constant__ rows::RowPlan P, const RelaxRange R) {
  uint32_t s = 0;
  while (blockIdx.x >= P.block[s + 1]) ++s;
  const uint32_t part = blockIdx.x - P.block[s], nparts = P.block[s + 1] - P.block[s], count = P.count[s];
  const uint32_t* rows = P.rows + P.row0[s];
  unsigned long long arcs[1] = {0};
  if (s < 2) {
    // a CTA per row, or per chunk of a longer row: arcs [chunk_begin[c], + chunk) cut to the range
    for (uint64_t c = part; c < count; c += nparts) {
      const uint32_t v = rows[s == 0 ? P.chunk_row[c] : c];
      if (!R.in(v)) continue;
      uint64_t lo, hi;
      R.range(v, &lo, &hi);
      if (s == 0) {
        const uint64_t c0 = P.chunk_begin[c], c1 = c0 + P.chunk;
        lo = lo > c0 ? lo : c0;
        hi = hi < c1 ? hi : c1;
      }
      if (lo >= hi) continue;
      if (threadIdx.x == 0) arcs[0] += hi - lo;
      R.template relax<OFFER>(R.template own<OFFER>(v), lo + threadIdx.x, hi, 256);
    }
  } else if (s == 2) {
    relax_lanes<32, OFFER>(rows, count, part, nparts, R, arcs);
  } else if (s == 3) {
    relax_lanes<16, OFFER>(rows, count, part, nparts, R, arcs);
  } else if (s == 4) {
    relax_lanes<8, OFFER>(rows, count, part, nparts, R, arcs);
  } else if (s == 5) {
    relax_lanes<4, OFFER>(rows, count, part, nparts, R, arcs);
  } else if (s == 6) {
    relax_lanes<2, OFFER>(rows, count, part, nparts, R, arcs);
  } else {
    relax_lanes<1, OFFER>(rows, count, part, nparts, R, arcs);
  }
  __shared__ BlockSums<1> sums;
  if (R.arcs) sums.add(arcs, {R.arcs});  // null: the caller counts the arcs another way
}

template <bool OFFER>
static int relax_binned(const DegreeBins& B, const RelaxRange& R, cudaStream_t s) {
  const rows::RowPlan P = rows::plan_rows(B, false);
  if (P.block[8]) k_relax_all<OFFER><<<P.block[8], 256, 0, s>>>(P, R);
  GRE_LAUNCH_CHECK();
  return GRE_SUCCESS;
}

// Pull form of a large pass (direction-optimising, as bottom-up BFS): instead of the frontier
// pushing along its arcs, every vertex that can still improve scans its own light (or heavy)
// arcs for neighbours in the frontier bitmap and takes the smallest dist[u] + w.  Valid when the
// graph is symmetric and w(u->v) == w(v->u) (g->w32_symmetric): v's arc to u then carries the
// weight, and the light/heavy class, of u's arc to v, so the candidate values are exactly those
// the push would offer.  What it saves: the push's reads and atomics land on the heads, spread
// over all of dist (DRAM); the pull reads dist only at frontier vertices (on RMAT mostly the
// hubs, which the degree-ordered ids keep in L2) and writes each improved vertex once.  Rows
// whose distance is below `lo` are settled (every earlier bucket is final) and are skipped
// after one read of dist.
struct PullRange {
  const uint32_t* __restrict__ front;  // sources: the near frontier (light pass) or the bucket (heavy pass)
  const uint64_t* __restrict__ off;
  const uint64_t* __restrict__ lend;
  const uint32_t* __restrict__ col;
  const uint32_t* __restrict__ w;
  uint32_t* __restrict__ dist;               // the rows' distances (improved in place)
  uint32_t* __restrict__ changed;            // a bit per improved row
  unsigned long long* __restrict__ counts;  // [0] arcs scanned, [1] frontier hits
  bool heavy;
  uint32_t lo;
  const uint32_t* __restrict__ srcdist;      // the frontier's distances, indexed by column (the
                                             // one-GPU path: dist itself)
  __device__ __forceinline__ void range(uint32_t v, uint64_t* a0, uint64_t* a1) const {
    *a0 = heavy ? lend[v] : off[v];
    *a1 = heavy ? off[v + 1] : lend[v];
  }
  // smallest dist[u] + w over the arcs a, a + step, ... < hi whose tail u is in the frontier;
  // four column loads and bit tests in flight, then the hits' weights and distances
  __device__ __forceinline__ uint32_t best(uint64_t a, uint64_t hi, uint64_t step, unsigned long long* hits) const {
    uint32_t b = 0xffffffffu;
    for (; a + 3 * step < hi; a += 4 * step) {
      uint32_t u[4];
      bool in[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) u[k] = __ldg(col + a + k * step);
#pragma unroll
      for (int k = 0; k < 4; ++k) in[k] = (__ldg(front + (u[k] >> 5)) >> (u[k] & 31u)) & 1u;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (in[k]) {
          const uint32_t nd = __ldcg(srcdist + u[k]) + __ldg(w + a + k * step);
          b = nd < b ? nd : b;
          ++*hits;
        }
    }
    for (; a < hi; a += step) {
      const uint32_t u = __ldg(col + a);
      if ((__ldg(front + (u >> 5)) >> (u & 31u)) & 1u) {
        const uint32_t nd = __ldcg(srcdist + u) + __ldg(w + a);
        b = nd < b ? nd : b;
        ++*hits;
      }
    }
    return b;
  }
  __device__ __forceinline__ void improve(uint32_t v, uint32_t dv, uint32_t b) const {
    if (b < dv) {
      atomicMin(dist + v, b);
      atomicOr(changed + (v >> 5), 1u << (v & 31u));
    }
  }
};

// G lanes per row; the group's lanes share the row, so they take every branch together and the
// group minimum is a shuffle over the group's own lanes
template <int G>
__device__ __forceinline__ void pull_lanes(const uint32_t* __restrict__ rows, uint64_t count, uint32_t part, uint32_t nparts,
                                           const PullRange& R, unsigned long long (&n)[2]) {
  const uint32_t lane = threadIdx.x & 31u, lig = lane % G;
  const unsigned gmask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (lane - lig));
  for (uint64_t i = (uint64_t)part * (256 / G) + threadIdx.x / G; i < count; i += (uint64_t)nparts * (256 / G)) {
    const uint32_t v = rows[i];
    const uint32_t dv = __ldcg(R.dist + v);
    if (dv < R.lo) continue;
    uint64_t a0, a1;
    R.range(v, &a0, &a1);
    if (a0 >= a1) continue;
    if (lig == 0) n[0] += a1 - a0;
    uint32_t b = R.best(a0 + lig, a1, G, &n[1]);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      const uint32_t x = __shfl_xor_sync(gmask, b, o);
      b = x < b ? x : b;
    }
    if (lig == 0) R.improve(v, dv, b);
  }
}

// All bins in one launch, as k_relax_all.
__global__ void __launch_bounds__(256) k_pull_all(const __grid_constant__ rows::RowPlan P, const PullRange R) {
  uint32_t s = 0;
  while (blockIdx.x >= P.block[s + 1]) ++s;
  const uint32_t part = blockIdx.x - P.block[s], nparts = P.block[s + 1] - P.block[s], count = P.count[s];
  const uint32_t* rows = P.rows + P.row0[s];
  unsigned long long n[2] = {0, 0};  // arcs scanned, frontier hits
  if (s < 2) {
    // a CTA per row, or per chunk of a longer row, cut to the light or heavy range; each warp
    // offers its own minimum (at most 8 atomics per improved row or chunk)
    for (uint64_t c = part; c < count; c += nparts) {
      const uint32_t v = rows[s == 0 ? P.chunk_row[c] : c];
      const uint32_t dv = __ldcg(R.dist + v);
      if (dv < R.lo) continue;
      uint64_t a0, a1;
      R.range(v, &a0, &a1);
      if (s == 0) {
        const uint64_t c0 = P.chunk_begin[c], c1 = c0 + P.chunk;
        a0 = a0 > c0 ? a0 : c0;
        a1 = a1 < c1 ? a1 : c1;
      }
      if (a0 >= a1) continue;
      if (threadIdx.x == 0) n[0] += a1 - a0;
      const uint32_t b = __reduce_min_sync(0xffffffffu, R.best(a0 + threadIdx.x, a1, 256, &n[1]));
      if ((threadIdx.x & 31u) == 0) R.improve(v, dv, b);
    }
  } else if (s == 2) {
    pull_lanes<32>(rows, count, part, nparts, R, n);
  } else if (s == 3) {
    pull_lanes<16>(rows, count, part, nparts, R, n);
  } else if (s == 4) {
    pull_lanes<8>(rows, count, part, nparts, R, n);
  } else if (s == 5) {
    pull_lanes<4>(rows, count, part, nparts, R, n);
  } else if (s == 6) {
    pull_lanes<2>(rows, count, part, nparts, R, n);
  } else {
    pull_lanes<1>(rows, count, part, nparts, R, n);
  }
  __shared__ BlockSums<2> sums;
  sums.add(n, {R.counts, R.counts + 1});
}

static int pull_binned(const DegreeBins& B, const PullRange& R, cudaStream_t s) {
  const rows::RowPlan P = rows::plan_rows(B, false);
  if (P.block[8]) k_pull_all<<<P.block[8], 256, 0, s>>>(P, R);
  GRE_LAUNCH_CHECK();
  return GRE_SUCCESS;
}

int sssp_relax_binned_offer(cudaStream_t stream, const DegreeBins& B, const uint32_t* front, const uint64_t* off,
                            const uint64_t* lend, bool heavy, const uint32_t* col, const uint32_t* w, const uint32_t* srcdist,
                            uint32_t* offers, uint32_t* touched, const uint32_t* known, const OwnHeads& own,
                            unsigned long long* arcs) {
  RelaxRange R{front, off, lend, col, w, offers, touched, arcs, heavy, srcdist, known, own};
  return relax_binned<true>(B, R, stream);
}

int sssp_pull_binned(cudaStream_t stream, const DegreeBins& B, const uint32_t* front, const uint64_t* off, const uint64_t* lend,
                     bool heavy, const uint32_t* col, const uint32_t* w, const uint32_t* srcdist, uint32_t* dist, uint32_t* changed,
                     uint32_t lo, unsigned long long* counts) {
  PullRange P{front, off, lend, col, w, dist, changed, counts, heavy, lo, srcdist};
  return pull_binned(B, P, stream);
}

int sssp_split_rows(cudaStream_t stream, uint64_t rows, const uint64_t* off, const uint32_t* col, const uint32_t* w, uint32_t delta,
                    uint32_t* ocol, uint32_t* ow, uint64_t* lend) {
  if (rows) k_split_light_heavy<<<grid_for(rows * 32, 256), 256, 0, stream>>>(rows, off, col, w, delta, ocol, ow, lend);
  GRE_LAUNCH_CHECK();
  return GRE_SUCCESS;
}

struct AddU64 {
  __device__ __forceinline__ uint64_t operator()(uint64_t a, uint64_t b) const { return a + b; }
};

// Bucket width of the near-far split.  Default: 3/8 of the mean arc weight (RMAT-26, weights in
// [1, 255], heavy passes pulled: delta 24 / 32 / 40 / 48 / 64 / 96 / 128 gave 23.3 / 20.6 / 20.4
// / 19.9 / 20.4 / 22.2 / 25.0 ms); 0 relaxes every improved vertex at once (Bellman-Ford frontier).
// On a smaller graph a pass is a chain of round trips whatever its arcs, and arcs relaxed again cost less
// than a bucket more: 3/4 of the mean below 2^22 arcs, twice the mean below 2^20.  Four sources, weights in
// [1, 255], at 3/8, 3/4 and 2 of the mean: 26K arcs 1381 / 1076 / 1019 us, 135K 1827 / 1483 / 1353, 670K (directed)
// 2409 / 1993 / 1852, 1.9M 2356 / 2280 / 2407, 2.4M 3150 / 2761 / 3163, 9.7M 4520 / 4493 / 4783, 34M
// 5490 / 5823 / 6752.  (No buckets at all is faster still on these graphs up to 2^20 arcs, 1651 us at 670K, but
// nothing bounds what it relaxes again.)  The partitioned path takes the same width: a pass there is host-driven, so fewer
// buckets are worth more (two parts on one GPU, 3/8, 3/4 and 2 of the mean: 25K arcs 12.7 / 9.3 / 6.7 ms, 205K 12.6 / 9.2 / 5.9,
// 884K 15.2 / 10.6 / 6.7, 2.6M 15.4 / 11.2 / 7.0, 3.7M 16.6 / 11.4 / 7.9).
// The GRE_SSSP_DELTA environment variable overrides it.
constexpr uint64_t kWideBucketArcs = 1ull << 20, kNarrowBucketArcs = 1ull << 22;
int sssp_delta(gre_graph g, uint32_t* delta) {
  if (const char* e = getenv("GRE_SSSP_DELTA")) {
    *delta = (uint32_t)strtoul(e, nullptr, 10);
    return GRE_SUCCESS;
  }
  if (g->w32_mean < 0) {
    uint64_t* dsum = nullptr;
    GRE_CHECK(ws_array(g, WS_COUNTERS, 1, &dsum));
    size_t tb = 0;
    cub::DeviceReduce::Reduce(nullptr, tb, g->w32, dsum, g->m, AddU64(), (uint64_t)0, g->stream);
    void* tmp = nullptr;
    GRE_CHECK(g->ws.get(WS_CUB, tb, &tmp));
    GRE_CUDA(cub::DeviceReduce::Reduce(tmp, tb, g->w32, dsum, g->m, AddU64(), (uint64_t)0, g->stream));
    uint64_t sum = 0;
    GRE_CUDA(cudaMemcpyAsync(&sum, dsum, sizeof sum, cudaMemcpyDeviceToHost, g->stream));
    GRE_CUDA(cudaStreamSynchronize(g->stream));
    g->w32_mean = g->m ? (double)sum / (double)g->m : 1.0;
  }
  const double d = g->w32_mean * (g->m < kWideBucketArcs ? 2.0 : g->m < kNarrowBucketArcs ? 0.75 : 0.375);
  *delta = d < 1.0 ? 1u : d > 1e9 ? 1000000000u : (uint32_t)d;
  return GRE_SUCCESS;
}

// Resident CTAs of the relaxation kernel per SM: the grid is exactly one wave, so that no
// CTA starts its tiles late.
static int relax_blocks_per_sm() {
  static int per_sm = 0;
  if (!per_sm) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_sssp_relax, kTileThreads, 0) != cudaSuccess || b < 1) b = 1;
    per_sm = b;
  }
  return per_sm;
}

uint64_t sssp_tile_arcs() { return kTile; }

// Frontiers of at least n / binned_frontier() vertices are relaxed through the degree bins
// (default 16; the GRE_SSSP_BINNED environment variable overrides it, 0 = never).
static uint64_t binned_frontier() {
  if (const char* e = getenv("GRE_SSSP_BINNED")) return strtoull(e, nullptr, 10);
  return 16;
}
uint64_t sssp_binned_divisor() { return binned_frontier(); }

// A pass of the loop's kernel with at least this many arcs takes the wide form: no lane waits for
// its atomics, and a second phase over the bitmap classifies
// (GRE_SSSP_WIDE=<arcs> overrides).  RMAT-22, a pass of 8.5M arcs: 304 us classified on the spot, 145 us
// wide; thresholds of 2^16, 2^18 and 2^20 arcs measured alike (10.0-10.6 ms for four sources).
static uint64_t wide_pass() {
  if (const char* e = getenv("GRE_SSSP_WIDE")) return strtoull(e, nullptr, 10);
  return 1ull << 18;
}

// Below this many arcs no pass is long enough to leave the loop's kernel for (about 35 us of
// launches and a counter read), unless GRE_SSSP_BINNED asks for it.
constexpr uint64_t kBinnedMinArcs = 1ull << 22;

// Whether the large heavy passes pull (over the vertices that can still improve) instead of
// pushing (along the bucket's heavy arcs), where the weights allow it (g->w32_symmetric).
// Default on; the GRE_SSSP_PULL environment variable set to 0 keeps the push form.
static bool pull_enabled() {
  if (const char* e = getenv("GRE_SSSP_PULL")) return strtoul(e, nullptr, 10) != 0;
  return true;
}
bool sssp_pull_enabled() { return pull_enabled(); }

// A heavy pass whose bucket has at least m / d heavy arcs pulls even when the bucket has fewer
// than n / sssp_binned_divisor() members (a few hubs can carry a large share of the arcs): d from
// GRE_SSSP_PULL_ARCS, default 16; 0 decides by the member count alone.
static uint64_t pull_arcs_divisor() {
  if (const char* e = getenv("GRE_SSSP_PULL_ARCS")) return strtoull(e, nullptr, 10);
  return 16;
}
uint64_t sssp_pull_arcs_divisor() { return pull_arcs_divisor(); }

// The tuner picks the row schedule for the PageRank gather (RMAT-26: 16 arcs per lane, a warp up
// to 65536 arcs); SSSP's pushes wait on two dependent loads per four arcs, so longer chains per
// lane cost them (RMAT-26 SSSP 18.0 -> 19.4 ms under that schedule).  Their bins keep at most 8
// arcs per lane and a CTA from 16384 arcs.
int sssp_bins(gre_graph g, bool in, const DegreeBins** out) {
  GRE_CHECK(ensure_bins(g, in));
  const DegreeBins& B = in ? g->bins_in : g->bins_out;
  if (B.sched.lane_arcs <= 8 && B.sched.cta_min <= 16384) {
    *out = &B;
    return GRE_SUCCESS;
  }
  RowSchedule s = B.sched;
  s.lane_arcs = std::min<uint32_t>(s.lane_arcs, 8);
  s.cta_min = std::min<uint64_t>(s.cta_min, 16384);
  s.hub_chunk = 65536;
  s.seg_window = 0;
  DegreeBins& S = g->bins_sssp;
  if (!S.ready || S.sched.lane_arcs != s.lane_arcs || S.sched.cta_min != s.cta_min || S.sched.hub_chunk != s.hub_chunk)
    GRE_CHECK(build_bins(g, S, in ? g->roff : g->off, in ? g->rcol : g->col, s));
  *out = &S;
  return GRE_SUCCESS;
}

// The relaxation of one frontier pass of the partitioned path: tile starts, then k_sssp_relax over one
// wave of CTAs.
int sssp_relax_tiles(cudaStream_t stream, const uint32_t* queue, uint64_t nq, const uint64_t* prefix, uint64_t total,
                     uint32_t* tstart, const uint64_t* base, const uint32_t* col, const uint32_t* w, const uint32_t* srcdist,
                     uint32_t* dist, uint32_t* changed, uint32_t* error, const uint32_t* known, const OwnHeads& own) {
  if (!total) return GRE_SUCCESS;
  const uint64_t ntiles = (total + kTile - 1) / kTile;
  k_tile_starts<<<grid_for(nq, 256), 256, 0, stream>>>(prefix, nq, tstart);
  // the arc count is a launch argument: read inside the kernel instead, the relaxation
  // measured 1.7x slower on RMAT-26
  const int grid = (int)std::min<uint64_t>(ntiles, (uint64_t)num_sms() * relax_blocks_per_sm());
  k_sssp_relax<<<grid, kTileThreads, 0, stream>>>(queue, nq, prefix, total, tstart, base, col, w, srcdist, dist, changed, error,
                                                  known, own);
  GRE_LAUNCH_CHECK();
  return GRE_SUCCESS;
}

// Light/heavy split of the arcs for bucket width delta (built once per graph, weights and delta).
static int ensure_split(gre_graph g, uint32_t delta) {
  auto& sp = g->sssp_split;
  if (sp.lsplit && sp.delta == delta) return GRE_SUCCESS;
  sp.release();
  const uint64_t n = g->n, m = g->m;
  cudaError_t e = cudaMalloc(&sp.col, sizeof(uint32_t) * (m ? m : 1));
  if (e == cudaSuccess) e = cudaMalloc(&sp.w, sizeof(uint32_t) * (m ? m : 1));
  if (e == cudaSuccess) e = cudaMalloc(&sp.lsplit, sizeof(uint64_t) * (n ? n : 1));
  if (e != cudaSuccess) {
    sp.release();
    return cuda_status(e, "cudaMalloc (SSSP light/heavy split)", __FILE__, __LINE__);
  }
  k_split_light_heavy<<<grid_for(n * 32, 256), 256, 0, g->stream>>>(n, g->off, g->col, g->w32, delta, sp.col, sp.w, sp.lsplit);
  GRE_LAUNCH_CHECK();
  sp.delta = delta;
  return GRE_SUCCESS;
}

// One SSSP.  With delta > 0, near-far buckets of width delta with the light/heavy split of
// delta-stepping (Meyer and Sanders 2003): inside a bucket only light arcs (w < delta) are
// relaxed, repeatedly, as the bucket's distances settle; when the bucket is done, the heavy arcs
// of every vertex it settled are relaxed once (they can only reach later buckets).  delta = 0:
// Bellman-Ford frontier over all arcs.  The loop runs in sssp_loop.cu's kernel, which comes back
// for the passes over a large share of the graph.
static int sssp_one(gre_graph g, uint32_t src, uint32_t* dist, gre_stats* st, bool record, uint32_t delta, uint64_t* reached_arcs) {
  const uint64_t n = g->n, m = g->m;
  const uint64_t nwords = (n + 31) >> 5;
  if (delta) GRE_CHECK(ensure_split(g, delta));
  SsspRun R{};
  R.n = n;
  R.m = m;
  R.nwords = nwords;
  R.off = g->off;
  R.lend = delta ? g->sssp_split.lsplit : g->off + 1;
  R.col = delta ? g->sssp_split.col : g->col;
  R.w = delta ? g->sssp_split.w : g->w32;
  R.outdeg = g->outdeg;
  R.dist = dist;
  const uint64_t cap = n + m / kPiece + 1;
  uint32_t *bits, *front;
  GRE_CHECK(ws_array(g, WS_A, cap, &R.near[0]));
  GRE_CHECK(ws_array(g, WS_B, cap, &R.near[1]));
  GRE_CHECK(ws_array(g, WS_C, cap, &R.heavy[0]));
  GRE_CHECK(ws_array(g, WS_D, cap, &R.heavy[1]));
  GRE_CHECK(ws_array(g, WS_E, 7 * nwords, &bits));
  R.changed = bits;
  R.infar = bits + nwords;
  R.nbits[0] = bits + 2 * nwords;
  R.nbits[1] = bits + 3 * nwords;
  R.hbits[0] = bits + 4 * nwords;
  R.hbits[1] = bits + 5 * nwords;
  front = bits + 6 * nwords;
  R.all_out = g->symmetric();
  GRE_CHECK(ws_array(g, WS_F, 1, &R.ctl));
  if (record) GRE_CHECK(ws_array(g, WS_G, GRE_MAX_RECORDED_SUPERSTEPS, &R.rec));
  R.nrec = GRE_MAX_RECORDED_SUPERSTEPS;
  R.wait_ns = grid_wait_ns();
  R.src = src;
  R.delta = delta;
  R.limit = delta ? delta : 0xffffffffu;
  R.fresh = true;
  // the passes that go through the degree bins of the CSR (the symmetric CSC is the CSR)
  const bool pull = g->w32_symmetric && pull_enabled();
  const uint64_t bdiv = binned_frontier(), pdiv = pull_arcs_divisor();
  R.big_verts = R.big_arcs = ~0ull;
  R.wide_arcs = wide_pass();
  const DegreeBins* bins = nullptr;
  if (bdiv && (getenv("GRE_SSSP_BINNED") || m >= kBinnedMinArcs)) {
    GRE_CHECK(sssp_bins(g, g->symmetric(), &bins));
    R.big_verts = std::max<uint64_t>(1, n / bdiv);
    if (pull && pdiv) R.big_arcs = std::max<uint64_t>(1, (m + pdiv - 1) / pdiv);
  }
  SsspCtl h{};
  h.dmin[0] = h.dmin[1] = h.dmin[2] = 0xffffffffu;
  GRE_CUDA(cudaMemcpyAsync(R.ctl, &h, sizeof h, cudaMemcpyHostToDevice, g->stream));  // pageable: staged before the call returns
  uint64_t bytes = 0;
  uint32_t big = 0;
  for (;;) {
    GRE_CHECK(sssp_loop_launch(g, R));
    GRE_CUDA(cudaMemcpyAsync(&h, R.ctl, sizeof h, cudaMemcpyDeviceToHost, g->stream));
    GRE_CUDA(cudaStreamSynchronize(g->stream));
    if (h.bar.err) {
      set_error("gre_sssp: a grid barrier wait of the superstep loop ran out (%lld ms budget)", (long long)(R.wait_ns / 1000000ll));
      return GRE_TIMEOUT;
    }
    if (h.reason == SSSP_DONE) break;
    if (h.reason == SSSP_STUCK) {
      set_error("gre_sssp: near-far split made no progress");
      return GRE_FAILURE;
    }
    R.fresh = false;
    R.record_entry = true;
    R.limit = h.limit;
    ++big;
    const uint32_t* of = front;  // the pass's frontier as bits
    if (h.reason == SSSP_BIG_HEAVY) of = R.hbits[h.hb];
    else GRE_CHECK(sssp_items_to_bits(g, R.near[h.nb], h.near[h.p].items, nwords, front));
    if (h.reason == SSSP_BIG_HEAVY && pull) {
      // only vertices at or above the limit can improve (heavy arcs from the bucket land there).
      // (Light passes push: every unsettled vertex would have to scan its light arcs at every pass
      // of the bucket, measured slower than the push.)
      PullRange P{of, R.off, R.lend, R.col, R.w, dist, R.changed, R.ctl->pull_counts, true, R.limit, dist};
      GRE_CHECK(pull_binned(*bins, P, g->stream));
      bytes += 16 * n;  // per row: its id, distance and range bounds (arcs at the end)
    } else {
      RelaxRange P{of, R.off, R.lend, R.col, R.w, dist, R.changed, &R.ctl->big_arcs, h.reason == SSSP_BIG_HEAVY, nullptr};
      GRE_CHECK(relax_binned<false>(*bins, P, g->stream));
    }
    // the frontier is used up, and the next counters' successors are empty again
    uint32_t* used = h.reason == SSSP_BIG_HEAVY ? R.hbits[h.hb] : R.nbits[h.nb];
    GRE_CUDA(cudaMemsetAsync(used, 0, sizeof(uint32_t) * nwords, g->stream));
    R.p = (h.p + 1) % 3;
    R.nb = h.nb ^ 1;
    GRE_CUDA(cudaMemsetAsync(&R.ctl->near[(h.p + 2) % 3], 0, sizeof(SsspQueue), g->stream));
    R.q = h.q;
    R.hb = h.hb;
    R.r = h.r;
    if (h.reason == SSSP_BIG_HEAVY) {
      R.q = (h.q + 1) % 3;
      R.hb = h.hb ^ 1;
      GRE_CUDA(cudaMemsetAsync(&R.ctl->heavy[(h.q + 2) % 3], 0, sizeof(SsspQueue), g->stream));
    }
    GRE_CHECK(sssp_classify_bits(g, R));
    bytes += 4 * n + n / 8;  // rows scanned, bitmap (arcs at the end)
  }
  *reached_arcs = h.reached_arcs;
  bytes += h.bytes + 12 * h.big_arcs;                          // push: column + weight + distance probe per arc
  bytes += 4 * h.pull_counts[0] + 8 * h.pull_counts[1];        // pull: column per arc scanned (+ L2-held bitmap), weight + distance per hit
  if (st) {
    const uint32_t steps = h.steps + big;
    st->supersteps += steps ? steps - 1 : 0;
    st->arcs_traversed += h.relaxed + h.big_arcs + h.pull_counts[0];
    st->algo_bytes += bytes;
    if (record) {
      const uint32_t k = std::min<uint32_t>(h.nrec, GRE_MAX_RECORDED_SUPERSTEPS);
      std::vector<unsigned long long> a(k);
      if (k) GRE_CUDA(cudaMemcpy(a.data(), R.rec, sizeof(unsigned long long) * k, cudaMemcpyDeviceToHost));
      for (unsigned long long x : a) stats_record(st, x);
    }
  }
  return GRE_SUCCESS;
}

}  // namespace gre

using namespace gre;

extern "C" {

int gre_sssp(gre_graph g, const uint32_t* srcs, uint32_t nsrc, uint32_t* dist, gre_stats* st) {
  if (!g || !dist || (nsrc && !srcs)) return GRE_NULL;
  if (!g->w32) {
    set_error("gre_sssp: the graph has no uint32 weights (gre_graph_set_weights_*)");
    return GRE_INVALID_ARG;
  }
  GRE_CHECK(use_graph(g));
  stats_reset(st);
  const uint64_t n = g->n;
  std::vector<uint32_t> hs(nsrc);
  if (nsrc) GRE_CUDA(cudaMemcpy(hs.data(), srcs, sizeof(uint32_t) * nsrc, cudaMemcpyDefault));
  GRE_CHECK(map_ids(g, &hs, "gre_sssp"));
  uint32_t delta = 0;
  GRE_CHECK(sssp_delta(g, &delta));  // before any workspace pointer is taken (it may grow WS_CUB)
  uint32_t *dfinal, *dd;
  GRE_CHECK(prepare_output(g, dist, (uint64_t)nsrc * n, WS_OUTBUF, &dfinal));
  GRE_CHECK(perm_out_begin(g, dfinal, nsrc, 4, (void**)&dd));
  RunTimer timer(g);
  uint64_t edges = 0;
  for (uint32_t i = 0; i < nsrc; ++i) {
    uint64_t arcs = 0;
    GRE_CHECK(sssp_one(g, hs[i], dd + (uint64_t)i * n, st, st && nsrc == 1, delta, &arcs));
    edges += g->symmetric() ? arcs / 2 : arcs;
  }
  GRE_CHECK(perm_out_end(g, dd, dfinal, nsrc, 4));
  GRE_CHECK(finish_output(g, dist, dfinal, (uint64_t)nsrc * n));
  GRE_CHECK(timer.stop(st));
  if (st) st->traversed_edges = edges;
  return GRE_SUCCESS;
}

}  // extern "C"
