// Betweenness centrality (Brandes), the reference's Forward/Backward plugins driven per source
// (Kernels/BC.hpp:56-163, usr/test_bc.cpp:63-110), accumulated bc(v) = sum_{s != v} dep_s(v).
//
// Per source the reference computes: forward, level and path count numPaths (sigma) by BFS
// with sum-combine; backward, one superstep per level i from the deepest down:
//   pathwgt[w] = (1 + dep[w]) / sigma[w] for w at level i, summed into each neighbour v,
//   dep[v] = sum[v] * sigma[v] for v at level i-1.
// Here both passes pull: a vertex v at level d adds, in its in-arc order, sigma[u] over
// neighbours u at level d-1 (forward) and (1 + dep[w]) / sigma[w] over neighbours w at level
// d+1 (backward).  Rows longer than 512 arcs are cut into fixed 512-arc chunks whose partial
// sums are added in chunk order.  Every per-(vertex, source) sum therefore has one association
// order, shared by:
//   * the single-source path (batched = 0): direction-optimising BFS levels, one thread per
//     vertex (or chunk) per level;
//   * the batched path (batched = 1): 64 sources per uint64 word.  The 64-source BFS (msbfs.cu) stores
//     the frontier word F_d[v] of every level; sigma and dep are [n][64] FP64 rows, a warp a row.
// so both produce bit-identical bc.  bc[v] adds dep_s(v) in source order in both.
//
// sigma is FP64 (the reference's int numPaths wraps beyond 2^31; the values agree below).
#include <algorithm>
#include <vector>

#include "gre_internal.cuh"
#include "item_queue.cuh"
#include "msbfs.cuh"

namespace gre {

constexpr uint64_t kBcChunk = 512;

template <class T>
static int ws_array(gre_graph g, int slot, uint64_t count, T** p) {
  void* v = nullptr;
  GRE_CHECK(g->ws.get(slot, sizeof(T) * (count ? count : 1), &v));
  *p = (T*)v;
  return GRE_SUCCESS;
}

// The arithmetic of one arc term, written with explicit rounding so that both paths (and any
// compiler contraction setting) perform exactly the same operations.
__device__ __forceinline__ double dep_term(double dep_w, double sigma_w) { return __ddiv_rn(__dadd_rn(1.0, dep_w), sigma_w); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }

// ---------------------------------------------------------------------------------------------
// single source
// ---------------------------------------------------------------------------------------------
__global__ void k_level_hist(uint64_t n, const int32_t* __restrict__ level, uint32_t* __restrict__ hist) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const int32_t l = level[v];
    if (l >= 0) atomicAdd(hist + l, 1u);
  }
}
__global__ void k_level_scatter(uint64_t n, const int32_t* __restrict__ level, uint32_t* __restrict__ cursor, uint32_t* __restrict__ list) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const int32_t l = level[v];
    if (l >= 0) list[atomicAdd(cursor + l, 1u)] = (uint32_t)v;
  }
}

struct Bc1 {
  const uint64_t* __restrict__ roff;
  const uint32_t* __restrict__ rcol;
  const int32_t* __restrict__ level;
  double* sigma;
  double* dep;
  // sum over arcs [a0, a1) of the forward (sigma) or backward (dep) term for level d
  __device__ __forceinline__ double fwd(uint64_t a0, uint64_t a1, int32_t d) const {
    double acc = 0.0;
    for (uint64_t a = a0; a < a1; ++a) {
      const uint32_t u = __ldg(rcol + a);
      if (level[u] == d - 1) acc = add(acc, sigma[u]);
    }
    return acc;
  }
  __device__ __forceinline__ double bwd(uint64_t a0, uint64_t a1, int32_t d) const {
    double acc = 0.0;
    for (uint64_t a = a0; a < a1; ++a) {
      const uint32_t w = __ldg(rcol + a);
      if (level[w] == d + 1) acc = add(acc, dep_term(dep[w], sigma[w]));
    }
    return acc;
  }
};

template <bool FWD>
__global__ void k_bc1_rows(const uint32_t* __restrict__ list, uint64_t cnt, int32_t d, Bc1 B, uint64_t ch) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < cnt; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = list[i];
    const uint64_t a0 = B.roff[v], a1 = B.roff[v + 1];
    if (a1 - a0 > ch) continue;  // chunked
    if (FWD) B.sigma[v] = B.fwd(a0, a1, d);
    else B.dep[v] = __dmul_rn(B.sigma[v], B.bwd(a0, a1, d));
  }
}

template <bool FWD>
__global__ void k_bc1_chunks(ChunkTable T, int32_t d, Bc1 B, double* __restrict__ partial) {
  for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < T.nchunks; c += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = T.rows[T.chunk_row[c]];
    if (B.level[v] != d) continue;
    const uint64_t a0 = T.chunk_begin[c];
    const uint64_t end = B.roff[v + 1];
    const uint64_t a1 = a0 + T.ch < end ? a0 + T.ch : end;
    partial[c] = FWD ? B.fwd(a0, a1, d) : B.bwd(a0, a1, d);
  }
}

template <bool FWD>
__global__ void k_bc1_finish(ChunkTable T, int32_t d, Bc1 B, const double* __restrict__ partial) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < T.nrows; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = T.rows[i];
    if (B.level[v] != d) continue;
    double s = 0.0;
    for (uint64_t c = T.first[i]; c < T.first[i + 1]; ++c) s = add(s, partial[c]);
    if (FWD) B.sigma[v] = s;
    else B.dep[v] = __dmul_rn(B.sigma[v], s);
  }
}

__global__ void k_bc1_init(uint64_t n, uint32_t s, double* __restrict__ sigma, double* __restrict__ dep) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    sigma[v] = (v == s) ? 1.0 : 0.0;
    dep[v] = 0.0;
  }
}

__global__ void k_bc1_accumulate(uint64_t n, uint32_t s, const double* __restrict__ dep, double* __restrict__ bc) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
    if (v != s) bc[v] = add(bc[v], dep[v]);
}

static int bc_single(gre_graph g, const std::vector<uint32_t>& hs, double* dbc, gre_stats* st) {
  const uint64_t n = g->n;
  const ChunkTable& T = g->bc_chunks;
  int32_t* level;
  double *sigma, *dep, *partial;
  uint32_t *list, *hist, *roots;
  GRE_CHECK(ws_array(g, WS_BC0, n, &level));
  GRE_CHECK(ws_array(g, WS_BC1, n, &sigma));
  GRE_CHECK(ws_array(g, WS_BC2, n, &dep));
  GRE_CHECK(ws_array(g, WS_BC3, n, &list));
  GRE_CHECK(ws_array(g, WS_BC5, T.nchunks + 1, &partial));
  GRE_CHECK(ws_array(g, WS_BC7, hs.size() + 1, &roots));
  GRE_CUDA(cudaMemcpyAsync(roots, hs.data(), sizeof(uint32_t) * hs.size(), cudaMemcpyHostToDevice, g->stream));
  uint64_t arcs = 0, bytes = 0;
  for (size_t i = 0; i < hs.size(); ++i) {
    const uint32_t s = hs[i];
    GRE_CHECK(bfs_levels(g, roots + i, 1, level, nullptr));
    // vertices grouped by level
    uint32_t nl = 0;
    {
      int32_t maxl = 0;
      // levels fit below n; a histogram of n+1 bins is enough
      GRE_CHECK(ws_array(g, WS_BC4, n + 2, &hist));
      GRE_CUDA(cudaMemsetAsync(hist, 0, sizeof(uint32_t) * (n + 2), g->stream));
      k_level_hist<<<grid_for(n, 256), 256, 0, g->stream>>>(n, level, hist);
      // BFS levels are contiguous from 0, so the first empty bin ends them; the bins are read
      // back in growing blocks until one holds an empty bin (one 16 KB read for most graphs)
      std::vector<uint32_t> hh;
      uint64_t have = 0;
      maxl = -1;
      while (maxl < 0 && have < n + 2) {
        const uint64_t take = std::min<uint64_t>(n + 2 - have, std::max<uint64_t>(4096, have));
        hh.resize(have + take);
        GRE_CUDA(cudaMemcpyAsync(hh.data() + have, hist + have, sizeof(uint32_t) * take, cudaMemcpyDeviceToHost,
                                 g->stream));
        GRE_CUDA(cudaStreamSynchronize(g->stream));
        uint64_t l = have;
        while (l < have + take && hh[l]) ++l;
        if (l < have + take) maxl = (int32_t)l - 1;
        have += take;
      }
      nl = (uint32_t)maxl + 1;
      std::vector<uint32_t> start(nl + 1, 0);
      for (uint32_t l = 0; l < nl; ++l) start[l + 1] = start[l] + hh[l];
      GRE_CUDA(cudaMemcpyAsync(hist, start.data(), sizeof(uint32_t) * nl, cudaMemcpyHostToDevice, g->stream));
      k_level_scatter<<<grid_for(n, 256), 256, 0, g->stream>>>(n, level, hist, list);
      k_bc1_init<<<grid_for(n, 256), 256, 0, g->stream>>>(n, s, sigma, dep);
      GRE_LAUNCH_CHECK();
      Bc1 B{g->roff, g->rcol, level, sigma, dep};
      for (int32_t d = 1; d < (int32_t)nl; ++d) {
        const uint64_t cnt = hh[d];
        k_bc1_rows<true><<<grid_for(cnt, 128, 8), 128, 0, g->stream>>>(list + start[d], cnt, d, B, T.ch);
        if (T.nchunks) {
          k_bc1_chunks<true><<<grid_for(T.nchunks, 128, 8), 128, 0, g->stream>>>(T, d, B, partial);
          k_bc1_finish<true><<<grid_for(T.nrows, 128, 4), 128, 0, g->stream>>>(T, d, B, partial);
        }
      }
      for (int32_t d = (int32_t)nl - 2; d >= 0; --d) {
        const uint64_t cnt = hh[d];
        k_bc1_rows<false><<<grid_for(cnt, 128, 8), 128, 0, g->stream>>>(list + start[d], cnt, d, B, T.ch);
        if (T.nchunks) {
          k_bc1_chunks<false><<<grid_for(T.nchunks, 128, 8), 128, 0, g->stream>>>(T, d, B, partial);
          k_bc1_finish<false><<<grid_for(T.nrows, 128, 4), 128, 0, g->stream>>>(T, d, B, partial);
        }
      }
      k_bc1_accumulate<<<grid_for(n, 256), 256, 0, g->stream>>>(n, s, dep, dbc);
      GRE_LAUNCH_CHECK();
    }
    arcs += 2 * g->m;
    bytes += 2 * (8 * (n + 1) + 4 * g->m) + 24 * n;
    if (st) st->supersteps += 2 * nl;
  }
  if (st) {
    st->arcs_traversed += arcs;
    st->algo_bytes += bytes;
  }
  return GRE_SUCCESS;
}

// ---------------------------------------------------------------------------------------------
// batched: 64 sources per word, a launch a level
//
// A warp takes a row, lane l on the columns 2l and 2l + 1 (one 16-byte load an arc).  A pass gathers rows
// of sigma: some 9 of 64 columns of an arc's neighbour are on the level before, in 5 of its 16 sectors, and
// 1.5 arcs of m meet a level in each pass (RMAT-18).  Instructions and the wait for those loads bound it:
//   * arcs are looked at 128 at a time (one long row, or four short ones side by side: column, frontier
//     word; the next 128 columns are on their way meanwhile), and what meets the row's word is queued in shared
//     memory.  Eight entries are loaded together, across the short rows' borders, without a test but the
//     columns' own bits: a queue ends in empty entries;
//   * a level is one launch: chunks of the long rows, whose last taker adds the partial sums (in chunk
//     order), long rows, short rows; the lists of the next level's vertices are made beside it and kept
//     for the backward pass;
//   * the backward pass turns an entry's sigma into the weight its parents pull, (1 + dep) / sigma, as
//     soon as its dependency is known (no other level reads that entry before the next one does);
//   * nothing is cleared: an entry is read only where a frontier word says it was written.
// Measured against a warp a row without these (nine launches a level, both tables cleared, the weights in
// a pass of their own; with the 64-source BFS of msbfs.cu on both sides): 64 sources at RMAT-20 8.5 -> 5.5 ms, RMAT-22
// 36.8 -> 24.3, RMAT-16 1.4 -> 0.8.  A level of RMAT-20 takes up to 1.1 ms at half of the issue slots.  Both passes in
// one cooperative kernel held the loop's state in the inner loops' registers: 7.0 ms.  Half a warp a row with
// 32-byte loads: 7.1-7.7 ms (unequal halves).  Four entries at a time and more warps: 7.2 ms.
// ---------------------------------------------------------------------------------------------
namespace {

using u64 = unsigned long long;
constexpr int kBcThreads = 256;
constexpr uint32_t kBcShort = 32;  // arcs of a short row at most
constexpr int kBcSegs = 4;         // segments of 32 arcs a warp looks at together
constexpr int kBcGroup = 8;        // entries loaded together

struct __align__(16) BcEntry {
  uint32_t v, pad;
  u64 mask;  // columns
};

// A level's part of the two lists of vertices.
struct BcList {
  uint64_t short0, long0;          // where it begins (known when the level before is complete); all levels together
                                   // may hold up to 64 n vertices
  unsigned int nshort, nlong;
};

struct BcRun {
  uint64_t n;
  const uint64_t* __restrict__ roff;
  const uint32_t* __restrict__ rcol;
  const u64* __restrict__ F;     // [levels + 1][n]
  const u64* __restrict__ seen;
  const uint32_t* __restrict__ srcs;
  uint32_t k, nl;                // levels 0 .. nl - 1 hold vertices; those of nl are zero
  ChunkTable T;
  double* sigma;                 // [n][64]
  double* dep;                   // [n][64]
  double* partial;               // [chunks][64]
  unsigned int* arrived;         // chunks of a long row so far (zero between levels)
  uint32_t* shorts;              // vertices of up to kBcShort in-arcs, level after level
  uint32_t* longs;               // up to the chunk length
  BcList* list;                  // [nl + 1], zero at first
};

struct BcStage {
  BcEntry entry[kBcThreads / 32][kBcSegs * 32 + kBcGroup];
  ItemStage<kBcThreads> shorts, longs;
};

template <bool FWD>
struct BcWarp {
  const uint64_t* __restrict__ roff;
  const uint32_t* __restrict__ rcol;
  const u64* __restrict__ fother;  // the level pulled from
  const u64* __restrict__ fd;      // the level at hand
  double* sigma;                   // from this lane's columns on
  double* dep;
  BcEntry* buf;                    // this warp's
  uint32_t lane;
  double a = 0.0, b = 0.0;

  __device__ __forceinline__ uint32_t cols(u64 mask) const {
    return ((lane < 16 ? (uint32_t)mask : (uint32_t)(mask >> 32)) >> (2 * (lane & 15u))) & 3u;
  }
  static __device__ __forceinline__ void store(double* to, double x, double y, uint32_t t) {
    if (t == 3u) *(double2*)to = make_double2(x, y);
    else if (t) to[t >> 1] = t & 1u ? x : y;
  }
  // the sums x, y of row v in its columns t; s: its sigma there (backward)
  __device__ __forceinline__ void finish(uint32_t v, uint32_t t, double x, double y, double2 s) const {
    const uint64_t row = (uint64_t)v * 64;
    if (!FWD) {
      x = __dmul_rn(s.x, x);
      y = __dmul_rn(s.y, y);
      store(dep + row, x, y, t);
      x = dep_term(x, s.x);
      y = dep_term(y, s.y);
    }
    store(sigma + row, x, y, t);
  }
  __device__ __forceinline__ double2 own_sigma(uint32_t v, uint32_t t) const {
    return !FWD && t ? *(const double2*)(sigma + (uint64_t)v * 64) : make_double2(1.0, 1.0);
  }
  // The queue's entries 0 .. cnt - 1 in order; before(p) ahead of entry p.
  template <int G, class Before>
  __device__ __forceinline__ void take(int cnt, Before&& before) {
    if (lane < G) buf[cnt + lane] = BcEntry{0u, 0u, 0ull};
    __syncwarp();
    for (int i = 0; i < cnt; i += G) {
      double2 x[G];
      uint32_t t[G];
#pragma unroll
      for (int j = 0; j < G; ++j) {
        const BcEntry e = buf[i + j];
        t[j] = cols(e.mask);
        // where a bit is set only
        asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p ld.global.v2.f64 {%0, %1}, [%2];\n}"
                     : "=d"(x[j].x), "=d"(x[j].y)
                     : "l"(sigma + (uint64_t)e.v * 64), "r"(t[j]));
      }
#pragma unroll
      for (int j = 0; j < G; ++j) {
        before(i + j);
        if (t[j] & 1u) a = add(a, x[j].x);
        if (t[j] & 2u) b = add(b, x[j].y);
      }
    }
    __syncwarp();
  }
  // this lane's arc of a segment joins the queue where it meets the row's word
  __device__ __forceinline__ void put(int& held, uint32_t u, u64 m) {
    const uint32_t ball = __ballot_sync(0xffffffffu, m != 0);
    if (m) buf[held + __popc(ball & ((1u << lane) - 1u))] = BcEntry{u, 0u, m};
    held += __popc(ball);
  }
  // arcs [a0, a1) into a, b
  __device__ __forceinline__ void row(uint64_t a0, uint32_t len, u64 mine) {
    const uint32_t* c = rcol + a0;
    uint32_t u[kBcSegs];
#pragma unroll
    for (int j = 0; j < kBcSegs; ++j) u[j] = 32 * j + lane < len ? __ldg(c + 32 * j + lane) : 0u;
    for (uint32_t base = 0; base < len; base += 32 * kBcSegs) {
      u64 m[kBcSegs];
#pragma unroll
      for (int j = 0; j < kBcSegs; ++j) m[j] = base + 32 * j + lane < len ? __ldg(fother + u[j]) & mine : 0ull;
      int held = 0;
#pragma unroll
      for (int j = 0; j < kBcSegs; ++j) {
        put(held, u[j], m[j]);
        const uint32_t p = base + 32 * (kBcSegs + j) + lane;
        u[j] = p < len ? __ldg(c + p) : 0u;
      }
      take<kBcGroup>(held, [](int) {});
    }
  }
  // vertices list[0 .. cnt - 1], at most kBcSegs of them
  __device__ __forceinline__ void short_rows(const uint32_t* list, uint32_t cnt) {
    uint32_t v = 0, len = 0;
    uint64_t a0 = 0;
    u64 mine = 0;
    if (lane < cnt) {
      v = list[lane];
      a0 = roff[v];
      len = (uint32_t)(roff[v + 1] - a0);
      mine = __ldg(fd + v);
    }
    uint32_t u[kBcSegs];
    u64 m[kBcSegs];
#pragma unroll
    for (int j = 0; j < kBcSegs; ++j) {
      const uint64_t p = __shfl_sync(0xffffffffu, a0, j) + lane;
      m[j] = lane < __shfl_sync(0xffffffffu, len, j) ? ~0ull : 0ull;
      u[j] = m[j] ? __ldg(rcol + p) : 0u;
    }
#pragma unroll
    for (int j = 0; j < kBcSegs; ++j) {
      const u64 word = __shfl_sync(0xffffffffu, mine, j);
      m[j] = m[j] ? __ldg(fother + u[j]) & word : 0ull;
    }
    int held = 0, end[kBcSegs];
#pragma unroll
    for (int j = 0; j < kBcSegs; ++j) {
      put(held, u[j], m[j]);
      end[j] = held;
    }
    double2 sum[kBcSegs];
    int r = 0, next = end[0];
    // the rows that end before entry p
    auto close = [&](int p) {
      while (p == next && r < kBcSegs) {
#pragma unroll
        for (int j = 0; j < kBcSegs; ++j)
          if (j == r) {
            sum[j] = make_double2(a, b);
            next = j + 1 < kBcSegs ? end[j + 1 < kBcSegs ? j + 1 : 0] : -1;
          }
        ++r;
        a = b = 0.0;
      }
    };
    take<kBcGroup / 2>(held, close);
    close(held);
    double2 s[kBcSegs];
    uint32_t t[kBcSegs];
#pragma unroll
    for (int j = 0; j < kBcSegs; ++j) {
      t[j] = cols(__shfl_sync(0xffffffffu, mine, j));
      s[j] = own_sigma(__shfl_sync(0xffffffffu, v, j), t[j]);
    }
#pragma unroll
    for (int j = 0; j < kBcSegs; ++j) {
      const uint32_t rv = __shfl_sync(0xffffffffu, v, j);
      if (t[j]) finish(rv, t[j], sum[j].x, sum[j].y, s[j]);
    }
  }
};

// The vertices of level d join the lists, behind those of the level before.
__device__ __forceinline__ void bc_lists(const BcRun& R, uint32_t d, BcStage& st) {
  const uint32_t gwarp = (blockIdx.x * kBcThreads + threadIdx.x) >> 5, nwarps = gridDim.x * (kBcThreads / 32);
  BcList at{0, 0, 0, 0};
  if (d) {
    at = R.list[d - 1];
    at.short0 += at.nshort;
    at.long0 += at.nlong;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      R.list[d].short0 = at.short0;
      R.list[d].long0 = at.long0;
    }
  }
  ItemAppend<kBcThreads, uint32_t> shorts(st.shorts, &R.list[d].nshort, R.shorts + at.short0),
      longs(st.longs, &R.list[d].nlong, R.longs + at.long0);
  const u64* f = R.F + d * R.n;
  for (uint64_t base = (uint64_t)gwarp * 32; base < R.n; base += (uint64_t)nwarps * 32) {
    const uint64_t v = base + lane_id();
    const bool on = v < R.n && __ldg(f + v) != 0;
    const uint64_t len = on ? R.roff[v + 1] - R.roff[v] : 0;
    shorts.push_one((uint32_t)v, on && len <= kBcShort);
    longs.push_one((uint32_t)v, on && len > kBcShort && len <= R.T.ch);
  }
  shorts.finish();
  longs.finish();
}

// Level d's lists (0, with the sources' path counts, and 1).
__global__ void __launch_bounds__(kBcThreads) k_bcm_first(const __grid_constant__ BcRun R, uint32_t d) {
  __shared__ BcStage st;
  if (d == 0 && blockIdx.x == 0 && threadIdx.x < R.k) R.sigma[(uint64_t)R.srcs[threadIdx.x] * 64 + threadIdx.x] = 1.0;
  bc_lists(R, d, st);
}

// Level d of a pass: chunks, long rows, short rows kBcSegs at a time; forward, the next level's lists.
template <bool FWD>
__global__ void __launch_bounds__(kBcThreads, 4) k_bcm_level(const __grid_constant__ BcRun R, uint32_t d) {
  __shared__ BcStage st;
  const uint32_t gwarp = (blockIdx.x * kBcThreads + threadIdx.x) >> 5, nwarps = gridDim.x * (kBcThreads / 32), lane = lane_id();
  BcWarp<FWD> W{R.roff, R.rcol, R.F + (FWD ? d - 1 : d + 1) * R.n, R.F + d * R.n, R.sigma + 2 * lane, R.dep + 2 * lane,
                st.entry[threadIdx.x >> 5], lane};
  const BcList at = R.list[d];
  const ChunkTable& T = R.T;
  uint64_t i = gwarp;
  const uint64_t nchunks = T.nchunks, nlong = at.nlong, rows = nchunks + nlong;
  const uint32_t* longs = R.longs + at.long0;
  for (; i < rows; i += nwarps) {
    const bool chunk = i < nchunks;
    const uint64_t r = chunk ? T.chunk_row[i] : 0;
    const uint32_t v = chunk ? T.rows[r] : longs[i - nchunks];
    const u64 mine = __ldg(W.fd + v);
    if (!mine) continue;
    const uint64_t a0 = chunk ? T.chunk_begin[i] : W.roff[v], left = W.roff[v + 1] - a0;
    W.row(a0, (uint32_t)min(left, T.ch), mine);
    if (chunk) {
      *(double2*)(R.partial + i * 64 + 2 * lane) = make_double2(W.a, W.b);
      W.a = W.b = 0.0;
      __threadfence();
      __syncwarp();
      uint64_t c = T.first[r];
      const uint64_t end = T.first[r + 1];
      unsigned int before = 0;
      if (lane == 0) before = atomicAdd(R.arrived + r, 1u);
      if (__shfl_sync(0xffffffffu, before, 0) + 1 < end - c) continue;
      // the row's last chunk
      __threadfence();
      if (lane == 0) R.arrived[r] = 0;
      for (; c < end; c += 8) {
        double2 x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          x[j] = c + j < end ? __ldcg((const double2*)(R.partial + (c + j) * 64 + 2 * lane)) : make_double2(0.0, 0.0);
#pragma unroll
        for (int j = 0; j < 8; ++j) {  // sums of positive terms: adding 0.0 changes nothing
          W.a = add(W.a, x[j].x);
          W.b = add(W.b, x[j].y);
        }
      }
    }
    const uint32_t t = W.cols(mine);
    if (t) W.finish(v, t, W.a, W.b, W.own_sigma(v, t));
    W.a = W.b = 0.0;
  }
  i -= rows;
  const uint64_t nshort = at.nshort;
  for (uint64_t t = i * kBcSegs; t < nshort; t += (uint64_t)nwarps * kBcSegs)
    W.short_rows(R.shorts + at.short0 + t, (uint32_t)min((uint64_t)kBcSegs, nshort - t));
  if (FWD && d + 1 < R.nl) bc_lists(R, d + 1, st);
}

// bc[v] adds the dependencies in source order; a source's own does not count.
__global__ void __launch_bounds__(256) k_bcm_accumulate(uint64_t n, const u64* __restrict__ seen, const u64* __restrict__ f0,
                                                        const double* __restrict__ dep, double* __restrict__ bc) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const u64 bits = seen[v] & ~f0[v];
    if (!bits) continue;
    double s = bc[v];
#pragma unroll 1
    for (uint32_t j0 = 0; j0 < 64; j0 += 16) {
      if (!((bits >> j0) & 0xffffull)) continue;
      double2 x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        x[j] = (bits >> (j0 + 2 * j)) & 3u ? *(const double2*)(dep + v * 64 + j0 + 2 * j) : make_double2(0.0, 0.0);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if ((bits >> (j0 + 2 * j)) & 1u) s = add(s, x[j].x);
        if ((bits >> (j0 + 2 * j)) & 2u) s = add(s, x[j].y);
      }
    }
    bc[v] = s;
  }
}

}  // namespace

static int bc_batched(gre_graph g, const std::vector<uint32_t>& hs, double* dbc, gre_stats* st) {
  if (hs.empty()) return GRE_SUCCESS;
  const uint64_t n = g->n;
  const ChunkTable& T = g->bc_chunks;
  BcRun R{};
  uint32_t* srcs;
  MsBfs word;
  GRE_CHECK(ws_array(g, WS_BC1, n * 64, &R.sigma));
  GRE_CHECK(ws_array(g, WS_BC2, n * 64, &R.dep));
  GRE_CHECK(ws_array(g, WS_BC5, (T.nchunks + 1) * 64, &R.partial));
  GRE_CHECK(ws_array(g, WS_BC7, hs.size(), &srcs));
  GRE_CHECK(word.prepare(g, true));
  GRE_CUDA(cudaMemcpyAsync(srcs, hs.data(), sizeof(uint32_t) * hs.size(), cudaMemcpyHostToDevice, g->stream));
  R.n = n;
  R.roff = g->roff;
  R.rcol = g->rcol;
  R.T = T;
  R.seen = word.seen;
  GRE_CHECK(ws_array(g, WS_BC6, T.nrows, &R.arrived));
  GRE_CUDA(cudaMemsetAsync(R.arrived, 0, sizeof(unsigned int) * T.nrows, g->stream));
  static int per_sm = 0;
  if (!per_sm) {
    int b = 0;
    GRE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_bcm_level<true>, kBcThreads, 0));
    per_sm = b > 0 ? b : 1;
  }
  const int grid = grid_for(std::max(n, g->m / 4), kBcThreads, per_sm);
  uint64_t bytes = 0;
  for (size_t j0 = 0; j0 < hs.size(); j0 += 64) {
    R.k = (uint32_t)std::min<size_t>(64, hs.size() - j0);
    R.srcs = srcs + j0;
    GRE_CHECK(word.run(R.srcs, R.k, false));
    R.nl = word.levels + 1;
    R.F = (const u64*)g->bc_fpool;
    GRE_CHECK(ws_array(g, WS_BC3, 2 * word.frontier_vertices, &R.shorts));
    GRE_CHECK(ws_array(g, WS_BC4, R.nl + 1, &R.list));
    R.longs = R.shorts + word.frontier_vertices;
    GRE_CUDA(cudaMemsetAsync(R.list, 0, sizeof(BcList) * (R.nl + 1), g->stream));
    for (uint32_t d = 0; d < std::min(R.nl, 2u); ++d) k_bcm_first<<<grid, kBcThreads, 0, g->stream>>>(R, d);
    for (uint32_t d = 1; d < R.nl; ++d) k_bcm_level<true><<<grid, kBcThreads, 0, g->stream>>>(R, d);
    for (uint32_t d = R.nl; d-- > 0;) k_bcm_level<false><<<grid, kBcThreads, 0, g->stream>>>(R, d);
    k_bcm_accumulate<<<grid_for(n, 256), 256, 0, g->stream>>>(n, R.seen, R.F, R.dep, dbc);
    GRE_LAUNCH_CHECK();
    bytes += 2 * R.nl * 8 * n + 2 * (8 * (n + 1) + 12 * g->m) + 2 * 512 * n;
    if (st) {
      st->supersteps += 2 * R.nl;
      st->arcs_traversed += 2 * g->m;
    }
  }
  if (st) {
    st->arcs_traversed += word.scanned;
    st->algo_bytes += bytes + word.bytes;
  }
  return GRE_SUCCESS;
}

}  // namespace gre

using namespace gre;

extern "C" {

int gre_bc(gre_graph g, const uint32_t* srcs, uint32_t nsrc, int batched, double* bc, gre_stats* st) {
  if (!g || !bc || (nsrc && !srcs)) return GRE_NULL;
  GRE_CHECK(use_graph(g));
  stats_reset(st);
  const uint64_t n = g->n;
  std::vector<uint32_t> hs(nsrc);
  if (nsrc) GRE_CUDA(cudaMemcpy(hs.data(), srcs, sizeof(uint32_t) * nsrc, cudaMemcpyDefault));
  GRE_CHECK(map_ids(g, &hs, "gre_bc"));
  GRE_CHECK(ensure_chunk_table(g, g->bc_chunks, kBcChunk));
  double *dfinal, *dbc;
  GRE_CHECK(prepare_output(g, bc, n, WS_OUTBUF, &dfinal));
  GRE_CHECK(perm_out_begin(g, dfinal, 1, 8, (void**)&dbc));
  RunTimer timer(g);
  GRE_CUDA(cudaMemsetAsync(dbc, 0, sizeof(double) * n, g->stream));
  if (batched) GRE_CHECK(bc_batched(g, hs, dbc, st));
  else GRE_CHECK(bc_single(g, hs, dbc, st));
  GRE_CHECK(perm_out_end(g, dbc, dfinal, 1, 8));
  GRE_CHECK(finish_output(g, bc, dfinal, n));
  GRE_CHECK(timer.stop(st));
  if (st) st->traversed_edges = (uint64_t)nsrc * (g->symmetric() ? g->m / 2 : g->m);
  return GRE_SUCCESS;
}

}  // extern "C"
