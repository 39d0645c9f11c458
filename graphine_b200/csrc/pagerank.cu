// PageRank fast paths (FP64, pull over in-arcs):
//   gre_pagerank           one superstep = one degree-binned pull over the CSC
//   gre_ppr                personalised PageRank, looped or batched (128 vectors per pass)
//   gre_pagerank_weighted  weighted forward to a tolerance
//   gre_pagerank_adjoint   implicit adjoint (transposed fixed point) + gradients
//
// The reference superstep (Engine.hpp:592-625 + PageRank.hpp:51-74) pushes pr_scatter[u] along
// every out-arc and adds it into pr_combine[v] under a spin lock, then applies
// pr = 0.15 + 0.85*pr_combine to every vertex that received a message.  The pull form computes
// the same sum per vertex without atomics: pr[v] = tele + d * sum_{u->v} contrib[u], where
// contrib[u] = pr_scatter[u] (0.15/outdeg for the reference variant, pr/outdeg for the power
// iteration).  Vertices without in-arcs receive no message and keep their init value, exactly
// as in the reference (apply is never called for them).
//
// HBM bytes per superstep (algorithmic): 8(n+1) offsets + 4m columns + 8m gathered contrib
// + 4n outdeg + 16n (pr and contrib writes) = 8(n+1) + 12m + 20n.
#include <algorithm>

#include "gre_internal.cuh"
#include "rows.cuh"

namespace gre {

// ---------------------------------------------------------------------------------------------
// plain PageRank
// ---------------------------------------------------------------------------------------------
struct GatherContrib {
  // eight blocks an SM: left alone, plain loads take 40 registers and six blocks (PageRank-20, default schedule: RMAT-18
  // 403 -> 436 us, RMAT-20 1663 -> 1889, RMAT-22 7498 -> 8191, RMAT-24 33.5 -> 35.3 ms; directed RMAT-16 alone 167 -> 146)
  static constexpr int kBlocks = 8;
  const uint32_t* __restrict__ rcol;
  const double* contrib;  // plain loads: the launch before may still write it when this one starts (launch_early)
  __device__ __forceinline__ double operator()(uint32_t, uint64_t a) const { return contrib[__ldg(rcol + a)]; }
  __device__ __forceinline__ void warm(uint64_t a) const { asm volatile("" ::"r"(__ldg(rcol + a))); }
};

struct FinishPR {
  double* __restrict__ pr;
  double* __restrict__ contrib_next;  // null: scatter value never refreshed (reference variant)
  const uint32_t* __restrict__ outdeg;
  double tele, d;
  __device__ __forceinline__ void operator()(uint32_t v, double sum) const {
    const double x = tele + d * sum;
    pr[v] = x;
    if (contrib_next) {
      const uint32_t od = outdeg[v];
      contrib_next[v] = od ? x / (double)od : 0.0;
    }
  }
};

__global__ void k_pr_init(uint64_t n, const uint32_t* __restrict__ outdeg, double tele, double* __restrict__ pr,
                          double* __restrict__ c0, double* __restrict__ c1) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t od = outdeg[v];
    const double c = od ? tele / (double)od : 0.0;
    pr[v] = tele;
    c0[v] = c;
    if (c1) c1[v] = c;
  }
}

static uint64_t pr_bytes_per_iter(uint64_t n, uint64_t m) { return 8 * (n + 1) + 12 * m + 20 * n; }

template <class T>
static int ws_array(gre_graph g, int slot, uint64_t count, T** p) {
  void* v = nullptr;
  GRE_CHECK(g->ws.get(slot, sizeof(T) * (count ? count : 1), &v));
  *p = (T*)v;
  return GRE_SUCCESS;
}

// ---------------------------------------------------------------------------------------------
// personalised PageRank, batched: the vectors in slices of C = 64 (or 32) columns, X[v][C]
// row-major, a warp per in-arc row, each lane C/32 columns; rows longer than kPprChunk arcs are
// split into chunks whose partial vectors are added in order.
//
// A superstep gathers a row of X per arc, 8C bytes, from L2 where it is there.  128 columns a row
// (1 KB) kept an eighth of RMAT-20's rows in L2 and two arcs in flight a warp: 2.85 ms a superstep, DRAM
// at 43%, L2 at 46%, warps waiting for loads (ncu).  64 columns keep a quarter of the rows there (which
// draw nine tenths of the arcs), one 16-byte load a lane and arc, eight arcs in flight; the columns' second
// reading of the topology is 4 bytes an arc: 0.95 ms a slice and superstep, 17 TB/s of gathered rows,
// L2 and L1 at 64% (RMAT-20, 128 vectors, 20 supersteps: 61.2 -> 42.7 ms; slices of 32 columns: 46.2).
//
// The columns are independent: a slice runs all its supersteps before the next, or, where a slice's warps leave
// most of the GPU idle, several do side by side (3000 vertices of 16 arcs, 128 vectors, 20 supersteps: 788 us one after the
// other, 196 side by side).  The values themselves are written by the last superstep only, in place of the
// next contributions.
// ---------------------------------------------------------------------------------------------
constexpr uint64_t kPprChunk = 1024;
constexpr int kPprBatch = 8;           // short rows a warp takes together
constexpr uint32_t kPprShort = 32;     // arcs of a short row at most
// Slices side by side: up to so many warps an SM together (counted with kPprBatch rows each), and two short rows a
// warp, since there are more warps than work.  128 vectors, 20 supersteps, uniform rows of 16 arcs; 128-column rows of one slice /
// slices of 64 in turn / side by side with 8, 4, 2, 1 rows a warp: 300 vertices 225 / 539 / 280, 231, 154, 149 us; 3000 252 / 788 /
// 386, 282, 196, 198; 10000 411 / 802 / 443, 373, 346, 357; 40000 1233 / 1252 / 1066, 1011, 976, 1060.  Skewed rows, 20000 vertices
// 7543 / 2015 / 1176, 1463, 1511, 1525.  At 100000 vertices two slices fill the GPU one by one: 2689 in turn, 2755 side by side.
constexpr uint64_t kPprSideWarps = 128;
constexpr int kPprSideBatch = 2;

template <int C>
struct PprVec;  // a lane's columns of a row: C/32 of them, side by side
template <>
struct PprVec<64> {
  double a = 0.0, b = 0.0;
  static __device__ __forceinline__ PprVec load(const double* row) {
    const double2 x = __ldg((const double2*)row + lane_id());
    PprVec r;
    r.a = x.x;
    r.b = x.y;
    return r;
  }
  __device__ __forceinline__ void add(const PprVec& o) {
    a += o.a;
    b += o.b;
  }
  __device__ __forceinline__ void store(double* row) const { ((double2*)row)[lane_id()] = make_double2(a, b); }
};
template <>
struct PprVec<32> {
  double a = 0.0;
  static __device__ __forceinline__ PprVec load(const double* row) {
    PprVec r;
    r.a = __ldg(row + lane_id());
    return r;
  }
  __device__ __forceinline__ void add(const PprVec& o) { a += o.a; }
  __device__ __forceinline__ void store(double* row) const { row[lane_id()] = a; }
};

struct PprStep {
  const uint64_t* __restrict__ roff;
  const uint32_t* __restrict__ rcol;
  const uint32_t* __restrict__ outdeg;
  const uint32_t* __restrict__ seeds;  // kk of them
  const double* __restrict__ cur;      // contributions
  double* __restrict__ next;           // the next ones; the values themselves in the last superstep
  double* __restrict__ partial;        // chunk sums
  const uint32_t* __restrict__ rows;   // the bins' rows, short bins first
  uint32_t nrows, nshort;              // of which the first nshort have at most kPprShort arcs
  ChunkTable chunks;
  uint32_t kk;                         // columns of all slices side by side
  uint64_t n;
  bool last;
  double tele, d;
  // slice `i` of those side by side, each with buffers of its own
  template <int C>
  __device__ __forceinline__ PprStep slice(uint32_t i) const {
    PprStep r = *this;
    r.seeds += i * C;
    r.kk = kk - i * C < C ? kk - i * C : C;
    r.cur += i * n * C;
    r.next += i * n * C;
    r.partial += i * (chunks.nchunks + 1) * C;
    return r;
  }
};

// The place of the restart mass in a row: bit j of a lane's mask, its column j seeds vertex v.
template <int C>
__device__ __forceinline__ void ppr_finish(const PprStep& P, uint32_t v, uint32_t od, PprVec<C> acc, uint32_t seed0, uint32_t seed1) {
  acc.a = (seed0 == v ? P.tele : 0.0) + P.d * acc.a;
  if constexpr (C == 64) acc.b = (seed1 == v ? P.tele : 0.0) + P.d * acc.b;
  if (!P.last) {
    acc.a = od ? acc.a / (double)od : 0.0;
    if constexpr (C == 64) acc.b = od ? acc.b / (double)od : 0.0;
  }
  acc.store(P.next + (uint64_t)v * C);
}

// acc += the rows of the columns that lanes 0 .. cnt-1 hold, in order; eight in flight
template <int C>
__device__ __forceinline__ void ppr_gather(const double* __restrict__ cur, uint32_t idx, uint32_t cnt, PprVec<C>& acc) {
  uint32_t i = 0;
  for (; i + 8 <= cnt; i += 8) {
    PprVec<C> x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = PprVec<C>::load(cur + (uint64_t)__shfl_sync(0xffffffffu, idx, i + j) * C);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc.add(x[j]);
  }
  if (i + 4 <= cnt) {
    PprVec<C> x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = PprVec<C>::load(cur + (uint64_t)__shfl_sync(0xffffffffu, idx, i + j) * C);
#pragma unroll
    for (int j = 0; j < 4; ++j) acc.add(x[j]);
    i += 4;
  }
  if (i + 2 <= cnt) {
    const PprVec<C> x = PprVec<C>::load(cur + (uint64_t)__shfl_sync(0xffffffffu, idx, i) * C);
    const PprVec<C> y = PprVec<C>::load(cur + (uint64_t)__shfl_sync(0xffffffffu, idx, i + 1) * C);
    acc.add(x);
    acc.add(y);
    i += 2;
  }
  if (i < cnt) acc.add(PprVec<C>::load(cur + (uint64_t)__shfl_sync(0xffffffffu, idx, i) * C));
}

template <int C>
__device__ __forceinline__ PprVec<C> ppr_sum(const PprStep& P, uint64_t a0, uint64_t a1) {
  const uint32_t lane = lane_id();
  PprVec<C> acc;
  uint32_t idx = a0 + lane < a1 ? __ldg(P.rcol + a0 + lane) : 0u;
  for (uint64_t b = a0; b < a1; b += 32) {
    const uint32_t following = b + 32 + lane < a1 ? __ldg(P.rcol + b + 32 + lane) : 0u;
    ppr_gather(P.cur, idx, a1 - b < 32 ? (uint32_t)(a1 - b) : 32u, acc);
    idx = following;
  }
  return acc;
}

// One superstep but for the chunked rows' finish: first the chunks, then the rows from long to short
// (the resident warps stride over them, each a share of every length).
// SIDE: slice blockIdx.y of several.
template <int C, bool SIDE>
__global__ void __launch_bounds__(256) k_ppr_step(const __grid_constant__ PprStep all) {
  const PprStep P = SIDE ? all.slice<C>(blockIdx.y) : all;
  const uint32_t lane = lane_id();
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  constexpr int V = C / 32, B = SIDE ? kPprSideBatch : kPprBatch;
  const uint32_t seed0 = V * lane < P.kk ? P.seeds[V * lane] : 0xffffffffu;
  const uint32_t seed1 = V == 2 && V * lane + 1 < P.kk ? P.seeds[V * lane + 1] : 0xffffffffu;
  uint64_t i = warp;
  for (; i < P.chunks.nchunks; i += nwarps) {
    const uint64_t a0 = P.chunks.chunk_begin[i], end = P.roff[P.chunks.rows[P.chunks.chunk_row[i]] + 1];
    ppr_sum<C>(P, a0, a0 + kPprChunk < end ? a0 + kPprChunk : end).store(P.partial + i * C);
  }
  i -= P.chunks.nchunks;
  const uint64_t nlong = P.nrows - P.nshort;
  for (; i < nlong; i += nwarps) {
    const uint32_t v = P.rows[P.nrows - 1 - i];
    const uint64_t a0 = P.roff[v], a1 = P.roff[v + 1];
    const uint32_t od = P.outdeg[v];
    if (a1 - a0 > kPprChunk) continue;  // chunked
    ppr_finish<C>(P, v, od, ppr_sum<C>(P, a0, a1), seed0, seed1);
  }
  i -= nlong;
  const uint64_t nbatches = ((uint64_t)P.nshort + B - 1) / B;
  for (; i < nbatches; i += nwarps) {
    // lane j < B: row j of the batch; then the columns of all of them
    uint64_t a0 = 0;
    uint32_t v = 0, len = 0, od = 0;
    const uint64_t at = i * B + lane;
    if (lane < B && at < P.nshort) {
      v = P.rows[P.nshort - 1 - at];
      a0 = P.roff[v];
      len = (uint32_t)(P.roff[v + 1] - a0);
      od = P.outdeg[v];
    }
    uint32_t idx[B];
#pragma unroll
    for (int j = 0; j < B; ++j) {
      const uint64_t b = __shfl_sync(0xffffffffu, a0, j);
      idx[j] = lane < __shfl_sync(0xffffffffu, len, j) ? __ldg(P.rcol + b + lane) : 0u;
    }
#pragma unroll
    for (int j = 0; j < B; ++j) {
      const uint32_t n = __shfl_sync(0xffffffffu, len, j);
      PprVec<C> acc;
      ppr_gather(P.cur, idx[j], n, acc);
      if (n) ppr_finish<C>(P, __shfl_sync(0xffffffffu, v, j), __shfl_sync(0xffffffffu, od, j), acc, seed0, seed1);
    }
  }
}

// Chunked rows: partial sums in chunk order, four loads in flight.
template <int C, bool SIDE>
__global__ void __launch_bounds__(256) k_ppr_chunk_finish(const __grid_constant__ PprStep all) {
  const PprStep P = SIDE ? all.slice<C>(blockIdx.y) : all;
  const uint32_t lane = lane_id();
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  constexpr int V = C / 32;
  const uint32_t seed0 = V * lane < P.kk ? P.seeds[V * lane] : 0xffffffffu;
  const uint32_t seed1 = V == 2 && V * lane + 1 < P.kk ? P.seeds[V * lane + 1] : 0xffffffffu;
  for (uint64_t i = warp; i < P.chunks.nrows; i += nwarps) {
    const uint32_t v = P.chunks.rows[i];
    const uint32_t od = P.outdeg[v];
    PprVec<C> acc;
    uint64_t c = P.chunks.first[i];
    const uint64_t end = P.chunks.first[i + 1];
    for (; c + 4 <= end; c += 4) {
      PprVec<C> x[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = PprVec<C>::load(P.partial + (c + j) * C);
#pragma unroll
      for (int j = 0; j < 4; ++j) acc.add(x[j]);
    }
    for (; c < end; ++c) acc.add(PprVec<C>::load(P.partial + c * C));
    ppr_finish<C>(P, v, od, acc, seed0, seed1);
  }
}

// The restart mass in both buffers of contributions (zeroed before).
template <int C>
__global__ void k_ppr_seed(uint64_t n, uint32_t kk, const uint32_t* __restrict__ seeds, const uint32_t* __restrict__ outdeg, double tele,
                           double* __restrict__ c0, double* __restrict__ c1) {
  for (uint32_t j = threadIdx.x; j < kk; j += blockDim.x) {
    const uint32_t s = seeds[j];
    const uint32_t od = outdeg[s];
    const double c = od ? tele / (double)od : 0.0;
    const uint64_t at = (j / C * n + s) * C + j % C;
    c0[at] = c;
    c1[at] = c;
  }
}

// A seed whose row has no in-arcs (or all seeds, before any superstep) keeps its restart mass as its
// value: no superstep wrote it.
template <int C>
__global__ void k_ppr_seed_values(uint64_t n, uint32_t kk, const uint32_t* __restrict__ seeds, const uint64_t* __restrict__ roff, bool all,
                                  double tele, double* __restrict__ x) {
  for (uint32_t j = threadIdx.x; j < kk; j += blockDim.x) {
    const uint32_t s = seeds[j];
    if (all || roff[s + 1] == roff[s]) x[(j / C * n + s) * C + j % C] = tele;
  }
}

// out[j * n + u] = x[row of u][j] for the slice's kk vectors, u in the caller's order: 32 rows at a
// time through shared memory, so that both sides move whole lines.
template <int C>
__global__ void __launch_bounds__(256) k_ppr_out(uint64_t n, uint32_t kk, const double* __restrict__ x,
                                                 const uint32_t* __restrict__ iperm, double* __restrict__ out) {
  __shared__ double tile[32][C + 1];
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  x += blockIdx.y * n * C;  // slice blockIdx.y of those side by side
  out += blockIdx.y * n * C;
  kk = kk - blockIdx.y * C < C ? kk - blockIdx.y * C : C;
  for (uint64_t u0 = blockIdx.x * 32ull; u0 < n; u0 += gridDim.x * 32ull) {
    for (uint32_t r = w; r < 32; r += 8) {
      if (u0 + r >= n) break;
      const uint64_t v = iperm ? __ldg(iperm + u0 + r) : u0 + r;
#pragma unroll
      for (int j = 0; j < C / 32; ++j) tile[r][lane + 32 * j] = __ldg(x + v * C + lane + 32 * j);
    }
    __syncthreads();
    if (u0 + lane < n)
      for (uint32_t j = w; j < kk; j += 8) out[(uint64_t)j * n + u0 + lane] = tile[lane][j];
    __syncthreads();
  }
}

// Chunks, long rows and batches of short ones.
static uint64_t ppr_warps(const PprStep& P, uint32_t batch) {
  return P.chunks.nchunks + (P.nrows - P.nshort) + (P.nshort + batch - 1) / batch;
}

// One slice, or several side by side (SIDE): P.kk <= slices * C seeds (device), the results to out (kk rows of n in the
// caller's order).
template <int C, bool SIDE>
static int ppr_slices(gre_graph g, PprStep P, uint32_t slices, uint32_t iters, double* c0, double* c1, double* out) {
  const uint64_t n = g->n, warps = ppr_warps(P, SIDE ? kPprSideBatch : kPprBatch);
  static int per_sm = 0;
  if (!per_sm) {
    int b = 0;
    GRE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_ppr_step<C, SIDE>, 256, 0));
    per_sm = b > 0 ? b : 1;
  }
  auto side = [&](int blocks) { return dim3(blocks, slices); };
  GRE_CUDA(cudaMemsetAsync(c0, 0, sizeof(double) * n * C * slices, g->stream));
  GRE_CUDA(cudaMemsetAsync(c1, 0, sizeof(double) * n * C * slices, g->stream));
  k_ppr_seed<C><<<1, C, 0, g->stream>>>(n, P.kk, P.seeds, g->outdeg, P.tele, c0, c1);
  for (uint32_t it = 0; it < iters; ++it) {
    P.cur = c0;
    P.next = c1;
    P.last = it + 1 == iters;
    k_ppr_step<C, SIDE><<<side(grid_for(warps * 32, 256, per_sm)), 256, 0, g->stream>>>(P);
    if (P.chunks.nrows) k_ppr_chunk_finish<C, SIDE><<<side(grid_for(P.chunks.nrows * 32, 256, 8)), 256, 0, g->stream>>>(P);
    std::swap(c0, c1);
  }
  k_ppr_seed_values<C><<<1, C, 0, g->stream>>>(n, P.kk, P.seeds, g->roff, iters == 0, P.tele, c0);
  k_ppr_out<C><<<side(grid_for(n * 8, 256, 16)), 256, 0, g->stream>>>(n, P.kk, c0, g->iperm, out);
  GRE_LAUNCH_CHECK();
  return GRE_SUCCESS;
}

// ---------------------------------------------------------------------------------------------
// single-vector personalised PageRank (looped form): PageRank pull with a one-hot teleport
// ---------------------------------------------------------------------------------------------
struct FinishPPR1 {
  double* __restrict__ x;
  double* __restrict__ cnext;
  const uint32_t* __restrict__ outdeg;
  uint32_t seed;
  double tele, d;
  __device__ __forceinline__ void operator()(uint32_t v, double sum) const {
    const double val = (v == seed ? tele : 0.0) + d * sum;
    x[v] = val;
    const uint32_t od = outdeg[v];
    cnext[v] = od ? val / (double)od : 0.0;
  }
};

__global__ void k_ppr1_init(uint64_t n, uint32_t seed, const uint32_t* __restrict__ outdeg, double tele, double* __restrict__ x,
                            double* __restrict__ c0, double* __restrict__ c1) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const double t = (v == seed) ? tele : 0.0;
    const uint32_t od = outdeg[v];
    const double c = od ? t / (double)od : 0.0;
    x[v] = t;
    c0[v] = c;
    c1[v] = c;
  }
}

// ---------------------------------------------------------------------------------------------
// weighted PageRank and its adjoint
// ---------------------------------------------------------------------------------------------
struct GatherWeighted {  // sum_a p[a] * x[col[a]]
  static constexpr bool kDeep = true;
  const uint32_t* __restrict__ col;
  const double* __restrict__ p;
  const double* x;  // the launch before may still write it (launch_early)
  __device__ __forceinline__ double operator()(uint32_t, uint64_t a) const { return __ldg(p + a) * x[__ldg(col + a)]; }
  __device__ __forceinline__ void warm(uint64_t a) const { asm volatile("" ::"r"(__ldg(col + a))); }
};
struct GatherW {  // sum_a w[a]
  const double* __restrict__ w;
  __device__ __forceinline__ double operator()(uint32_t, uint64_t a) const { return __ldg(w + a); }
};
struct FinishStore {
  double* __restrict__ out;
  __device__ __forceinline__ void operator()(uint32_t v, double s) const { out[v] = s; }
};

// y[v] = base[v] + d*sum (base = (1-d)*pers for the forward, c for the adjoint); tracks max|dy|.
// The largest change is kept per thread (non-negative doubles order like their bit patterns, a NaN
// above all) and joins the global one once a block: one atomic a row serialised on that address
// and bounded the superstep (RMAT-20, 1M rows: 0.90 -> 0.41 ms an iteration).
struct FinishAffine {
  double* __restrict__ y;
  const double* xprev;               // this and `before`: the launch before may still write them
  const double* __restrict__ base;  // null: constant base_c
  double base_c, scale, d;
  double* __restrict__ maxdiff;
  const double* before;  // null, or the largest change at the last check: nothing is left to do
  double tol;
  unsigned long long largest = 0;
  __device__ __forceinline__ bool stopped() const { return before && *before <= tol; }
  __device__ __forceinline__ void operator()(uint32_t v, double sum) {
    const double b = base ? scale * base[v] : base_c;
    const double val = b + d * sum;
    y[v] = val;
    const unsigned long long diff = (unsigned long long)__double_as_longlong(fabs(val - xprev[v]));
    largest = diff > largest ? diff : largest;
  }
  __device__ __forceinline__ void end() {
    __shared__ unsigned long long s_largest;
    if (threadIdx.x == 0) s_largest = 0;
    __syncthreads();
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long x = __shfl_xor_sync(0xffffffffu, largest, o);
      largest = x > largest ? x : largest;
    }
    if ((threadIdx.x & 31u) == 0 && largest) atomicMax(&s_largest, largest);
    __syncthreads();
    if (threadIdx.x == 0 && s_largest > __ldcg((const unsigned long long*)maxdiff))
      atomicMax((unsigned long long*)maxdiff, s_largest);
  }
};

__global__ void k_affine_init(uint64_t n, const double* __restrict__ base, double base_c, double scale, double* __restrict__ a,
                              double* __restrict__ b) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
    const double x = base ? scale * base[v] : base_c;
    a[v] = x;
    b[v] = x;
  }
}

// Visits of every arc through the row schedule: a warp a row left a hub to one warp (RMAT-20: 1050 us to
// normalise, 1320 for the weight gradient).
struct VisitNormalise {  // p[a] = w[a] / s[row]
  const double* __restrict__ w;
  const double* s;  // the launch before may still write it
  double* __restrict__ p;
  __device__ __forceinline__ double operator()(uint32_t u, uint64_t a) const {
    p[a] = __ldg(w + a) / s[u];
    return 0.0;
  }
};
struct VisitGradW {  // gw[a] = d * r[u] / s[u] * (lambda[col[a]] - pl[u]), f[u] = d * r[u] / s[u]
  const uint32_t* __restrict__ col;
  const double* f;  // the launch before writes it; lambda and pl were complete when that one started
  const double* __restrict__ lambda;
  const double* __restrict__ pl;
  double* __restrict__ gw;
  __device__ __forceinline__ double operator()(uint32_t u, uint64_t a) const {
    gw[a] = f[u] * (__ldg(lambda + __ldg(col + a)) - __ldg(pl + u));
    return 0.0;
  }
};
struct VisitEnd {
  __device__ __forceinline__ void operator()(uint32_t, double) const {}
};

__global__ void k_grad_factor(uint64_t n, const double* __restrict__ r, const double* __restrict__ s, double d, double* __restrict__ f) {
  for (uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; u < n; u += (uint64_t)gridDim.x * blockDim.x) f[u] = d * r[u] / s[u];
}

// pw[slot] = rw[slot] / s[rcol[slot]] over the CSC
__global__ void k_csc_normalise(uint64_t m, const uint32_t* __restrict__ rcol, const double* __restrict__ rw,
                                const double* __restrict__ s, double* __restrict__ pw) {
  for (uint64_t a = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; a < m; a += (uint64_t)gridDim.x * blockDim.x)
    pw[a] = rw[a] / s[rcol[a]];
}

__global__ void k_scale(uint64_t n, const double* __restrict__ x, double f, double* __restrict__ y) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) y[v] = f * x[v];
}

// Row sums s of the FP64 weights and the normalised ones (in workspace): by CSC slot (pw) for the
// forward solve, by CSR arc (p) for the adjoint.
struct WeightedPrep {
  double* s;
  double* p;
  double* pw;
};
static int weighted_prep(gre_graph g, bool adjoint, WeightedPrep* wp) {
  if (!g->w64 || !g->rw64) {
    set_error("weighted PageRank needs FP64 arc weights (gre_graph_set_weights_f64)");
    return GRE_INVALID_ARG;
  }
  GRE_CHECK(ensure_bins(g, false));
  GRE_CHECK(ws_array(g, WS_I, g->n, &wp->s));
  double* partial;
  GRE_CHECK(ws_array(g, WS_H, g->bins_out.n_partials + 1, &partial));
  GRE_CUDA(cudaMemsetAsync(wp->s, 0, sizeof(double) * g->n, g->stream));
  GRE_CHECK(rows::reduce_rows(g->bins_out, g->off, GatherW{g->w64}, FinishStore{wp->s}, partial, g->stream));
  if (adjoint) {
    GRE_CHECK(ws_array(g, WS_J, g->m, &wp->p));
    GRE_CHECK(rows::reduce_rows(g->bins_out, g->off, VisitNormalise{g->w64, wp->s, wp->p}, VisitEnd{}, partial, g->stream));
  } else {
    GRE_CHECK(ws_array(g, WS_K, g->m, &wp->pw));
    k_csc_normalise<<<grid_for(g->m, 256), 256, 0, g->stream>>>(g->m, g->rcol, g->rw64, wp->s, wp->pw);
  }
  GRE_LAUNCH_CHECK();
  return GRE_SUCCESS;
}

// Jacobi iteration y = base + d * (A x) with A given by (bins, off, col, p), to tolerance.
//
// The largest change is looked at after every fourth iteration.  The host launches kAhead iterations
// and then reads their changes; a kernel whose last looked-at change was small enough returns at
// once, so the result is that of the first such look whatever was launched behind it (a host read every
// four iterations cost 5 us an iteration, RMAT-20: 113).
static int affine_solve(gre_graph g, const DegreeBins& B, const uint64_t* off, const uint32_t* col, const double* p,
                        const double* base, double scale, double base_c, double d, double tol, uint32_t max_iters,
                        double* xa, double* xb, double** result, uint32_t* iters_done, gre_stats* st) {
  constexpr uint32_t kCheck = 4, kAhead = 32;  // even: the buffers are back in place
  double* partial;
  double* maxdiff;  // of the iterations launched together
  GRE_CHECK(ws_array(g, WS_H, B.n_partials + 1, &partial));
  GRE_CHECK(ws_array(g, WS_COUNTERS, kAhead, &maxdiff));
  k_affine_init<<<grid_for(g->n, 256), 256, 0, g->stream>>>(g->n, base, base_c, scale, xa, xb);
  GRE_LAUNCH_CHECK();
  double *x = xa, *y = xb;
  uint32_t it = 0;
  for (bool small = false; !small && it < max_iters;) {
    const uint32_t k = std::min(kAhead, max_iters - it);
    GRE_CUDA(cudaMemsetAsync(maxdiff, 0, sizeof(double) * k, g->stream));
    double *from = x, *to = y;
    for (uint32_t i = 0; i < k; ++i) {
      // rows without arcs keep base (set by init in both buffers)
      const double* before = i >= kCheck ? maxdiff + i / kCheck * kCheck - 1 : nullptr;
      GRE_CHECK(rows::reduce_rows(B, off, GatherWeighted{col, p, from},
                                  FinishAffine{to, from, base, base_c, scale, d, maxdiff + i, before, tol}, partial, g->stream));
      std::swap(from, to);
    }
    double h[kAhead];
    GRE_CUDA(cudaMemcpyAsync(h, maxdiff, sizeof(double) * k, cudaMemcpyDeviceToHost, g->stream));
    GRE_CUDA(cudaStreamSynchronize(g->stream));
    uint32_t ran = k;
    for (uint32_t i = kCheck; i <= k && !small; i += kCheck)
      if (h[i - 1] <= tol) {
        small = true;
        ran = i;
      }
    it += ran;
    if (ran & 1) std::swap(x, y);
  }
  *result = x;
  *iters_done = it;
  return GRE_SUCCESS;
}

}  // namespace gre

using namespace gre;

extern "C" {

int gre_pagerank(gre_graph g, int variant, double d, uint32_t iters, double* pr, gre_stats* st) {
  if (!g || !pr) return GRE_NULL;
  if ((variant != GRE_PR_REFERENCE && variant != GRE_PR_ITER) || !(d >= 0.0 && d < 1.0)) return GRE_INVALID_ARG;
  GRE_CHECK(use_graph(g));
  stats_reset(st);
  GRE_CHECK(ensure_bins(g, true));
  const uint64_t n = g->n;
  double *dout, *dpr, *c0, *c1, *partial;
  GRE_CHECK(prepare_output(g, pr, n, WS_OUTBUF, &dout));
  GRE_CHECK(perm_out_begin(g, dout, 1, 8, (void**)&dpr));
  GRE_CHECK(ws_array(g, WS_A, n, &c0));
  GRE_CHECK(ws_array(g, WS_B, n, &c1));
  GRE_CHECK(ws_array(g, WS_C, g->bins_in.n_partials + 1, &partial));
  const double tele = 1.0 - d;
  const bool refresh = variant == GRE_PR_ITER;
  RunTimer timer(g);
  k_pr_init<<<grid_for(n, 256), 256, 0, g->stream>>>(n, g->outdeg, tele, dpr, c0, refresh ? c1 : nullptr);
  GRE_LAUNCH_CHECK();
  // one superstep reads contributions `a` and (power iteration) writes the next ones to `b`
  auto superstep = [&](double* a, double* b) -> int {
    FinishPR fin{dpr, refresh ? b : nullptr, g->outdeg, tele, d};
    return rows::reduce_rows(g->bins_in, g->roff, GatherContrib{g->rcol, a}, fin, partial, g->stream);
  };
  // one or two launches a superstep: launched as they come (recording and instantiating a CUDA
  // graph each call cost more than the launches it saved)
  for (uint32_t done = 0; done < iters; ++done) {
    GRE_CHECK(superstep(c0, c1));
    if (refresh) std::swap(c0, c1);
  }
  GRE_CHECK(perm_out_end(g, dpr, dout, 1, 8));
  GRE_CHECK(finish_output(g, pr, dout, n));
  GRE_CHECK(timer.stop(st));
  if (st) {
    st->supersteps = iters;
    for (uint32_t i = 0; i < iters; ++i) stats_record(st, rows::nonempty_rows(g->bins_in));
    st->arcs_traversed = g->m * (uint64_t)iters;
    st->traversed_edges = g->m * (uint64_t)iters;
    st->algo_bytes = pr_bytes_per_iter(n, g->m) * iters;
  }
  return GRE_SUCCESS;
}

int gre_ppr(gre_graph g, const uint32_t* seeds, uint32_t k, double d, uint32_t iters, int batched, double* out, gre_stats* st) {
  if (!g || !out || (k && !seeds)) return GRE_NULL;
  if (!(d >= 0.0 && d < 1.0)) return GRE_INVALID_ARG;
  GRE_CHECK(use_graph(g));
  stats_reset(st);
  if (k == 0) return GRE_SUCCESS;
  const uint64_t n = g->n;
  std::vector<uint32_t> hs(k);
  GRE_CUDA(cudaMemcpy(hs.data(), seeds, sizeof(uint32_t) * k, cudaMemcpyDefault));
  GRE_CHECK(map_ids(g, &hs, "gre_ppr"));
  GRE_CHECK(ensure_bins(g, true));
  const double tele = 1.0 - d;
  double* dfinal;
  GRE_CHECK(prepare_output(g, out, (uint64_t)k * n, WS_OUTBUF, &dfinal));
  RunTimer timer(g);
  if (!batched) {
    double *dout, *c0, *c1, *partial;
    GRE_CHECK(perm_out_begin(g, dfinal, k, 8, (void**)&dout));
    GRE_CHECK(ws_array(g, WS_A, n, &c0));
    GRE_CHECK(ws_array(g, WS_B, n, &c1));
    GRE_CHECK(ws_array(g, WS_C, g->bins_in.n_partials + 1, &partial));
    for (uint32_t j = 0; j < k; ++j) {
      double* x = dout + (uint64_t)j * n;
      k_ppr1_init<<<grid_for(n, 256), 256, 0, g->stream>>>(n, hs[j], g->outdeg, tele, x, c0, c1);
      double* cur = c0;
      double* nxt = c1;
      for (uint32_t it = 0; it < iters; ++it) {
        GRE_CHECK(rows::reduce_rows(g->bins_in, g->roff, GatherContrib{g->rcol, cur}, FinishPPR1{x, nxt, g->outdeg, hs[j], tele, d},
                                    partial, g->stream));
        std::swap(cur, nxt);
      }
    }
    GRE_CHECK(perm_out_end(g, dout, dfinal, k, 8));
    if (st) st->algo_bytes = (uint64_t)k * iters * pr_bytes_per_iter(n, g->m);
  } else {
    GRE_CHECK(ensure_chunk_table(g, g->ppr_chunks, kPprChunk));
    double *c0, *c1, *partial;
    uint32_t* dseeds;
    PprStep P{};
    const DegreeBins& B = g->bins_in;
    P.n = n;
    P.roff = g->roff;
    P.rcol = g->rcol;
    P.outdeg = g->outdeg;
    P.rows = B.rows;
    P.chunks = g->ppr_chunks;
    P.tele = tele;
    P.d = d;
    for (int b = 0; b < DegreeBins::NB; ++b) {
      P.nrows += (uint32_t)B.count[b];
      if (b < 5 && ((uint64_t)B.sched.lane_arcs << b) <= kPprShort) P.nshort += (uint32_t)B.count[b];
    }
    const uint64_t fit = kPprSideWarps * (uint64_t)num_sms() / std::max<uint64_t>(1, ppr_warps(P, kPprBatch));
    const uint32_t slices = k <= 64 ? 1 : (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(fit, (k + 63) / 64));
    const uint64_t cols = k > 32 ? 64ull * slices : 32;
    GRE_CHECK(ws_array(g, WS_A, n * cols, &c0));
    GRE_CHECK(ws_array(g, WS_B, n * cols, &c1));
    GRE_CHECK(ws_array(g, WS_D, (g->ppr_chunks.nchunks + 1) * cols, &partial));
    GRE_CHECK(ws_array(g, WS_E, k, &dseeds));
    GRE_CUDA(cudaMemcpyAsync(dseeds, hs.data(), sizeof(uint32_t) * k, cudaMemcpyHostToDevice, g->stream));
    P.partial = partial;
    for (uint32_t j0 = 0; j0 < k;) {
      // 64 columns a slice; a rest of at most 32 in a slice of 32
      const uint32_t left = k - j0;
      P.seeds = dseeds + j0;
      double* o = dfinal + (uint64_t)j0 * n;
      if (slices > 1 && left > 64) {
        P.kk = std::min<uint32_t>(64 * slices, left);
        GRE_CHECK((ppr_slices<64, true>(g, P, (P.kk + 63) / 64, iters, c0, c1, o)));
      } else if (left > 32) {
        P.kk = std::min<uint32_t>(64, left);
        GRE_CHECK((ppr_slices<64, false>(g, P, 1, iters, c0, c1, o)));
      } else {
        P.kk = left;
        GRE_CHECK((ppr_slices<32, false>(g, P, 1, iters, c0, c1, o)));
      }
      j0 += P.kk;
    }
    if (st) {
      const uint64_t passes = (k + 63) / 64;
      st->algo_bytes = iters * (passes * (8 * (n + 1) + 4 * g->m) + (uint64_t)k * (8 * g->m + 16 * n));
    }
  }
  GRE_CHECK(finish_output(g, out, dfinal, (uint64_t)k * n));
  GRE_CHECK(timer.stop(st));
  if (st) {
    st->supersteps = iters;
    st->arcs_traversed = g->m * (uint64_t)iters * k;
    st->traversed_edges = st->arcs_traversed;
  }
  return GRE_SUCCESS;
}

int gre_pagerank_weighted(gre_graph g, double d, const double* pers, double tol, uint32_t max_iters, double* r, gre_stats* st) {
  if (!g || !r) return GRE_NULL;
  if (!(d >= 0.0 && d < 1.0) || !(tol >= 0.0)) return GRE_INVALID_ARG;
  GRE_CHECK(use_graph(g));
  stats_reset(st);
  const uint64_t n = g->n;
  GRE_CHECK(ensure_bins(g, true));
  WeightedPrep wp{};
  GRE_CHECK(weighted_prep(g, false, &wp));
  const double* dpers;
  double *dr, *xa, *xb, *res;
  GRE_CHECK(stage_input(g, pers, n, WS_G, &dpers));
  GRE_CHECK(perm_in(g, dpers, 8, WS_PERM_IN, (const void**)&dpers));
  GRE_CHECK(prepare_output(g, r, n, WS_OUTBUF, &dr));
  GRE_CHECK(ws_array(g, WS_A, n, &xa));
  GRE_CHECK(ws_array(g, WS_B, n, &xb));
  RunTimer timer(g);
  uint32_t done = 0;
  GRE_CHECK(affine_solve(g, g->bins_in, g->roff, g->rcol, wp.pw, dpers, 1.0 - d, 1.0 - d, d, tol, max_iters, xa, xb, &res, &done, st));
  if (g->perm) GRE_CHECK(perm_out_end(g, res, dr, 1, 8));
  else GRE_CUDA(cudaMemcpyAsync(dr, res, sizeof(double) * n, cudaMemcpyDeviceToDevice, g->stream));
  GRE_CHECK(finish_output(g, r, dr, n));
  GRE_CHECK(timer.stop(st));
  if (st) {
    st->supersteps = done;
    st->arcs_traversed = g->m * (uint64_t)done;
    st->traversed_edges = st->arcs_traversed;
    st->algo_bytes = (uint64_t)done * (8 * (n + 1) + 20 * g->m + 16 * n);
  }
  return done < max_iters || max_iters == 0 ? GRE_SUCCESS : GRE_UNFINISHED;
}

int gre_pagerank_adjoint(gre_graph g, double d, const double* r, const double* c, double tol, uint32_t max_iters, double* lambda,
                         double* grad_pers, double* grad_w, gre_stats* st) {
  if (!g || !r || !c || !grad_w) return GRE_NULL;
  if (!(d > 0.0 && d < 1.0) || !(tol >= 0.0)) return GRE_INVALID_ARG;
  GRE_CHECK(use_graph(g));
  stats_reset(st);
  const uint64_t n = g->n, m = g->m;
  GRE_CHECK(ensure_bins(g, true));
  WeightedPrep wp{};
  GRE_CHECK(weighted_prep(g, true, &wp));
  const double *dr, *dc;
  double *xa, *xb, *res, *pl, *dgw, *dlam = nullptr, *dgp = nullptr;
  GRE_CHECK(stage_input(g, r, n, WS_F, &dr));
  GRE_CHECK(stage_input(g, c, n, WS_G, &dc));
  GRE_CHECK(perm_in(g, dr, 8, WS_PERM_IN, (const void**)&dr));
  GRE_CHECK(perm_in(g, dc, 8, WS_PERM_IN2, (const void**)&dc));
  GRE_CHECK(ws_array(g, WS_A, n, &xa));
  GRE_CHECK(ws_array(g, WS_B, n, &xb));
  GRE_CHECK(ws_array(g, WS_C, n, &pl));
  double* dgw_final;
  GRE_CHECK(prepare_output(g, grad_w, m, WS_OUTBUF, &dgw_final));
  dgw = dgw_final;
  if (g->perm) GRE_CHECK(ws_array(g, WS_PERM_OUT, m, &dgw));  // internal arc order first
  if (lambda) GRE_CHECK(prepare_output(g, lambda, n, WS_D, &dlam));
  if (grad_pers) GRE_CHECK(prepare_output(g, grad_pers, n, WS_E, &dgp));
  RunTimer timer(g);
  uint32_t done = 0;
  // lambda = c + d P lambda: pull over the CSR rows (out-arcs) with p = W/s
  GRE_CHECK(affine_solve(g, g->bins_out, g->off, g->col, wp.p, dc, 1.0, 0.0, d, tol, max_iters, xa, xb, &res, &done, st));
  // pl[u] = sum_k P_uk lambda_k (rows without arcs keep 0)
  double* partial;
  GRE_CHECK(ws_array(g, WS_H, g->bins_out.n_partials + 1, &partial));
  GRE_CUDA(cudaMemsetAsync(pl, 0, sizeof(double) * n, g->stream));
  GRE_CHECK(rows::reduce_rows(g->bins_out, g->off, GatherWeighted{g->col, wp.p, res}, FinishStore{pl}, partial, g->stream));
  double* f = res == xa ? xb : xa;
  k_grad_factor<<<grid_for(n, 256), 256, 0, g->stream>>>(n, dr, wp.s, d, f);
  GRE_CHECK(rows::reduce_rows(g->bins_out, g->off, VisitGradW{g->col, f, res, pl, dgw}, VisitEnd{}, partial, g->stream));
  GRE_LAUNCH_CHECK();
  if (g->perm) GRE_CHECK(arcs_to_caller(g, dgw, dgw_final, 8));
  dgw = dgw_final;
  if (dgp) {
    // (1-d) lambda into pl (free now), then to caller order
    k_scale<<<grid_for(n, 256), 256, 0, g->stream>>>(n, res, 1.0 - d, g->perm ? pl : dgp);
    if (g->perm) GRE_CHECK(perm_out_end(g, pl, dgp, 1, 8));
  }
  if (dlam) {
    if (g->perm) GRE_CHECK(perm_out_end(g, res, dlam, 1, 8));
    else GRE_CUDA(cudaMemcpyAsync(dlam, res, sizeof(double) * n, cudaMemcpyDeviceToDevice, g->stream));
  }
  GRE_LAUNCH_CHECK();
  GRE_CHECK(finish_output(g, grad_w, dgw, m));
  if (lambda) GRE_CHECK(finish_output(g, lambda, dlam, n));
  if (grad_pers) GRE_CHECK(finish_output(g, grad_pers, dgp, n));
  GRE_CHECK(timer.stop(st));
  if (st) {
    st->supersteps = done;
    st->arcs_traversed = m * (uint64_t)(done + 2);
    st->traversed_edges = st->arcs_traversed;
    st->algo_bytes = (uint64_t)(done + 1) * (8 * (n + 1) + 20 * m + 16 * n) + (8 * (n + 1) + 4 * m + 8 * m + 8 * m + 24 * n);
  }
  return done < max_iters || max_iters == 0 ? GRE_SUCCESS : GRE_UNFINISHED;
}

}  // extern "C"
