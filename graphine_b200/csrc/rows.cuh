// Degree-binned row reductions over a CSR or CSC: the pull form of the superstep's
// scatter+combine for sums (PageRank, weighted PageRank, its adjoint).
//
// Rows are grouped once per graph by degree (DegreeBins, schedule chosen in bins.cu): bins 0..5
// give a row 1, 2, 4, 8, 16 or 32 lanes (4 arcs per lane and a warp up to 4096 arcs: degree 1-4,
// 5-8, 9-16, 17-32, 33-64, 65-4096); bin 6 gives a row one CTA (4097-65536 there); bin 7 splits a
// row into chunks of hub_chunk arcs (65536), one CTA each, whose partial sums are added in chunk
// order by a second kernel.  Lane j of a group adds arcs j, j+L, j+2L, ... (four independent loads
// per pass) and the group reduces with xor shuffles, so every row's sum has a fixed association
// order for a given schedule: results are deterministic run to run.  Column indices of one group
// are contiguous (coalesced); the gathered value is the only random access.
//
//   Gather: __device__ double operator()(uint32_t row, uint64_t arc) const   value of one arc
//           __device__ bool skips(uint32_t row) const   (optional) rows left out: no arcs, sum 0
//           __device__ void warm(uint64_t arc) const   (optional) loads of the arc that no launch changes
//           static constexpr bool kDeep   (optional) true: eight arcs a lane in flight
//           static constexpr int kBlocks   (optional) blocks an SM that the kernel's registers must allow
//   Finish: __device__ void operator()(uint32_t row, double sum)
//           __device__ void end()   (optional) after the block's last row, by all its threads
//           __device__ bool stopped() const   (optional) true: the launch does nothing
#pragma once
#include "gre_internal.cuh"

namespace gre {
namespace rows {

constexpr int kCta = 256;

// A Finish that gathers something over the rows of a thread (a largest change) hands it on here,
// once a block instead of once a row.
template <class F>
__device__ __forceinline__ auto finish_end(F& f, int) -> decltype(f.end()) { f.end(); }
template <class F>
__device__ __forceinline__ void finish_end(F&, long) {}
template <class F>
__device__ __forceinline__ auto launch_stopped(const F& f, int) -> decltype(f.stopped()) { return f.stopped(); }
template <class F>
__device__ __forceinline__ bool launch_stopped(const F&, long) { return false; }
template <class G>
constexpr auto deep_gather(int) -> decltype(G::kDeep) { return G::kDeep; }
template <class G>
constexpr bool deep_gather(long) { return false; }
template <class G>
constexpr auto gather_blocks(int) -> decltype(G::kBlocks) { return G::kBlocks; }
template <class G>
constexpr int gather_blocks(long) { return 0; }  // the compiler chooses
template <class G>
__device__ __forceinline__ auto row_skipped(const G& g, uint32_t v, int) -> decltype(g.skips(v)) { return g.skips(v); }
template <class G>
__device__ __forceinline__ bool row_skipped(const G&, uint32_t, long) { return false; }

// The next superstep's blocks start while this one's last run (launch_early); a block looks its first row
// up (row, offsets, the first arcs' columns: the graph's own arrays) before it waits for them.
// PageRank-20, launches one after the other / early / with the look-up: RMAT-14 171 / 135 / 122 us, RMAT-16
// directed 220 / 209 / 193, RMAT-18 489 / 452 / 451, RMAT-20 1738 / 1627 / 1611; an iteration of the weighted solves at
// RMAT-20 108.7 / 107.1 / 105.7 us.
template <class G>
__device__ __forceinline__ auto warm_arc(const G& g, uint64_t a, int) -> decltype(g.warm(a)) { g.warm(a); }
template <class G>
__device__ __forceinline__ void warm_arc(const G&, uint64_t, long) {}
struct Ready {
  bool waited = false, stop = false;
  template <int L, class Gather, class Finish>
  __device__ __forceinline__ bool operator()(const Gather& gat, const Finish& fin, uint64_t a0, uint64_t a1, uint32_t lig) {
    if (!waited) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (a0 + lig + j * L < a1) warm_arc(gat, a0 + lig + j * L, 0);
      wait_previous();
      stop = launch_stopped(fin, 0);
      waited = true;
    }
    return !stop;
  }
};

// Sum of gat(v, a) over a = a0 + lig, a0 + lig + L, ... < a1.  Four arcs per pass so that each
// lane has four independent (column, gathered value) load chains in flight: the loop is bound
// by memory latency, not bandwidth, when a lane waits on one chain at a time.  Eight where the gather
// asks for it: with a stream of FP64 weights beside the columns (RMAT-20, an iteration) 118 -> 113 us; the plain
// PageRank, at 70-80% of what L1 and L2 give to gathers, lost 1% at RMAT-22.  The two or three arcs left are in
// flight together as well (PageRank-20 at RMAT-22, default schedule: 7695 us one by one, 7498 so; 96 iterations of the weighted
// solve at RMAT-20 10.91 -> 10.53 ms, RMAT-16 1163 -> 1050 us).
template <int L, class Gather>
__device__ __forceinline__ double strided_sum(Gather& gat, uint32_t v, uint64_t a0, uint64_t a1, uint32_t lig) {
  double acc = 0.0;
  uint64_t a = a0 + lig;
  if constexpr (deep_gather<Gather>(0))
    for (; a + 7 * (uint64_t)L < a1; a += 8 * (uint64_t)L) {
      double x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = gat(v, a + j * (uint64_t)L);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc += x[j];
    }
  for (; a + 3 * (uint64_t)L < a1; a += 4 * (uint64_t)L) {
    const double x0 = gat(v, a), x1 = gat(v, a + L), x2 = gat(v, a + 2 * L), x3 = gat(v, a + 3 * L);
    acc += x0;
    acc += x1;
    acc += x2;
    acc += x3;
  }
  if (a + L < a1) {
    const double x0 = gat(v, a), x1 = gat(v, a + L);
    acc += x0;
    acc += x1;
    a += 2 * (uint64_t)L;
  }
  if (a < a1) acc += gat(v, a);
  return acc;
}

// The rows of one bin, L lanes each: block `part` of `nparts` takes every nparts-th group of
// 256 / L rows.
template <int L, class Gather, class Finish>
__device__ __forceinline__ void rows_lanes(const uint32_t* __restrict__ rows, uint32_t count, uint32_t part, uint32_t nparts,
                                           const uint64_t* __restrict__ off, Gather& gat, Finish& fin, Ready& ready) {
  const uint32_t lig = threadIdx.x % L;
  const uint64_t step = (uint64_t)nparts * (kCta / L);
  // the warp stays together for the shuffles: its first row decides
  for (uint64_t base = (uint64_t)part * (kCta / L) + (threadIdx.x & ~31u) / L; base < count; base += step) {
    const uint64_t i = base + (threadIdx.x & 31u) / L;
    const bool valid = i < count;
    double acc = 0.0;
    uint32_t v = 0;
    if (valid) v = rows[i];
    if (!ready.waited) {
      if (!ready.template operator()<L>(gat, fin, valid ? off[v] : 0, valid ? off[v + 1] : 0, lig)) return;
    }
    if (valid && !row_skipped(gat, v, 0)) acc = strided_sum<L>(gat, v, off[v], off[v + 1], lig);
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (valid && lig == 0) fin(v, acc);
  }
}

__device__ __forceinline__ double block_sum(double x, double* smem) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) smem[w] = x;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += smem[i];
  }
  __syncthreads();
  return t;  // valid in thread 0
}

// What one block of k_rows_all works on.  Segment 0: chunks of the multi-CTA rows (window chunks
// when the schedule splits rows by source window); 1: a CTA per row; 2..7: 32, 16, 8, 4, 2, 1
// lanes per row.  Segment s owns blocks [block[s], block[s + 1]).
struct RowPlan {
  uint32_t block[9];
  uint32_t count[8];        // chunks or rows
  uint32_t row0[8];         // first entry of the segment in `rows`
  const uint32_t* rows;     // DegreeBins::rows
  const uint64_t* chunk_row;
  const uint64_t* chunk_begin;
  uint64_t chunk;           // arcs per chunk
  const uint32_t* seg_row;  // window chunks: null when not split
  const uint64_t* seg_begin;
  const uint64_t* seg_end;
  const uint64_t* seg_slot;
};

// Blocks of one segment: enough for one pass, at most kSegBlocks an SM (the blocks of a long
// segment stride over it).
constexpr int kSegBlocks = 16;

// The bins' rows (the window chunks instead of bins 6 and 7 with `windows`).
inline RowPlan plan_rows(const DegreeBins& B, bool windows, int seg_blocks = kSegBlocks) {
  RowPlan P{};
  P.rows = B.rows;
  P.chunk_row = B.hub_chunk_row;
  P.chunk_begin = B.hub_chunk_begin;
  P.chunk = B.sched.hub_chunk;
  if (windows) {
    P.seg_row = B.seg_row;
    P.seg_begin = B.seg_begin;
    P.seg_end = B.seg_end;
    P.seg_slot = B.seg_slot;
  }
  for (int k = 0; k < 8; ++k) {
    const int b = 7 - k;  // segment k holds bin 7 - k
    const uint64_t items = k == 0 ? (windows ? B.seg_nchunks : B.n_hub_chunks) : (k == 1 && windows) ? 0 : B.count[b];
    P.count[k] = (uint32_t)items;
    P.row0[k] = (uint32_t)B.start[b];
    const uint64_t threads = items * (k < 2 ? kCta : 1ull << b);
    P.block[k + 1] = P.block[k] + (items ? grid_for(threads, kCta, seg_blocks) : 0);
  }
  return P;
}

// Every bin of a superstep in one launch.  Latency and tails bound a superstep of a small graph
// when its bins run one after the other (RMAT-16, seven bins: 40 us a superstep, each bin 7-20 us
// alone); side by side they take as long as the slowest.  The blocks of the longest rows come
// first, so that the short ones fill the gaps at the end (PageRank-20: RMAT-16
// directed 820 -> 314 us, RMAT-24 36.1 -> 31.9 ms; weighted solves at RMAT-20 147 -> 60 ms).  The sums are
// those of a launch per bin: a row's association order depends on its bin alone.
template <class Gather, class Finish>
__global__ void __launch_bounds__(kCta, gather_blocks<Gather>(0)) k_rows_all(const __grid_constant__ RowPlan P, const uint64_t* __restrict__ off, Gather gat,
                                                   Finish fin, double* __restrict__ partial) {
  __shared__ double smem[kCta / 32];
  launch_next();
  Ready ready;
  uint32_t s = 0;
  while (blockIdx.x >= P.block[s + 1]) ++s;
  const uint32_t part = blockIdx.x - P.block[s], nparts = P.block[s + 1] - P.block[s], count = P.count[s];
  const uint32_t* rows = P.rows + P.row0[s];
  if (s == 0) {
    for (uint64_t c = part; c < count; c += nparts) {
      uint32_t v;
      uint64_t a0, a1, slot = c;
      if (P.seg_row) {
        v = P.seg_row[c];
        a0 = P.seg_begin[c];
        a1 = P.seg_end[c];
        slot = P.seg_slot[c];
      } else {
        v = rows[P.chunk_row[c]];
        a0 = P.chunk_begin[c];
        const uint64_t end = off[v + 1];
        a1 = (a0 + P.chunk < end) ? a0 + P.chunk : end;
      }
      if (!ready.template operator()<kCta>(gat, fin, a0, a1, threadIdx.x)) return;
      if (row_skipped(gat, v, 0)) a1 = a0;
      const double acc = block_sum(strided_sum<kCta>(gat, v, a0, a1, threadIdx.x), smem);
      if (threadIdx.x == 0) partial[slot] = acc;
    }
    return;
  }
  if (s == 1) {
    for (uint64_t i = part; i < count; i += nparts) {
      const uint32_t v = rows[i];
      const uint64_t a0 = off[v];
      uint64_t a1 = off[v + 1];
      if (!ready.template operator()<kCta>(gat, fin, a0, a1, threadIdx.x)) return;
      if (row_skipped(gat, v, 0)) a1 = a0;
      const double acc = block_sum(strided_sum<kCta>(gat, v, a0, a1, threadIdx.x), smem);
      if (threadIdx.x == 0) fin(v, acc);
    }
  } else if (s == 2) {
    rows_lanes<32>(rows, count, part, nparts, off, gat, fin, ready);
  } else if (s == 3) {
    rows_lanes<16>(rows, count, part, nparts, off, gat, fin, ready);
  } else if (s == 4) {
    rows_lanes<8>(rows, count, part, nparts, off, gat, fin, ready);
  } else if (s == 5) {
    rows_lanes<4>(rows, count, part, nparts, off, gat, fin, ready);
  } else if (s == 6) {
    rows_lanes<2>(rows, count, part, nparts, off, gat, fin, ready);
  } else {
    rows_lanes<1>(rows, count, part, nparts, off, gat, fin, ready);
  }
  if (!ready.template operator()<1>(gat, fin, 0, 0, 0)) return;  // warps without a row wait too
  finish_end(fin, 0);
}

// The partial sums of the chunked rows, added in chunk order.
template <class Finish>
__global__ void k_rows_chunk_finish(const uint32_t* __restrict__ rows, uint64_t count, const uint64_t* __restrict__ first,
                                    const double* __restrict__ partial, Finish fin) {
  if (launch_stopped(fin, 0)) return;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (uint64_t c = first[i]; c < first[i + 1]; ++c) s += partial[c];
    fin(rows[i], s);
  }
  finish_end(fin, 0);
}

// Launch the reductions of every non-empty row.  `partial` holds bins.n_partials doubles.
template <class Gather, class Finish>
int reduce_rows(const DegreeBins& B, const uint64_t* off, Gather gat, Finish fin, double* partial, cudaStream_t s,
                int seg_blocks = kSegBlocks) {
  const bool windows = B.seg_nchunks != 0;  // the rows above cta_min, window by window
  const RowPlan P = plan_rows(B, windows, seg_blocks);
  if (!P.block[8]) return GRE_SUCCESS;
  GRE_CHECK(launch_early(s, P.block[8], kCta, k_rows_all<Gather, Finish>, P, off, gat, fin, partial));
  if (windows)
    k_rows_chunk_finish<<<grid_for(B.seg_nrows, 128, 4), 128, 0, s>>>(B.seg_rows, B.seg_nrows, B.seg_first, partial, fin);
  else if (B.count[7])
    k_rows_chunk_finish<<<grid_for(B.count[7], 128, 4), 128, 0, s>>>(B.rows + B.start[7], B.count[7], B.hub_chunk_first, partial, fin);
  GRE_LAUNCH_CHECK();
  return GRE_SUCCESS;
}

// Visits of every arc whose sums nobody reads: the bins one after the other, short rows first.
template <class Gather, class Finish>
int visit_rows_apart(const DegreeBins& B, const uint64_t* off, Gather gat, Finish fin, double* partial, cudaStream_t s,
                     int seg_blocks) {
  const RowPlan all = plan_rows(B, B.seg_nchunks != 0, seg_blocks);
  for (int k = 7; k >= 0; --k) {
    const uint32_t blocks = all.block[k + 1] - all.block[k];
    if (!blocks) continue;
    RowPlan P = all;
    for (int i = 0; i <= 8; ++i) P.block[i] = i > k ? blocks : 0;
    GRE_CHECK(launch_early(s, blocks, kCta, k_rows_all<Gather, Finish>, P, off, gat, fin, partial));
  }
  return GRE_SUCCESS;
}

// Number of non-empty rows of the bins (for byte models).
inline uint64_t nonempty_rows(const DegreeBins& B) {
  uint64_t s = 0;
  for (int i = 0; i < DegreeBins::NB; ++i) s += B.count[i];
  return s;
}

}  // namespace rows
}  // namespace gre
