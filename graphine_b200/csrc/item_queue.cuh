// Queues of the persistent frontier kernels (BFS, SSSP): a vertex's arcs as items of kPiece arcs,
// so that a hub's row is spread over the grid, appended through shared memory, and walked by warps
// that lay the arcs of up to 32 items side by side.
#pragma once
#include "gre_internal.cuh"

namespace gre {

constexpr uint32_t kPiece = 128;  // arcs per queue item: one pass of a warp

__host__ __device__ __forceinline__ uint32_t items_of(uint64_t arcs) { return (uint32_t)((arcs + kPiece - 1) / kPiece); }

#ifdef __CUDACC__
// Queue appends of one block in one phase.  Vertices of one item are gathered per warp in shared
// memory and moved out kStage at a time, the rest of all warps with one atomic a block at the
// phase's end: an atomic a warp and step on the one counter bounded the large levels (BFS at
// RMAT-22, a frontier of hubs: 73 us).  Vertices of several items go straight to the queue.
constexpr uint32_t kStage = 96;

template <int THREADS>
struct ItemStage {
  uint32_t item[THREADS / 32][kStage];
  uint32_t held[THREADS / 32];
  uint32_t base;
};

__device__ __forceinline__ void put_item(uint2* q, uint32_t v, uint32_t piece) { *q = make_uint2(v, piece); }
__device__ __forceinline__ void put_item(uint32_t* q, uint32_t v, uint32_t) { *q = v; }  // a plain list

template <int THREADS, class T>
struct ItemAppend {
  ItemStage<THREADS>& st;
  uint32_t held = 0;
  unsigned int* count;
  T* queue;
  __device__ __forceinline__ ItemAppend(ItemStage<THREADS>& s, unsigned int* c, T* q) : st(s), count(c), queue(q) {}
  __device__ __forceinline__ void move(uint32_t base) {
    const uint32_t* buf = st.item[threadIdx.x >> 5];
    for (uint32_t i = lane_id(); i < held; i += 32) put_item(queue + base + i, buf[i], 0);
    held = 0;
  }
  // vertex v where `want` (warp-uniform call)
  __device__ __forceinline__ void push_one(uint32_t v, bool want) {
    const uint32_t lane = lane_id();
    const uint32_t one = __ballot_sync(0xffffffffu, want);
    if (!one) return;
    if (held + 32 > kStage) {
      __syncwarp();
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(count, held);
      move(__shfl_sync(0xffffffffu, base, 0));
      __syncwarp();
    }
    if (want) st.item[threadIdx.x >> 5][held + __popc(one & ((1u << lane) - 1u))] = v;
    held += __popc(one);
  }
  // nit[k] items of vertex v[k] per lane (warp-uniform call)
  template <int U>
  __device__ __forceinline__ void push(const uint32_t (&v)[U], const uint32_t (&nit)[U]) {
    constexpr uint32_t kOwn = 8;  // more items than that are written by the whole warp
    const uint32_t lane = lane_id();
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      push_one(v[k], nit[k] == 1);
      if (nit[k] > 1) sum += nit[k];
    }
    if (!__any_sync(0xffffffffu, sum)) return;
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (uint32_t)o) incl += x;
    }
    uint32_t at = 0;
    if (lane == 31) at = atomicAdd(count, incl);
    at = __shfl_sync(0xffffffffu, at, 31) + incl - sum;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const uint32_t mine = nit[k] > 1 ? nit[k] : 0;
      if (mine <= kOwn)
        for (uint32_t i = 0; i < mine; ++i) put_item(queue + at + i, v[k], i);
      for (uint32_t many = __ballot_sync(0xffffffffu, mine > kOwn); many; many &= many - 1) {
        const int src = __ffs(many) - 1;
        const uint32_t sv = __shfl_sync(0xffffffffu, v[k], src), sn = __shfl_sync(0xffffffffu, mine, src);
        const uint32_t sb = __shfl_sync(0xffffffffu, at, src);
        for (uint32_t i = lane; i < sn; i += 32) put_item(queue + sb + i, sv, i);
      }
      at += mine;
    }
  }
  // The end of a phase, by all threads of the block: post, a barrier, claim by a warp, a barrier,
  // take (and a barrier before the stage is used again).  Several queues share the barriers.
  __device__ __forceinline__ void post() {
    if (lane_id() == 0) st.held[threadIdx.x >> 5] = held;
  }
  __device__ __forceinline__ void claim() {  // by one whole warp
    const uint32_t lane = lane_id(), h = lane < THREADS / 32 ? st.held[lane] : 0;
    uint32_t incl = h;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (uint32_t)o) incl += x;
    }
    if (lane < THREADS / 32) st.held[lane] = incl - h;  // the warp's place
    if (lane == 31 && incl) st.base = atomicAdd(count, incl);
  }
  __device__ __forceinline__ void take() { move(st.base + st.held[threadIdx.x >> 5]); }
  __device__ __forceinline__ void finish() {
    post();
    if (!__syncthreads_or(held)) return;
    if (threadIdx.x < 32) claim();
    __syncthreads();
    take();
    __syncthreads();
  }
};

// Per-thread sums of a phase, one atomic each a block (all threads call).
template <int K>
struct BlockSums {
  unsigned long long sum[K];
  __device__ __forceinline__ void add(const unsigned long long (&x)[K], unsigned long long* const (&to)[K]) {
    if (threadIdx.x < K) sum[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) {
      unsigned long long s = x[k];
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane_id() == 0 && s) atomicAdd(&sum[k], s);
    }
    __syncthreads();
    if (threadIdx.x < K && sum[threadIdx.x]) {
#pragma unroll
      for (int k = 0; k < K; ++k)  // no indexing by thread: `to` stays in registers
        if (threadIdx.x == k) atomicAdd(to[k], sum[k]);
    }
    __syncthreads();
  }
};

// The k-th (from 0) set bit of a word that has more than k.
__device__ __forceinline__ uint32_t nth_bit(uint32_t w, uint32_t k) {
  uint32_t pos = 0;
#pragma unroll
  for (uint32_t s = 16; s; s >>= 1) {
    const uint32_t low = __popc(w & ((1u << s) - 1u));
    if (k >= low) {
      k -= low;
      w >>= s;
      pos += s;
    }
  }
  return pos;
}

// The words of a bitmap, 32 to a warp: eight neighbours (a sector) from each quarter, so that where
// the set bits crowd in one part of the ids, every warp has a share of it.  Word of `lane` in chunk
// c of bit_chunks(nwords); >= nwords: none.
__host__ __device__ __forceinline__ uint64_t bit_chunks(uint64_t nwords) { return (nwords + 31) / 32; }
__device__ __forceinline__ uint64_t chunk_word(uint64_t c, uint64_t chunks) {
  return ((lane_id() >> 3) * chunks + c) * 8 + (lane_id() & 7);
}

// Calls f(valid, index) for the set bits of a warp's 32 words (each lane's word and its number), U
// times 32 bits at a time on 32 lanes however they are spread over the words: f gets U of both.
template <int U, class F>
__device__ __forceinline__ void for_bits(uint64_t number, uint32_t word, F&& f) {
  const uint32_t cnt = __popc(word);
  uint32_t incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane_id() >= (uint32_t)o) incl += x;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31), excl = incl - cnt;
  for (uint32_t t = 0; t < total; t += 32 * U) {
    bool valid[U];
    uint32_t index[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const uint32_t pos = t + 32 * k + lane_id();
      uint32_t own = 0;  // last lane that begins at or before pos: it holds the bit (those after begin later)
#pragma unroll
      for (uint32_t step = 16; step; step >>= 1)
        if (__shfl_sync(0xffffffffu, excl, own + step) <= pos) own += step;
      const uint32_t w = __shfl_sync(0xffffffffu, word, own), j = pos - __shfl_sync(0xffffffffu, excl, own);
      const uint32_t num = __shfl_sync(0xffffffffu, (uint32_t)number, own);
      valid[k] = pos < total;
      index[k] = valid[k] ? (num << 5) + nth_bit(w, j) : 0u;
    }
    f(valid, index);
  }
}

// The arcs of a warp's items side by side: position pos in [0, total) belongs to the item of lane
// owner(pos), at arc arc_of(pos, owner).  All lanes call.
struct ItemSpan {
  uint64_t a0;
  uint32_t excl, total;
  __device__ __forceinline__ ItemSpan(uint64_t first, uint32_t len) : a0(first) {
    uint32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane_id() >= (uint32_t)o) incl += x;
    }
    excl = incl - len;
    total = __shfl_sync(0xffffffffu, incl, 31);
  }
  // last item that begins at or before pos (items are not empty; lanes without one begin at total)
  __device__ __forceinline__ uint32_t owner(uint32_t pos) const {
    uint32_t own = 0;
#pragma unroll
    for (uint32_t step = 16; step; step >>= 1)
      if (__shfl_sync(0xffffffffu, excl, own + step) <= pos) own += step;
    return own;
  }
  __device__ __forceinline__ uint64_t arc_of(uint32_t pos, uint32_t own) const {
    return __shfl_sync(0xffffffffu, a0, own) + (pos - __shfl_sync(0xffffffffu, excl, own));
  }
};
#endif

}  // namespace gre
