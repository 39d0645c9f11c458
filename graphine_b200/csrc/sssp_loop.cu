// SSSP's superstep loop in one cooperative kernel.
//
// A run has some 45 supersteps (light passes of the buckets, one heavy pass a bucket, limit
// rises), nearly all over a few thousand vertices.  Driven from the host each cost 5-7 launches and
// 2-3 counter reads, which bounded the run (RMAT-22: 4.2 ms a source; 60000 vertices: 2.9 ms).  Here
// the loop runs in the kernel, the blocks meeting at a grid barrier after the relaxation and after
// the classification of a pass; only the few passes over a large share of the graph are left to
// the binned kernels (sssp.cu), which stream rows with more warps resident: the kernel ends with its
// state, the host launches the pass and then the kernel again.
//
// Frontiers are queues of items (vertex, 128-arc piece of its light or heavy range).  The thread that
// improves a vertex also says where it goes: below the limit the first to set its near bit appends
// its light items to the next queue and the first to set its bucket bit its heavy items; at or above
// the limit it sets the far bit.  So a pass is one phase and one barrier.  The near bits are two
// bitmaps in turn: a pass sets one and clears, with the items that it reads, the other.  A far bit
// stays set when its vertex comes below the limit in the same bucket; the next rise drops it.
//
// Counters: every block decides from the same counters after a barrier, so nothing a block may
// still read there is changed before the next one.  A phase fills the next of three near counters
// (a heavy pass or a rise the next bucket's too, a rise the next far count) and clears the one after.
//
// Measured against the host-driven loop: RMAT-22, four sources, 16.9 -> 8.3 ms; RMAT-26 17.3 -> 12.2 ms
// a source; 60000 vertices, directed, 2810 -> 446 us (630 at the same bucket width); a grid of 1000 x 1000
// 690 -> 73 ms.  A pass over a handful of vertices is 4 us (half of it the barrier), one over a few thousand 8-18 us
// (five dependent round trips).
#include <algorithm>

#include "sssp_loop.cuh"

namespace gre {

constexpr int kSsspThreads = 512;

struct SsspTop {  // what the blocks decide from
  uint32_t nit, nv, hit, hv, dmin;
  int nfar;
  unsigned long long na, ha;
};

struct SsspStage {
  SsspTop top;
  ItemStage<kSsspThreads> a, b;
  unsigned int verts[2], dmin;
  int far;
  unsigned long long arcs[2];
};

// Appends of a phase: vertices that enter the near queue or the bucket, and changes of the far count.
struct Entries {
  const SsspRun& R;
  SsspStage& st;
  SsspQueue *nq, *hq;
  int* nfar;
  uint32_t *nbits, *hbits;  // the near and bucket bits that this phase sets
  ItemAppend<kSsspThreads, uint2> near, heavy;
  uint32_t nv = 0, hv = 0;
  int far = 0;
  unsigned long long na = 0, ha = 0;
  __device__ __forceinline__ Entries(const SsspRun& r, SsspStage& s, SsspQueue* n, uint32_t nbuf, uint32_t* bits, SsspQueue* h, uint32_t hbuf, int* f)
      : R(r), st(s), nq(n), hq(h), nfar(f), nbits(bits), hbits(r.hbits[hbuf]), near(s.a, &n->items, r.near[nbuf]),
        heavy(s.b, &h->items, r.heavy[hbuf]) {}
  // Of U vertices per lane (warp-uniform call), those `below` the limit enter the near queue and the
  // bucket, those `above` the far set, each once; a vertex without out-arcs goes nowhere.  Stage by
  // stage over the U, so that their loads and atomics are in flight together.
  template <int U>
  __device__ __forceinline__ void classify(const uint32_t (&v)[U], const bool (&below)[U], const bool (&above)[U]) {
    bool near_new[U], heavy_new[U], far_new[U], some = false;
#pragma unroll
    for (int k = 0; k < U; ++k) some = some || below[k] || above[k];
    if (!__any_sync(0xffffffffu, some)) return;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const uint32_t w = v[k] >> 5, bit = 1u << (v[k] & 31u);
      near_new[k] = below[k] && !(__ldcg(nbits + w) & bit);
      heavy_new[k] = below[k] && !(__ldcg(hbits + w) & bit);
      far_new[k] = above[k] && !(__ldcg(R.infar + w) & bit);
    }
    uint32_t nl[U], nh[U];
    bool any = false;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      nl[k] = nh[k] = 0;
      if (near_new[k] || heavy_new[k] || (far_new[k] && !R.all_out)) {
        const uint64_t a0 = R.off[v[k]], am = R.lend[v[k]], a1 = R.off[v[k] + 1];
        near_new[k] = near_new[k] && am > a0;
        heavy_new[k] = heavy_new[k] && a1 > am;
        far_new[k] = far_new[k] && a1 > a0;
        nl[k] = (uint32_t)(am - a0);
        nh[k] = (uint32_t)(a1 - am);
      }
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const uint32_t w = v[k] >> 5, bit = 1u << (v[k] & 31u);
      if (near_new[k]) near_new[k] = !(atomicOr(nbits + w, bit) & bit);
      if (heavy_new[k]) heavy_new[k] = !(atomicOr(hbits + w, bit) & bit);
      if (far_new[k]) far_new[k] = !(atomicOr(R.infar + w, bit) & bit);
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      far += far_new[k];
      if (near_new[k]) {
        ++nv;
        na += nl[k];
      }
      if (heavy_new[k]) {
        ++hv;
        ha += nh[k];
      }
      nl[k] = near_new[k] ? items_of(nl[k]) : 0;
      nh[k] = heavy_new[k] ? items_of(nh[k]) : 0;
      any = any || nl[k] || nh[k];
    }
    if (!__any_sync(0xffffffffu, any)) return;
    near.push(v, nl);
    heavy.push(v, nh);
  }
  // the end of the phase, by all threads; the block's counters in `st` are zero before and after
  __device__ __forceinline__ void finish() {
    near.post();
    heavy.post();
    nv = __reduce_add_sync(0xffffffffu, nv);
    hv = __reduce_add_sync(0xffffffffu, hv);
    far = __reduce_add_sync(0xffffffffu, far);
    if (nv | hv) {  // uniform in the warp
      for (int o = 16; o > 0; o >>= 1) {
        na += __shfl_xor_sync(0xffffffffu, na, o);
        ha += __shfl_xor_sync(0xffffffffu, ha, o);
      }
    }
    if (lane_id() == 0) {
      if (nv) atomicAdd(&st.verts[0], nv), atomicAdd(&st.arcs[0], na);
      if (hv) atomicAdd(&st.verts[1], hv), atomicAdd(&st.arcs[1], ha);
      if (far) atomicAdd(&st.far, far);
    }
    if (!__syncthreads_or(near.held | heavy.held | nv | hv | far)) return;
    if (threadIdx.x < 32) {
      near.claim();
    } else if (threadIdx.x < 64) {
      heavy.claim();
    } else if (threadIdx.x == 64) {
      if (st.verts[0]) atomicAdd(&nq->verts, st.verts[0]), atomicAdd(&nq->arcs, st.arcs[0]);
      if (st.verts[1]) atomicAdd(&hq->verts, st.verts[1]), atomicAdd(&hq->arcs, st.arcs[1]);
      if (st.far) atomicAdd(nfar, st.far);
      clear();
    }
    __syncthreads();
    near.take();
    heavy.take();
    __syncthreads();
  }
  __device__ __forceinline__ void clear() {
    st.verts[0] = st.verts[1] = 0;
    st.arcs[0] = st.arcs[1] = 0;
    st.far = 0;
  }
};

// Relaxes the arcs of the items.  WIDE: an improvement sets its bit in `changed` and nobody waits for
// an atomic's answer (classify_bits follows); else it is classified on the spot.
template <bool HEAVY, bool WIDE, int U>
__device__ __forceinline__ void relax_items(const SsspRun& R, const uint2* items, uint32_t nitems, uint32_t* bits, uint32_t limit,
                                            Entries& E, uint32_t gwarp, uint32_t nwarps) {
  const uint32_t lane = lane_id();
  // few items: one a warp, so that all warps share the arcs
  const uint32_t per = min(32u, max(1u, (nitems + nwarps - 1) / nwarps));
  for (uint64_t base = (uint64_t)gwarp * per; base < nitems; base += (uint64_t)nwarps * per) {
    uint64_t a0 = 0;
    uint32_t len = 0, du = 0;
    if (lane < per && base + lane < nitems) {
      const uint2 it = __ldcg(items + base + lane);
      const uint64_t mid = R.lend[it.x];
      a0 = (HEAVY ? mid : R.off[it.x]) + (uint64_t)it.y * kPiece;
      len = (uint32_t)min((uint64_t)kPiece, (HEAVY ? R.off[it.x + 1] : mid) - a0);
      du = __ldcg(R.dist + it.x);
      if (it.y == 0) atomicAnd(bits + (it.x >> 5), ~(1u << (it.x & 31u)));  // leaves the queue
    }
    const ItemSpan span(a0, len);
    for (uint32_t t = 0; t < span.total; t += 32 * U) {
      uint32_t x[U], nd[U], dv[U];
      bool ok[U];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const uint32_t pos = t + 32 * k + lane;
        const uint32_t own = span.owner(pos);
        const uint64_t arc = span.arc_of(pos, own);
        nd[k] = __shfl_sync(0xffffffffu, du, own);
        ok[k] = pos < span.total;
        x[k] = 0;
        if (ok[k]) {
          x[k] = __ldg(R.col + arc);
          nd[k] += __ldg(R.w + arc);
        }
      }
#pragma unroll
      for (int k = 0; k < U; ++k) dv[k] = ok[k] ? __ldcg(R.dist + x[k]) : 0u;
      if (WIDE) {
#pragma unroll
        for (int k = 0; k < U; ++k)
          if (ok[k] && nd[k] < dv[k]) {
            atomicMin(R.dist + x[k], nd[k]);
            atomicOr(R.changed + (x[k] >> 5), 1u << (x[k] & 31u));
          }
      } else {
        bool above[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const bool better = ok[k] && nd[k] < dv[k];
          if (better) atomicMin(R.dist + x[k], nd[k]);
          ok[k] = better && nd[k] < limit;
          above[k] = better && nd[k] >= limit;
        }
        E.classify(x, ok, above);
      }
    }
  }
}

// The vertices with a `changed` bit (cleared) enter the queues and the far set.
__device__ __forceinline__ void classify_bits(const SsspRun& R, uint32_t limit, Entries& E, uint32_t gwarp, uint32_t nwarps) {
  constexpr int U = 2;
  const uint64_t chunks = bit_chunks(R.nwords);
  for (uint64_t ch = gwarp; ch < chunks; ch += nwarps) {
    const uint64_t num = chunk_word(ch, chunks);
    uint32_t word = 0;
    if (num < R.nwords) {
      word = R.changed[num];
      if (word) R.changed[num] = 0;
    }
    for_bits<U>(num, word, [&](const bool (&valid)[U], const uint32_t (&v)[U]) {
      bool below[U], above[U];
      uint32_t d[U];
#pragma unroll
      for (int k = 0; k < U; ++k) d[k] = valid[k] ? __ldcg(R.dist + v[k]) : 0u;
#pragma unroll
      for (int k = 0; k < U; ++k) {
        below[k] = valid[k] && d[k] < limit;
        above[k] = valid[k] && d[k] >= limit;
      }
      E.classify(v, below, above);
    });
  }
}

__device__ __forceinline__ void clear_queue(SsspQueue* q) {
  q->items = q->verts = 0;
  q->arcs = 0;
}
__device__ __forceinline__ uint32_t next3(uint32_t i) { return i == 2 ? 0 : i + 1; }

__global__ void __launch_bounds__(kSsspThreads, 2) k_sssp_loop(const __grid_constant__ SsspRun R) {
  __shared__ SsspStage st;
  const uint32_t lane = lane_id();
  const uint32_t gwarp = (blockIdx.x * kSsspThreads + threadIdx.x) >> 5, nwarps = gridDim.x * (kSsspThreads / 32);
  const uint64_t gtid = blockIdx.x * (uint64_t)kSsspThreads + threadIdx.x, nthreads = (uint64_t)gridDim.x * kSsspThreads;
  const bool first = blockIdx.x == 0 && threadIdx.x == 0;
  SsspCtl* c = R.ctl;
  unsigned int target = 0;
  uint32_t limit = R.limit, p = R.p, q = R.q, r = R.r;
  uint32_t nb = R.nb, hb = R.hb;  // the near and bucket buffers in use (with their bits)
  uint32_t tries = 0;  // limit rises since a vertex came below the limit
  if (threadIdx.x == 0) {
    st.verts[0] = st.verts[1] = 0;
    st.arcs[0] = st.arcs[1] = 0;
    st.far = 0;
  }
  if (R.fresh) {
    for (uint64_t v = gtid; v < R.n; v += nthreads) R.dist[v] = 0xffffffffu;
    for (uint64_t i = gtid; i < R.nwords; i += nthreads) R.changed[i] = R.infar[i] = R.hbits[0][i] = R.hbits[1][i] = R.nbits[0][i] = R.nbits[1][i] = 0;
    if (!grid_barrier(&c->bar, target, R.wait_ns)) return;
    if (blockIdx.x == 0) {
      Entries E(R, st, &c->near[p], nb, R.nbits[nb], &c->heavy[q], hb, &c->nfar[r]);
      if (threadIdx.x == 0) R.dist[R.src] = 0;
      const uint32_t v[1] = {R.src};
      const bool below[1] = {threadIdx.x == 0}, above[1] = {false};
      E.classify(v, below, above);
      E.finish();
    }
  }
  uint32_t reason = SSSP_DONE;
  bool record = R.record_entry;
  for (;;) {
    if (!grid_barrier(&c->bar, target, R.wait_ns, [&] {
          const SsspQueue *nq = &c->near[p], *hq = &c->heavy[q];
          st.top.nit = __ldcg(&nq->items);
          st.top.nv = __ldcg(&nq->verts);
          st.top.na = __ldcg(&nq->arcs);
          st.top.hit = __ldcg(&hq->items);
          st.top.hv = __ldcg(&hq->verts);
          st.top.ha = __ldcg(&hq->arcs);
          st.top.nfar = __ldcg(&c->nfar[r]);
          st.top.dmin = __ldcg(&c->dmin[next3(next3(r))]);
        }))
      return;
    const uint32_t nit = st.top.nit, nv = st.top.nv, hit = st.top.hit, hv = st.top.hv;
    const int nfar = st.top.nfar;
    if (record) {
      if (first && R.rec) {
        if (c->nrec < R.nrec) R.rec[c->nrec] = nv;
        c->nrec += 1;
      }
      record = false;
    }
    // what is next: the near queue's light arcs; the settled bucket's heavy arcs; a limit rise
    const bool light = nit != 0, heavy = !light && hit != 0;
    if (light || heavy) {
      tries = 0;
      const unsigned long long arcs = heavy ? st.top.ha : st.top.na;
      const uint32_t verts = heavy ? hv : nv;
      if (verts >= R.big_verts || (heavy && arcs >= R.big_arcs)) {
        reason = heavy ? SSSP_BIG_HEAVY : SSSP_BIG_LIGHT;
        break;
      }
      const uint32_t pn = next3(p), qn = heavy ? next3(q) : q;
      if (first) {
        c->relaxed += arcs;
        c->bytes += 16 * verts + 12 * arcs;
        c->steps += 1;
        clear_queue(&c->near[next3(pn)]);
        if (heavy) clear_queue(&c->heavy[next3(qn)]);
      }
      // heavy arcs land at or above the limit, so that pass normally enters nothing (a distance that
      // wrapped around 2^32 may): what it enters goes to the next bucket
      Entries E(R, st, &c->near[pn], nb ^ 1, R.nbits[nb ^ 1], &c->heavy[qn], heavy ? hb ^ 1 : hb, &c->nfar[r]);
      if (arcs < R.wide_arcs) {
        if (heavy) relax_items<true, false, 4>(R, R.heavy[hb], hit, R.hbits[hb], limit, E, gwarp, nwarps);
        else relax_items<false, false, 4>(R, R.near[nb], nit, R.nbits[nb], limit, E, gwarp, nwarps);
      } else {
        if (heavy) relax_items<true, true, 8>(R, R.heavy[hb], hit, R.hbits[hb], limit, E, gwarp, nwarps);
        else relax_items<false, true, 8>(R, R.near[nb], nit, R.nbits[nb], limit, E, gwarp, nwarps);
        if (!grid_barrier(&c->bar, target, R.wait_ns)) return;
        classify_bits(R, limit, E, gwarp, nwarps);
      }
      E.finish();
      p = pn;
      q = qn;
      hb ^= heavy;
      record = true;
    } else {
      if (nfar == 0) break;
      if (tries == 2) {  // the second rise starts at the smallest distance left: cannot come back empty
        reason = SSSP_STUCK;
        break;
      }
      // raise the limit (past empty buckets) and take the far vertices below it
      const uint32_t rn = next3(r), rp = next3(rn), pn = next3(p), qn = next3(q);
      const uint32_t settled = limit;
      const uint32_t from = tries == 0 ? limit : st.top.dmin;
      limit = from > 0xffffffffu - R.delta ? 0xffffffffu : from + R.delta;
      ++tries;
      if (threadIdx.x == 0) st.dmin = 0xffffffffu;
      __syncthreads();
      Entries E(R, st, &c->near[pn], nb ^ 1, R.nbits[nb ^ 1], &c->heavy[qn], hb ^ 1, &c->nfar[rn]);
      uint32_t dmin = 0xffffffffu;
      const uint64_t chunks = bit_chunks(R.nwords);
      for (uint64_t ch = gwarp; ch < chunks; ch += nwarps) {
        const uint64_t num = chunk_word(ch, chunks);
        for_bits<4>(num, num < R.nwords ? R.infar[num] : 0u, [&](const bool (&valid)[4], const uint32_t (&v)[4]) {
          uint32_t d[4];
          bool below[4];
          const bool none[4] = {false, false, false, false};
#pragma unroll
          for (int k = 0; k < 4; ++k) d[k] = valid[k] ? __ldcg(R.dist + v[k]) : 0u;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            below[k] = valid[k] && d[k] < limit;
            if (below[k]) atomicAnd(R.infar + (v[k] >> 5), ~(1u << (v[k] & 31u)));
            if (valid[k] && !below[k]) {
              ++E.far;
              dmin = min(dmin, d[k]);
            }
            below[k] = below[k] && d[k] >= settled;  // else: relaxed in its bucket already
          }
          E.classify(v, below, none);
        });
      }
      dmin = __reduce_min_sync(0xffffffffu, dmin);
      if (lane == 0 && dmin != 0xffffffffu) atomicMin(&st.dmin, dmin);
      E.finish();
      if (threadIdx.x == 0 && st.dmin != 0xffffffffu) atomicMin(&c->dmin[r], st.dmin);
      if (first) {
        c->dmin[rn] = 0xffffffffu;
        c->nfar[rp] = 0;
        clear_queue(&c->near[next3(pn)]);
        clear_queue(&c->heavy[next3(qn)]);
        c->bytes += 4 * R.nwords + 4 * (uint64_t)nfar;
      }
      r = rn;
      p = pn;
      q = qn;
      hb ^= 1;
    }
    nb ^= 1;
  }
  if (reason == SSSP_DONE) {
    unsigned long long arcs[1] = {0};
    for (uint64_t v = gtid; v < R.n; v += nthreads)
      if (__ldcg(R.dist + v) != 0xffffffffu) arcs[0] += R.outdeg[v];
    __shared__ BlockSums<1> s;
    s.add(arcs, {&c->reached_arcs});
  }
  if (first) {
    c->limit = limit;
    c->p = p;
    c->q = q;
    c->r = r;
    c->nb = nb;
    c->hb = hb;
    c->reason = reason;
  }
}

// The vertices improved by a binned pass (bits of R.changed, cleared) enter the queues p, q and the far set.
__global__ void __launch_bounds__(kSsspThreads) k_sssp_classify_bits(const __grid_constant__ SsspRun R) {
  __shared__ SsspStage st;
  const uint32_t gwarp = (blockIdx.x * kSsspThreads + threadIdx.x) >> 5, nwarps = gridDim.x * (kSsspThreads / 32);
  if (threadIdx.x == 0) {
    st.verts[0] = st.verts[1] = 0;
    st.arcs[0] = st.arcs[1] = 0;
    st.far = 0;
  }
  __syncthreads();
  Entries E(R, st, &R.ctl->near[R.p], R.nb, R.nbits[R.nb], &R.ctl->heavy[R.q], R.hb, &R.ctl->nfar[R.r]);
  classify_bits(R, R.limit, E, gwarp, nwarps);
  E.finish();
}

__global__ void k_items_to_bits(const uint2* __restrict__ items, uint32_t nitems, uint32_t* __restrict__ bits) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nitems; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint2 it = items[i];
    if (it.y == 0) atomicOr(bits + (it.x >> 5), 1u << (it.x & 31u));
  }
}

int sssp_loop_launch(gre_graph g, SsspRun& R) {
  static int per_sm = 0;
  if (!per_sm) {
    int b = 0;
    GRE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_sssp_loop, kSsspThreads, 0));
    per_sm = b > 0 ? b : 1;
  }
  // a small graph's passes are barriers more than work: fewer blocks, cheaper barriers
  const int grid = (int)std::min<uint64_t>((uint64_t)num_sms() * per_sm,
                                           std::max<uint64_t>(1, std::max(R.n, R.m / 4) / kSsspThreads));
  GRE_CUDA(cudaMemsetAsync(&R.ctl->bar, 0, sizeof(GridBar), g->stream));
  void* args[] = {&R};
  GRE_CUDA(cudaLaunchCooperativeKernel((const void*)k_sssp_loop, dim3(grid), dim3(kSsspThreads), args, 0, g->stream));
  launch_count_add(1);
  return GRE_SUCCESS;
}

int sssp_classify_bits(gre_graph g, const SsspRun& R) {
  k_sssp_classify_bits<<<grid_for(R.nwords, kSsspThreads, 2), kSsspThreads, 0, g->stream>>>(R);
  GRE_LAUNCH_CHECK();
  return GRE_SUCCESS;
}

int sssp_items_to_bits(gre_graph g, const uint2* items, uint32_t nitems, uint64_t nwords, uint32_t* bits) {
  GRE_CUDA(cudaMemsetAsync(bits, 0, sizeof(uint32_t) * nwords, g->stream));
  if (nitems) k_items_to_bits<<<grid_for(nitems, 256), 256, 0, g->stream>>>(items, nitems, bits);
  GRE_LAUNCH_CHECK();
  return GRE_SUCCESS;
}

}  // namespace gre
