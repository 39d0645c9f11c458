// The SSSP superstep loop in one cooperative kernel (sssp_loop.cu), for sssp.cu.
#pragma once
#include "grid_sync.cuh"
#include "item_queue.cuh"

namespace gre {

struct SsspQueue {
  unsigned int items, verts;
  unsigned long long arcs;
};

struct SsspCtl {
  GridBar bar;
  SsspQueue near[3], heavy[3];  // in use, next (empty), last
  unsigned int dmin[3];         // smallest distance a rise left in the far set (next, the one after, last)
  int nfar[3];                  // size of the far set (now, after the next rise, free)
  // state at the kernel's end (the next launch continues from it)
  unsigned int limit, p, q, r, nb, hb, reason, steps, nrec;
  unsigned int pad;
  unsigned long long relaxed, bytes, reached_arcs;
  unsigned long long big_arcs, pull_counts[2];  // the binned passes' arcs; the pulled ones' scanned arcs and hits
};

enum SsspReason { SSSP_DONE = 0, SSSP_BIG_LIGHT = 1, SSSP_BIG_HEAVY = 2, SSSP_STUCK = 3 };

struct SsspRun {
  uint64_t n, m, nwords;
  const uint64_t* __restrict__ off;
  const uint64_t* __restrict__ lend;  // end of each row's light arcs
  const uint32_t* __restrict__ col;
  const uint32_t* __restrict__ w;
  const uint32_t* __restrict__ outdeg;
  uint32_t* dist;
  uint32_t* changed;   // bits: improved by a binned pass
  uint32_t* infar;     // bits: far set
  uint32_t* nbits[2];  // bits: in the near queue, by buffer
  uint32_t* hbits[2];  // bits: in the bucket, by buffer
  uint2* near[2];
  uint2* heavy[2];
  bool all_out;        // every vertex that an arc reaches has out-arcs (symmetric)
  unsigned long long* rec;  // near vertices after every pass (null: not recorded)
  uint32_t nrec;
  SsspCtl* ctl;
  long long wait_ns;
  uint32_t src, delta;
  bool fresh;          // start from src (else continue)
  bool record_entry;   // a binned pass ran since the last launch: record its frontier
  // passes left to the binned kernels: a frontier of at least big_verts vertices, or (heavy, when
  // they pull) of at least big_arcs arcs; ~0: none
  uint64_t big_verts, big_arcs;
  uint64_t wide_arcs;  // a pass of at least so many arcs: improvements as bits, classified in a second phase
  uint32_t limit, p, q, r, nb, hb;
};

int sssp_loop_launch(gre_graph g, SsspRun& R);
// The vertices improved by a binned pass (bits of R.changed, cleared) join the near queue
// R.near[R.nb] (counter R.p), the bucket R.heavy[R.hb] (counter R.q) and the far set.
int sssp_classify_bits(gre_graph g, const SsspRun& R);
// Bits of the vertices that have items in the queue (zeroed first).
int sssp_items_to_bits(gre_graph g, const uint2* items, uint32_t nitems, uint64_t nwords, uint32_t* bits);

}  // namespace gre
