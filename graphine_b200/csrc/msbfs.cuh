// The 64-sources-per-word BFS (multi-source BFS, Then et al. 2014) as a cooperative level loop:
// gre_msbfs and the forward pass of the batched betweenness.
#pragma once
#include <vector>

#include "gre_internal.cuh"

namespace gre {

// The searches of one word.  seen[v]: the sources that have reached v; the frontier words of level d
// (the sources that reach v at distance d) are kept for every level in g->bc_fpool (keep_levels), or for
// two levels with the distances in bit planes.
struct MsBfs {
  gre_graph g = nullptr;
  unsigned long long* seen = nullptr;  // n words
  uint32_t levels = 0;                 // the deepest level with a vertex (last word)
  uint64_t frontier_vertices = 0;      // of all levels (last word)
  uint64_t scanned = 0, bytes = 0;     // running totals over the words
  std::vector<unsigned long long> found;  // (vertex, source) pairs of levels 1, 2, ..., the empty one included

  // Workspaces (slots WS_A..WS_F, WS_H; deep searches WS_G, WS_J..WS_N) and the launch shape.
  int prepare(gre_graph graph, bool keep_levels);
  // The level loop from k <= 64 sources (internal ids, device); waited for.
  int run(const uint32_t* dsrcs, uint32_t k, bool record);
  // After a run without keep_levels: out[j * n + u] for the k sources, u in the caller's order; adds
  // the out-arcs of the reached (vertex, source) pairs to *reached (device).
  int write_levels(uint32_t k, int32_t* out, unsigned long long* reached);

 private:
  bool keep_ = false;
  uint2 *q0_ = nullptr, *q1_ = nullptr;
  unsigned long long *acc_ = nullptr, *front_ = nullptr, *planes_ = nullptr;
  unsigned long long* deep_[7] = {};  // further groups of planes, taken when a search gets that deep
  uint32_t ngroups_ = 0;
  unsigned char* ctl_ = nullptr;
  int grid_ = 0;
};

}  // namespace gre
