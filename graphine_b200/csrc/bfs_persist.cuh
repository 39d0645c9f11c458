// The persistent direction-optimising BFS (bfs_persist.cu) for its callers.
#pragma once
#include <memory>

#include "gre_internal.cuh"

namespace gre {

struct BfsRun;

// Searches of one call over one graph, enqueued one after the other on the graph's stream and
// waited for once (uses slots WS_A..WS_D).
struct BfsPlan {
  gre_graph g = nullptr;
  uint32_t searches = 0;
  int grid = 0;
  void* ctl = nullptr;
  unsigned long long* rec = nullptr;
  std::unique_ptr<BfsRun> run;
  BfsPlan();
  ~BfsPlan();
  // caller_order: levels indexed by caller id (else by internal id); record: keep the vertices of
  // every level (one search)
  int prepare(gre_graph graph, uint32_t nsearch, bool caller_order, bool record);
  // from the device roots, or (droots null, nroots 1) from `root`
  int search(uint32_t i, const uint32_t* droots, uint32_t nroots, uint32_t root, int32_t* level);
  // waits; adds the statistics, and the out-arcs of all vertices reached
  int collect(gre_stats* st, uint64_t* reached_arcs);
};

}  // namespace gre
