// Edge-induced motif plans (motif.cu).
#pragma once
#include <algorithm>

#include "clique.cuh"
#include "common.cuh"
#include "graph.cuh"

namespace xgm {

cudaError_t launch_diamond_reduce(const unsigned* epart, int64_t ne, unsigned long long* out,
                                  cudaStream_t s);

cudaError_t launch_tailed_reduce(const GView& g, const unsigned long long* vpart,
                                 unsigned long long* out, cudaStream_t s);

// out[3], out[6] += the tailed-triangle sums of launch_motif_terms.
cudaError_t launch_tailed_edges(const GView& g, int64_t ne_dag, const unsigned* epart,
                                unsigned long long* out, cudaStream_t s);

// out[0..6] += the wedge / 3-star / 3-walk / tailed-triangle / diamond / 3 x triangle sums
// (edge-induced; see motif.cu; epart null for the 3-vertex census).  next, here and below: the
// kernel may start before the one launched before it has ended (launch_next).
cudaError_t launch_motif_terms(const GView& g, const unsigned* epart, unsigned long long* out,
                               cudaStream_t s, bool next = false);
// Edge-induced tailed triangles from the seven sums.
uint64_t tailed_from_terms(const unsigned long long* terms);

// wedges[r] = wedges r-v1-v2 with v1, v2 < r (the 4-cycle plan's algorithmic bytes).
cudaError_t launch_wedge_count(const GView& g, long long* wedges, cudaStream_t s);

// 4-cycles (cycle4.cu): adds the count to *out (or per graph to o).  q is zeroed before the
// call; l holds three lists of nv vertices.
struct C4Queue {
  unsigned long long vtx, n_hub, n_mid, n_hash, h_hub, h_mid, h_hash;
};
struct C4Lists {
  int32_t* hub;
  int32_t* mid;
  int32_t* hash;
};
cudaError_t launch_cycle4(const DevGraph& g, C4Queue* q, const C4Lists& l,
                          unsigned long long* out, int num_sms, cudaStream_t s,
                          const GOut& o = GOut{}, bool next = false);
// Whether launch_cycle4 launches k_c4_cta, which depends on its first kernel.
bool cycle4_has_cta(const DevGraph& g);

// Batched graphs: per-graph diamond (slot_d) and tailed-triangle (slot_t) totals from the
// participation counters; a slot < 0 is skipped.
cudaError_t launch_part_reduce_graphs(const GView& g, const int32_t* gid,
                                      const unsigned long long* vpart, const unsigned* epart,
                                      unsigned long long* out, int stride, int slot_d, int slot_t,
                                      cudaStream_t s);

// Batched graphs: per-graph triangles, diamonds and tailed triangles from the triangles per
// edge (a slot < 0 is skipped); sums: 3 values per graph, zeroed.
cudaError_t launch_graph_terms(const GView& g, const int32_t* gid, int graphs,
                               const unsigned* epart, unsigned long long* sums,
                               unsigned long long* out, int stride, int slot_tri, int slot_d,
                               int slot_t, cudaStream_t s, bool next = false);

}  // namespace xgm
