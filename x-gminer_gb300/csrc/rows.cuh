// Triangle and clique counting from the side of the later endpoint (rows.cu).
#pragma once
#include "clique.cuh"
#include "graph.cuh"

namespace xgm {

// Vertices of degree above kBigDeg are "big": their out-list becomes a shared-memory
// bitmap that the suffixes of their in-neighbours' lists are tested against.  Ranks are
// sorted by degree, so the big vertices are the top DevGraph::n_big ranks; at most
// kOwnBits of them are treated so (the bitmap of one CTA: 32 KB).
constexpr int kBigDeg = 64;
constexpr int64_t kOwnBits = int64_t(1) << 18;

// Queue heads of one call (zeroed before it).
struct OwnHeads {
  unsigned long long big, small;
};

// Adds the triangle count of g to *count.
cudaError_t launch_owner_count(const DevGraph& g, OwnHeads* heads, unsigned long long* count,
                               int num_sms, cudaStream_t s);

}  // namespace xgm
