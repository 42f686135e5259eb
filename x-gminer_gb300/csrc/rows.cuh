// Triangle and clique counting from the side of the later endpoint (rows.cu).
#pragma once
#include "clique.cuh"
#include "graph.cuh"

namespace xgm {

// Vertices of degree above kBigDeg are "big": their out-list becomes a shared-memory
// bitmap and their in-neighbours' suffixes are tested against it; at most the top
// own_bits of them are treated so.  kBigDeg 48 / 64 / 96 / 112 / 128 / 192: triangles R-MAT
// s20 1.49 / 1.41 / 1.41 / 1.41 / 1.47 / 1.69 ms, triangles per edge of a 1.5 M vertex
// Chung-Lu graph 3.71 / 3.29 / 2.80 / 2.75 / 2.72 / 2.82, rows R-MAT s20 2.13 / 2.02 / 2.03 /
// 2.03 / 2.13 / 2.60.
constexpr int kBigDeg = 112;
constexpr int64_t kOwnBits = int64_t(1) << 18;
// 2^17 bits (16 KB a CTA, so that L1 keeps the lists) where hits need no rank look-ups: rows
// R-MAT s22 10.4 ms (2^16 bits 16.0, 2^18 11.7), triangles s23 20.6 ms (2^18 28.9); with them
// 2^18, triangles per edge s23 48.0 ms (2^17 49.5).
constexpr int64_t own_bits(bool part) { return part ? kOwnBits : kOwnBits / 2; }

// Largest out-degree of a graph whose edges are all joined by lanes: a bitmap unit costs its
// phases' latency however short its lists.  Barabasi-Albert, 3,312 vertices (at most 7) triangles
// 25.7 -> 20.2 us; 200,001 vertices of degree 16 (17) triangles 75 -> 54 us, 4-cliques 109 -> 91;
// R-MAT s10 ef5 (26) diamonds 42 -> 50 us, 4-cliques 37.5 -> 39.9.
constexpr int kShortLists = 24;

// Row store up to 16 GB (R-MAT scale 22: 1.9 GB); larger graphs, and a device without that
// much memory left, count with the task kernel.
constexpr int64_t kRowStoreMax = int64_t(1) << 32;  // words
constexpr int kRowsCap = 1024;  // largest out-degree whose rows are stored
constexpr int kRowsMid = 512;   // largest one of the four-warp tasks

// Row store words of a task of out-degree s (the triangular bitmap, rounded to 16 bytes).
__host__ __device__ __forceinline__ unsigned row_words(int64_t s) {
  return s < 2 || s > kRowsCap ? 0u : ((unsigned)tri_words((int)s) + 3u) & ~3u;
}

// Queue heads of one call (zeroed before it).
struct OwnHeads {
  unsigned long long big, small;        // owner kernel: units, vertices
  unsigned long long wide, team, word, group;  // row tasks by width
};

// Adds the triangle count of g to *count.
cudaError_t launch_owner_count(const DevGraph& g, OwnHeads* heads, unsigned long long* count,
                               int num_sms, cudaStream_t s);

// Adds to epart[e] the number of triangles that contain the edge of every col entry e of the
// out-lists (the edge at its lower end).  For out-degrees up to kOwnPartMaxOut (16-bit ranks).
constexpr int64_t kOwnPartMaxOut = 0xFFFF;
cudaError_t launch_owner_part(const DevGraph& g, OwnHeads* heads, unsigned* epart, int num_sms,
                              cudaStream_t s);

// Clique counts from stored rows.  Row i of vertex v's local DAG (the DAG induced on N+(v))
// holds bit j iff N+(v)[j] is an out-neighbour of N+(v)[i]; the rows of a vertex of
// out-degree 2 .. kRowsCap are kept in the triangular layout (tri_row_off) at word roff[v]
// of the row store, DevGraph::row_store_words words in all.
//  ensure_rows_index: offsets and task lists by row width, once per graph.
//  launch_owner_rows: fills the row store.
//  launch_rows_count: adds the k-cliques (k = 4 .. 7) of all stored tasks to *count.
cudaError_t ensure_rows_index(const DevGraph& g, cudaStream_t s);
// The index and a row store of g's size, grown where it has fewer words than *cap; *fits:
// whether there was room (no error where there was not: *rows is null then, and the caller
// counts with the task kernel).
cudaError_t reserve_rows(const DevGraph& g, uint32_t** rows, int64_t* cap, bool* fits,
                         cudaStream_t s);
cudaError_t launch_owner_rows(const DevGraph& g, uint32_t* rows, OwnHeads* heads, int num_sms,
                              cudaStream_t s);
//  launch_owner_multi: fills the row store and credits epart (launch_owner_part) in one pass.
cudaError_t launch_owner_multi(const DevGraph& g, uint32_t* rows, unsigned* epart,
                               OwnHeads* heads, int num_sms, cudaStream_t s);
//  (o: per-graph totals of batched graphs instead; next: it may start before the kernel launched
//  before it has ended, launch_next)
cudaError_t launch_rows_count(int k, const DevGraph& g, const uint32_t* rows, OwnHeads* heads,
                              unsigned long long* count, int num_sms, cudaStream_t s,
                              const GOut& o = GOut{}, bool next = false);

}  // namespace xgm
