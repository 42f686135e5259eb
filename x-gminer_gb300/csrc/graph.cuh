// Device graph storage and the GPU CSR build (csr_build.cu).
#pragma once
#include <memory>
#include <mutex>

#include "common.cuh"

namespace xgm {

// Device-resident graph.  Two id spaces:
//  - original ids: the undirected CSR exactly as loaded / built (rowptr_o, col_o);
//  - rank ids: vertices renumbered by (degree, id), so the reference's orientation
//    rule (graph.cc:247-249) reads rank(v) > rank(u).  Rows are re-sorted in rank ids;
//    the counting kernels only read this space.
struct DevGraph {
  int64_t nv = 0;
  int64_t ne = 0;          // undirected CSR entries
  int64_t ne_dag = 0;      // entries kept by the orientation (= ne / 2)
  int64_t max_deg = 0;
  int64_t max_out = 0;     // max out-degree of the oriented DAG
  int64_t n_big = 0;       // vertices of degree > kBigDeg: the top ranks (rows.cuh; 0 for
                           // batched graphs, whose ranks are sorted by degree per graph)
  int64_t n_roots[5] = {0, 0, 0, 0, 0};  // vertices of out-degree >= 2 .. 6
  // elements that a count of triangles touches: sum of C(d+(v), 2) (the owner kernel's tests)
  // and of d+(u) over edges (v, u) (the task kernel's streams); the latter over the u that the
  // owner kernel holds as bitmaps, in its count and row modes and in its participation modes
  double pairs = 0, stream = 0, stream_big[2] = {0, 0};
  int64_t* rowptr_o = nullptr;
  int32_t* col_o = nullptr;
  int32_t* rank = nullptr;   // [nv] original -> rank
  int32_t* perm = nullptr;   // [nv] rank -> original
  int64_t* rowptr = nullptr; // [nv+1] rank space
  int32_t* col = nullptr;    // [ne] rank space, sorted rows
  longlong2* dptr = nullptr; // [nv] {first out-neighbour, row end}
  int32_t* gid = nullptr;    // [nv] rank -> graph id (batched graphs only)
  // Held while an index below is looked for and built: any context, on its own stream and
  // host thread, may be the first to need it (build_once).
  std::shared_ptr<std::recursive_mutex> index_lock = std::make_shared<std::recursive_mutex>();
  // bucket index (GView), built on first use by a schedule that can pick BUCKET
  mutable int32_t* bcol = nullptr;
  mutable uint32_t* boff = nullptr;
  mutable uint16_t* bmask = nullptr;
  // set-operation programs (setbits.cu), built on first use: plan_deg is the largest
  // degree whose tasks run in the bitmap form (-1 none, 0 not built); its units {v0, part,
  // parts} by class from plan_off[class], at most plan_cap[class], their numbers in plan_un;
  // adjacency rows among N(v) for v of degree 33..1024, lut_off[v] words into lut_rows
  mutable int plan_deg = 0;
  mutable int4* plan_units = nullptr;
  mutable int64_t plan_off[3] = {0, 0, 0}, plan_cap[3] = {0, 0, 0};
  mutable unsigned long long* plan_un = nullptr;
  mutable int plan_items = 0;  // list entries a block takes to a table at a time (0: no tables)
  mutable uint32_t* lut_rows = nullptr;
  mutable int64_t* lut_off = nullptr;
  // row store offsets, row tasks by width and their numbers (rows.cu), built on first use
  // by a clique count: rn = {words, tasks of <= 8 members, <= 32, <= kRowsMid, more}; rtask
  // holds the first list from its start, the second from nv - 1 down, the third from nv on,
  // the fourth from its end down
  int64_t row_store_words = 0;
  mutable int64_t* roff = nullptr;
  mutable int32_t* rtask = nullptr;
  mutable unsigned long long* rn = nullptr;
  // out-neighbour degree sums / maxima (the learned schedule's task features), built on
  // first use by the learned schedule
  mutable int64_t* tsum = nullptr;
  mutable int32_t* tmax = nullptr;

  GView view() const {
    std::lock_guard<std::recursive_mutex> hold(*index_lock);
    return GView{col, rowptr, dptr, nv, bcol, boff, bmask, tsum, tmax};
  }
};

// Builds one of g's indexes on stream s unless it is there.  Nobody else sees it before its
// kernels have run: the lock is held until the stream is through (once per graph and index).
// Not inside stream capture, but for an index that is there.
template <class Built, class Build>
cudaError_t build_once(const DevGraph& g, cudaStream_t s, Built built, Build build) {
  std::lock_guard<std::recursive_mutex> hold(*g.index_lock);
  if (built()) return cudaSuccess;
  const cudaError_t e = build();
  return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
}

void free_graph(DevGraph& g, cudaStream_t s);

// Builds g's out-neighbour degree sums and maxima once (learned.cu); later calls return
// at once.
cudaError_t ensure_task_stats(const DevGraph& g, cudaStream_t s);

// Builds g's bucket index once (bucket.cu); later calls return at once.
cudaError_t ensure_bucket_index(const DevGraph& g, cudaStream_t s);

// Raw samples on the device -> undirected CSR in original ids (g.rowptr_o/col_o).
// flags: XGM_BUILD_* bits.  err (device) gets ERR_BOUNDS for ids outside [0, nv).
cudaError_t build_csr_from_samples(int64_t nv, const int32_t* src, const int32_t* dst,
                                   int64_t m, int flags, DevGraph& g, uint32_t* err,
                                   cudaStream_t s);

// Checks an uploaded undirected CSR: ids in range, rows strictly increasing (sorted,
// no duplicates), no self-loops, symmetric.  Sets ERR_BOUNDS in err on failure.
cudaError_t validate_csr(const DevGraph& g, uint32_t* err, cudaStream_t s);

// From g.rowptr_o/col_o: degrees, ranks, the rank-space CSR, out-neighbour pointers
// and the size statistics.  `group` (optional, [nv] original ids, values below
// num_groups) keeps vertices of one group contiguous in rank order (batched graphs)
// and fills g.gid.
cudaError_t finish_graph(DevGraph& g, const int32_t* group, int num_groups, cudaStream_t s);

// The oriented DAG in original ids (graph.cc:233-275 output), device arrays
// allocated here; caller frees.
cudaError_t dag_original(const DevGraph& g, int64_t** rowptr, int32_t** col, cudaStream_t s);

int bits_for(int64_t n);  // smallest b with 2^b >= n (>= 1)

}  // namespace xgm
