// Internal definitions behind the C ABI.
#pragma once
#include <string>

#include "clique.cuh"
#include "graph.cuh"
#include "motif.cuh"
#include "rows.cuh"
#include "sched.cuh"
#include "setprog.cuh"

namespace xgm {

// Small device-side scalars of one call, zeroed by one memset and read back by one copy.
struct Scalars {
  unsigned long long count;
  unsigned long long aux;
  uint32_t err;
  uint32_t pad;
  QueueHeads q;
  C4Queue c4;
  int64_t n[8];  // task list sizes, copied back for the stats
  unsigned long long terms[7];  // motif-identity sums (launch_motif_terms)
  OwnHeads own;                 // queue heads of the owner kernels (rows.cu)
  // set-operation programs: unit heads of the bitmap form by class, then the list form's
  // entry head, split tail and split head
  unsigned long long prog[6];
};

struct Model;  // learned cost model (learned.cu)

}  // namespace xgm

struct xgm_ctx {
  int device = 0;
  int num_sms = 0;
  cudaStream_t stream = nullptr;
  std::string last_error;
  xgm::Scalars* d_sc = nullptr;
  xgm::Scalars* h_sc = nullptr;  // pinned
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
  // the call wants its times (statistics asked for): three event records cost a call 12 us
  bool timed = true;
  xgm::TaskBuf tb;
  // motif buffers (grown on demand)
  unsigned long long* vpart = nullptr;
  int64_t vpart_cap = 0;
  unsigned* epart = nullptr;
  int64_t epart_cap = 0;
  long long* wedges = nullptr;
  int64_t wedges_cap = 0;
  int32_t* c4_lists = nullptr;  // the three task lists of the 4-cycle kernels
  int64_t c4_lists_cap = 0;
  int clique_grid = 0;
  uint32_t* rows = nullptr;  // row store (rows.cu)
  int64_t rows_cap = 0;
  // set-operation programs (setprog.cu): per-warp slot scratch, split records, heads
  int32_t* prog_scratch = nullptr;
  int64_t prog_scratch_cap = 0;
  void* prog_split = nullptr;
};

struct xgm_graph {
  xgm_ctx* ctx = nullptr;
  xgm::DevGraph g;
};

struct xgm_plan {
  int pattern = 0;
  int induced = 0;     // vertex-induced motif counts (via the motif identities)
  uint64_t scale = 1;  // embeddings per match in the caller's convention (GLUMIN P2: 2)
  xgm::Prog prog;      // XGM_PATTERN_PROGRAM: the set-operation program
};

namespace xgm {

// Records timing event i of the call, and the time between two of them (0 when not asked for).
inline cudaError_t ctx_mark(xgm_ctx* ctx, int i) {
  return ctx->timed ? cudaEventRecord(ctx->ev[i], ctx->stream) : cudaSuccess;
}
inline float ctx_ms(xgm_ctx* ctx, int from, int to) {
  float ms = 0;
  if (ctx->timed) cudaEventElapsedTime(&ms, ctx->ev[from], ctx->ev[to]);
  return ms;
}

xgm_status finish_status(xgm_ctx* ctx, xgm_status st);
xgm_status check_device_flag(xgm_ctx* ctx, uint32_t flag);
xgm_status ctx_sync_scalars(xgm_ctx* ctx);

// count.cu
xgm_status count_dispatch(xgm_ctx* ctx, const DevGraph& g, int pattern, const xgm_sched& sp,
                          uint64_t* out, xgm_stats& st);
xgm_status algo_bytes_dispatch(xgm_ctx* ctx, const DevGraph& g, int pattern, uint64_t* out);
// One plan (pattern, edge- or vertex-induced), and the k = 3 / k = 4 motif census.
xgm_status count_plan(xgm_ctx* ctx, const DevGraph& g, int pattern, int induced,
                      const xgm_sched& sp, uint64_t* out, xgm_stats& st);
xgm_status count_motifs(xgm_ctx* ctx, const DevGraph& g, int k, const xgm_sched& sp,
                        uint64_t* out, xgm_stats& st);
xgm_status count_kernels(xgm_ctx* ctx, const DevGraph& g, int pattern, const xgm_sched& sp,
                         int* n_kernels);
void motif_buffers_free(xgm_ctx* ctx);
// setprog.cu
// Kernels a count of the program launches on g.
xgm_status program_kernels(xgm_ctx* ctx, const DevGraph& g, const Prog& p, int* n);
xgm_status count_program(xgm_ctx* ctx, const DevGraph& g, const Prog& p, uint64_t* out,
                         xgm_stats& st);
void program_buffers_free(xgm_ctx* ctx);
// k_feat: clique size the learned model's features describe (default k).
// hub: the launch is a clique count that runs the hub kernel (sp.hub_max applies).
xgm_status schedule_into(TaskBuf& tb, const DevGraph& g, int k, const xgm_sched& sp,
                         cudaStream_t s, int k_feat = 0, bool hub = false);
bool sched_may_bucket(const xgm_sched& sp);  // the policy can assign the BUCKET variant
// The schedule to follow: a tuned one whose table leaves the choice to the engine is the default.
xgm_sched sched_resolved(const xgm_sched& sp);
// The schedule leaves the choice of kernel to the engine: a default or learned policy with
// no threshold, hub limit or membership test asked for.
bool sched_is_open(const xgm_sched& sp);
// What the engine then chooses, by the graph (count.cu).
bool task_kernel_wins(const DevGraph& g, int k);
bool task_kernel_wins_part(const DevGraph& g);
bool task_kernel_wins_batch(const DevGraph& g, bool rows, bool part, bool five, bool tail);
int ensure_clique_grid(xgm_ctx* ctx);
int match_pattern(const xgm_plan_desc* d);  // builtin id, 0 unsupported, -1 malformed
// Builtin id for a pattern name (0 if unknown); GLUMIN ids also set induced / scale.
int pattern_from_name(const char* name, int* induced = nullptr, uint64_t* scale = nullptr);

}  // namespace xgm
