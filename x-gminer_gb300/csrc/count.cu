// Count dispatch behind xgm_count: schedule -> persistent counting launch -> uint64.
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "api_internal.h"
#include "learned.cuh"
#include "measure.cuh"
#include "motif.cuh"
#include "prim.cuh"

namespace xgm {

namespace {

template <class T>
cudaError_t grow(T** p, int64_t* cap, int64_t n, cudaStream_t s) {
  if (*cap >= n && *p) return cudaSuccess;
  if (*p) cudaFreeAsync(*p, s);
  *p = nullptr;
  *cap = 0;
  cudaError_t e = cudaMallocAsync((void**)p, sizeof(T) * (size_t)(n > 0 ? n : 1), s);
  if (e == cudaSuccess) *cap = n;
  return e;
}

// An allocation that fails while the context keeps an earlier call's row store: once more
// without it.
template <class F>
cudaError_t with_room(xgm_ctx* ctx, F alloc) {
  cudaError_t e = alloc();
  if (e != cudaErrorMemoryAllocation || !ctx->rows) return e;
  cudaGetLastError();
  cudaFreeAsync(ctx->rows, ctx->stream);
  ctx->rows = nullptr;
  ctx->rows_cap = 0;
  e = cudaStreamSynchronize(ctx->stream);
  return e == cudaSuccess ? alloc() : e;
}

int clique_kind(int pattern) {
  switch (pattern) {
    case XGM_PATTERN_TRIANGLE: return 3;
    case XGM_PATTERN_CLIQUE4: return 4;
    case XGM_PATTERN_CLIQUE5: return 5;
    case XGM_PATTERN_CLIQUE6: return 6;
    case XGM_PATTERN_CLIQUE7: return 7;
    default: return 0;
  }
}

}  // namespace

int ensure_clique_grid(xgm_ctx* ctx) {
  if (ctx->clique_grid == 0) {
    int per_sm = 0;
    if (clique_occupancy(&per_sm) != cudaSuccess || per_sm <= 0) per_sm = 1;
    ctx->clique_grid = per_sm * ctx->num_sms;
  }
  return ctx->clique_grid;
}

bool sched_may_bucket(const xgm_sched& sp) {
  if (sp.policy == XGM_SCHED_LEARNED) return true;
  if (sp.policy == XGM_SCHED_FIXED) return sp.variant == XGM_VAR_BUCKET;
  if (sp.policy == XGM_SCHED_TUNED && sp.table) {
    for (int b = 0; b < XGM_TUNE_BUCKETS; ++b)
      if (sp.table->variant[b] == XGM_VAR_BUCKET) return true;
    return false;
  }
  return sp.bucket_max > 0;
}

namespace {

// The hub kernel counts up to 5-cliques, by default up to 4-cliques: at 5 the split
// sub-tasks win (each works on the compressed rows of N+(v0) & N+(v1); R-MAT scale 23:
// split 6.47 s, whole hubs 7.37 s; 4-cliques 1.08 s -> 0.25 s with whole hubs).
int whole_hub_max(int k, int asked) {
  if (k > 5 || asked < 0 || (asked == 0 && k > 4)) return 0;
  return asked == 0 ? kHubCap : asked;
}

}  // namespace

xgm_sched sched_resolved(const xgm_sched& sp) {
  if (sp.policy != XGM_SCHED_TUNED || !sp.table) return sp;
  for (int b = 0; b < XGM_TUNE_BUCKETS; ++b)
    if (sp.table->variant[b] != XGM_TUNE_ENGINE) return sp;
  xgm_sched r;
  std::memset(&r, 0, sizeof(r));
  r.flags = sp.flags;
  r.hub_max = sp.hub_max;
  return r;
}

bool sched_is_open(const xgm_sched& sp) {
  if (sp.policy == XGM_SCHED_LEARNED) {
    if (!sp.model) return false;  // refused by schedule_into
  } else if (sp.policy != XGM_SCHED_HEURISTIC || sp.warp_max > 0 || sp.cta_max > 0 ||
             sp.wide_max != 0 || sp.search_max > 0 || sp.bucket_max > 0 || sp.group_max > 0) {
    return false;
  }
  return sp.hub_max == 0 && !(sp.flags & XGM_SCHED_HASH_ONLY);
}

// Whether the task kernel is the faster one for an open schedule.  It streams N+(u) for every
// edge (v, u); the owner kernel tests the part of N+(v) after u, coalesced against a bitmap
// where u is of its top ranks, else a lane an edge.  In skewed graphs the streams are several
// times the tests (R-MAT s14 and up 2.5 to 5 times, Chung-Lu 3 to 6) and mostly of bitmap
// vertices, and the owner kernel wins by 2 to 20 times; in even ones (stream < 2 pairs:
// Erdos-Renyi 1.05 to 1.2, geometric 1.3, Barabasi-Albert 2.0) it depends on how long the lists
// are and whether the bitmaps cover them.  Unions of cliques (stream = pairs: every test hits)
// keep the owner kernel.  Measured, task kernel against owner / row kernels in ms:
//  triangles: Erdos-Renyi 2^20 degree 256 30.8 / 36.1; 2^20 degree 192 21.3 / 20.6
//  4-cliques: Erdos-Renyi 2^20 degree 24 1.04 / 0.63, 48 2.41 / 2.75, 64 3.64 / 4.63, 128
//    12.3 / 14.8; all bitmaps (2^17): degree 128 1.41 / 1.57, 192 2.62 / 2.21; small (2^14):
//    degree 64 0.156 / 0.147, 96 0.208 / 0.282; Barabasi-Albert 1 M degree 64 4.03 / 4.68
//  5-cliques: Erdos-Renyi 2^20 degree 24 1.02 / 0.53, 48 2.39 / 4.28; 2^17 degree 256 3.90 /
//    4.26; 20,001 vertices of degree 300 1.06 / 0.88; geometric, degree 200 118 / 32.6
//  7-cliques without bitmaps: a lane's recursion is as long as the longest of 32 rows; ring
//    lattice 2^18 degree 80 956 / 2,044, cliques of 60 452 / 685, of 100 980 / 660
bool task_kernel_wins(const DevGraph& g, int k) {
  const double T = g.stream, P = g.pairs, E = (double)g.ne_dag, Tb = g.stream_big[0];
  if (k == 3) return T < 2 * P && 2 * Tb < T && T > 80 * E;
  if (g.max_out > kRowsCap || P < 12 * E) return false;
  // (a task kernel's call is 13 launches: worth it from some work on)
  if (P * (P / E) < (k == 4 ? 6e8 : 1.2e8)) return false;
  if (k == 7 && T < 2.5 * P && 2 * Tb < T && P < 32 * E) return true;
  if (T < 1.01 * P || T >= 2 * P) return false;
  const bool covered = 5 * Tb >= 3 * T && T >= (k == 4 ? 48 : k == 5 ? 70 : 100) * E;
  return !covered;
}

// The same for triangles per edge (diamonds, tailed triangles).  A bitmap owner's ranks cost a
// scan of its bitmap, a thirty-second of the bitmap vertices above it: n^2 / 64 words in all.
// Task kernel against owner kernel in ms, by n^2 / stream: Erdos-Renyi 2^17 degree 192 (21) 2.75
// / 2.20, 2^18 degree 256 (24) 8.06 / 9.87, degree 128 (81) 3.24 / 5.80, ring lattice 2^18
// degree 160 (41) 6.87 / 8.52, Barabasi-Albert 200,001 of degree 200 (13) 8.04 / 4.90.  Without
// bitmaps, by pairs an edge: Erdos-Renyi 2^20 (14) 2.73 / 2.77, (19) 4.14 / 4.75, (29) 8.16 /
// 9.93; Barabasi-Albert 1 M degree 64 (16) 4.56 / 4.07.
bool task_kernel_wins_part(const DevGraph& g) {
  const double T = g.stream, P = g.pairs, E = (double)g.ne_dag;
  const double n = (double)std::min<int64_t>(g.n_big, own_bits(true));
  if (g.max_out > kShortLists && n * n > 22 * T) return true;
  return 2 * g.stream_big[1] < T && P >= 17 * E && T > 1.01 * P && T < 3 * P;
}

// And for a batch, whose ranks are sorted per graph: no bitmaps, a lane an edge joins both
// lists.  rows, part: the plans need the row store, triangles per edge; five, tail: there are
// 5-cliques, tailed triangles among them.  By (pairs + stream) an edge, task kernel / owner and
// row kernels in ms: triangles + 4-cliques + diamonds 1,000
// R-MAT s9 ef16 (23) 0.75 / 0.75, 200 s12 ef4 (20) 0.53 / 0.64, 200 s11 ef8 (26) 0.47 / 0.60,
// 4,096 Barabasi-Albert (8) 5.5 / 1.16; 5-cliques 250 s10 ef16 (31) 0.61 / 0.78; 4-cliques alone
// 0.45 / 0.37 there, 100 s12 ef8 (33) 0.49 / 0.51; triangles + diamonds 0.49 / 0.41 and 0.52 /
// 0.61; tailed triangles 200 s11 ef8 0.45 / 0.50; 16 s16 ef16 (141) 6.3 / 22.9.
bool task_kernel_wins_batch(const DevGraph& g, bool rows, bool part, bool five, bool tail) {
  return g.pairs + g.stream > ((rows && part) || five || tail ? 20.0 : 31.0) * (double)g.ne_dag;
}

// Fills tb from the schedule policy for a k-clique style launch (k = 3 for the
// participation and multi-pattern launches).  Builds the graph's bucket index first
// when the policy can pick BUCKET (outside stream capture: callers that capture call
// ensure_bucket_index before they begin).
xgm_status schedule_into(TaskBuf& tb, const DevGraph& g, int k, const xgm_sched& sp,
                         cudaStream_t s, int k_feat, bool hub) {
  bool order = false;
  if (sp.policy == XGM_SCHED_LEARNED) {
    if (!sp.model) {
      set_thread_error("XGM_SCHED_LEARNED needs a trained model (xgm_sched.model)");
      return XGM_ERR_INVALID;
    }
    order = sp.order_by_cost != 0;
    XGM_CUDA_TRY(ensure_bucket_index(g, s));  // the model may pick BUCKET
    XGM_CUDA_TRY(ensure_task_stats(g, s));
    XGM_CUDA_TRY(classify_learned(g, k, *sp.model, tb, order, sp.margin, s, k_feat));
  } else if (sp.policy == XGM_SCHED_TUNED) {
    if (!sp.table) {
      set_thread_error("XGM_SCHED_TUNED needs a variant table (xgm_sched.table)");
      return XGM_ERR_INVALID;
    }
    for (int b = 0; b < XGM_TUNE_BUCKETS; ++b)
      if (sp.table->variant[b] == XGM_VAR_BUCKET) {
        XGM_CUDA_TRY(ensure_bucket_index(g, s));
        break;
      }
    XGM_CUDA_TRY(classify_table(g, k - 1, *sp.table, tb, s));
  } else {
    int gmax = sp.group_max > 0 ? sp.group_max : 0;
    int bmax = sp.bucket_max > 0 ? sp.bucket_max : 0;
    int smax = sp.search_max > 0 ? sp.search_max : 0;
    int wmax = sp.warp_max > 0 ? sp.warp_max : kWarpCap;
    int dmax = sp.wide_max > 0 ? sp.wide_max : (sp.wide_max < 0 ? 0 : kWideCap);
    int cmax = sp.cta_max > 0 ? sp.cta_max : kCtaCap;
    if (sp.policy == XGM_SCHED_FIXED) {
      switch (sp.variant) {
        case XGM_VAR_WARP: wmax = kWarpCap; dmax = kWideCap; cmax = kCtaCap; break;
        case XGM_VAR_SEARCH: smax = kWarpCap; wmax = 0; dmax = kWideCap; cmax = kCtaCap; break;
        case XGM_VAR_WIDE: wmax = 0; dmax = kWideCap; cmax = kCtaCap; break;
        case XGM_VAR_CTA: wmax = 0; dmax = 0; cmax = kCtaCap; break;
        case XGM_VAR_SPLIT: wmax = 0; dmax = 0; cmax = 0; break;
        case XGM_VAR_BUCKET: bmax = kWarpCap; wmax = 0; dmax = kWideCap; cmax = kCtaCap; break;
        case XGM_VAR_GROUP: gmax = kGroupCap; wmax = kWarpCap; dmax = kWideCap; cmax = kCtaCap; break;
        default:
          set_thread_error("unknown variant for XGM_SCHED_FIXED");
          return XGM_ERR_INVALID;
      }
    } else if (sp.policy != XGM_SCHED_HEURISTIC) {
      set_thread_error("unknown schedule policy");
      return XGM_ERR_INVALID;
    }
    if (bmax > 0) XGM_CUDA_TRY(ensure_bucket_index(g, s));
    XGM_CUDA_TRY(classify_heuristic(g, k, wmax, dmax, cmax, tb, s, smax, bmax, gmax));
  }
  XGM_CUDA_TRY(build_lists(g, tb, order, s, hub ? whole_hub_max(k, sp.hub_max) : 0));
  tb.hash_only = (sp.flags & XGM_SCHED_HASH_ONLY) ? 1 : 0;
  return XGM_OK;
}

namespace {

xgm_status schedule_tasks(xgm_ctx* ctx, const DevGraph& g, int k, const xgm_sched& sp,
                          bool hub = false) {
  return schedule_into(ctx->tb, g, k, sp, ctx->stream, 0, hub);
}

// What a clique count launches: the owner kernel (triangles), the row kernels (k >= 4; the
// task kernel then only runs the vertices above their capacity), or the task kernel.
enum class CliqueRoute { kOwner, kRows, kTasks };

// Chooses the route and gets its buffers and per-graph indexes (outside stream capture).  The
// row store comes last: what else the call needs is there (nothing else fails for it), and
// without room for the store the call is the task kernel's.
xgm_status clique_route(xgm_ctx* ctx, const DevGraph& g, int k, const xgm_sched& sp,
                        CliqueRoute* route) {
  cudaStream_t s = ctx->stream;
  *route = CliqueRoute::kTasks;
  if (sched_is_open(sp) && !task_kernel_wins(g, k)) {
    if (k == 3) {
      *route = CliqueRoute::kOwner;
    } else if (g.nv > 0 && g.row_store_words <= kRowStoreMax) {
      if (g.max_out > kRowsCap)
        XGM_CUDA_TRY(with_room(ctx, [&] { return taskbuf_reserve(ctx->tb, g.nv, s); }));
      bool fits = false;
      XGM_CUDA_TRY(reserve_rows(g, &ctx->rows, &ctx->rows_cap, &fits, s));
      if (fits) *route = CliqueRoute::kRows;
    }
  }
  if (*route == CliqueRoute::kTasks)
    XGM_CUDA_TRY(with_room(ctx, [&] { return taskbuf_reserve(ctx->tb, g.nv, s); }));
  if (*route == CliqueRoute::kTasks && sched_may_bucket(sp)) XGM_CUDA_TRY(ensure_bucket_index(g, s));
  if (sp.policy == XGM_SCHED_LEARNED &&
      (*route == CliqueRoute::kTasks || (*route == CliqueRoute::kRows && g.max_out > kRowsCap)))
    XGM_CUDA_TRY(ensure_task_stats(g, s));
  return XGM_OK;
}

// Enqueues the schedule, timing event 1 and the counting kernels.
xgm_status launch_route(xgm_ctx* ctx, const DevGraph& g, int k, const xgm_sched& sp,
                        CliqueRoute route, int* launches) {
  cudaStream_t s = ctx->stream;
  Scalars* sc = ctx->d_sc;
  const bool hubs = route == CliqueRoute::kRows && g.max_out > kRowsCap;
  if (route == CliqueRoute::kTasks) {
    xgm_status r = schedule_tasks(ctx, g, k, sp, true);
    if (r != XGM_OK) return r;
  } else if (hubs) {  // only the vertices above the row capacity are tasks: all split or whole,
                      // in the order of a learned schedule's model where it asks for one
    const bool learned = sp.policy == XGM_SCHED_LEARNED, order = learned && sp.order_by_cost != 0;
    XGM_CUDA_TRY(learned ? classify_learned(g, kRowsCap + 2, *sp.model, ctx->tb, order, sp.margin, s, k)
                         : classify_heuristic(g, kRowsCap + 2, kWarpCap, kWideCap, kCtaCap, ctx->tb, s));
    XGM_CUDA_TRY(build_lists(g, ctx->tb, order, s, whole_hub_max(k, 0)));
  }
  XGM_CUDA_TRY(ctx_mark(ctx, 1));
  if (launches) *launches = 1;
  if (route == CliqueRoute::kOwner)
    XGM_CUDA_TRY(launch_owner_count(g, &sc->own, &sc->count, ctx->num_sms, s));
  if (route == CliqueRoute::kTasks || hubs) {
    XGM_CUDA_TRY(launch_clique(k, g.view(), ctx->tb.lists(false), &sc->q, &sc->count, &sc->err,
                               ensure_clique_grid(ctx), s));
    if (launches && ctx->tb.hub_max > kCtaCap) *launches = 2;  // + the hub kernel
  }
  if (route == CliqueRoute::kRows) {
    XGM_CUDA_TRY(launch_owner_rows(g, ctx->rows, &sc->own, ctx->num_sms, s));
    XGM_CUDA_TRY(launch_rows_count(k, g, ctx->rows, &sc->own, &sc->count, ctx->num_sms, s));
  }
  return XGM_OK;
}

// Triangles per edge into ctx->epart; *tasks: the task kernel ran (explicit schedules).
// Records ev[1] between the preparation and the counting.
xgm_status launch_participation(xgm_ctx* ctx, const DevGraph& g, const xgm_sched& sp, bool* tasks) {
  cudaStream_t s = ctx->stream;
  xgm_sched tri = sp;
  if (tri.policy == XGM_SCHED_LEARNED && !tri.model) tri.policy = XGM_SCHED_HEURISTIC;
  *tasks = !sched_is_open(tri) || g.max_out > kOwnPartMaxOut || task_kernel_wins_part(g);
  XGM_CUDA_TRY(with_room(ctx, [&] { return grow(&ctx->epart, &ctx->epart_cap, g.ne, s); }));
  XGM_CUDA_TRY(cudaMemsetAsync(ctx->epart, 0, sizeof(unsigned) * (g.ne > 0 ? g.ne : 1), s));
  if (!*tasks) {
    XGM_CUDA_TRY(ctx_mark(ctx, 1));
    XGM_CUDA_TRY(launch_owner_part(g, &ctx->d_sc->own, ctx->epart, ctx->num_sms, s));
    return XGM_OK;
  }
  XGM_CUDA_TRY(with_room(ctx, [&] { return taskbuf_reserve(ctx->tb, g.nv, s); }));
  xgm_status r = schedule_tasks(ctx, g, 3, tri);
  if (r != XGM_OK) return r;
  XGM_CUDA_TRY(with_room(ctx, [&] { return grow(&ctx->vpart, &ctx->vpart_cap, g.nv, s); }));
  XGM_CUDA_TRY(cudaMemsetAsync(ctx->vpart, 0, sizeof(unsigned long long) * (g.nv > 0 ? g.nv : 1), s));
  XGM_CUDA_TRY(ctx_mark(ctx, 1));
  XGM_CUDA_TRY(launch_triangle_participation(g.view(), ctx->tb.lists(false), &ctx->d_sc->q,
                                             ctx->vpart, ctx->epart, &ctx->d_sc->err,
                                             ensure_clique_grid(ctx), s));
  return XGM_OK;
}

}  // namespace

void motif_buffers_free(xgm_ctx* ctx) {
  cudaStream_t s = ctx->stream;
  void* ps[] = {ctx->vpart, ctx->epart, ctx->wedges, ctx->c4_lists, ctx->rows};
  for (void* p : ps)
    if (p) cudaFreeAsync(p, s);
}

xgm_status count_dispatch(xgm_ctx* ctx, const DevGraph& g, int pattern, const xgm_sched& sp,
                          uint64_t* out, xgm_stats& st) {
  cudaStream_t s = ctx->stream;
  XGM_CUDA_TRY(cudaSetDevice(ctx->device));
  const int k = clique_kind(pattern);
  CliqueRoute route = CliqueRoute::kTasks;
  if (k) {
    xgm_status r = clique_route(ctx, g, k, sp, &route);
    if (r != XGM_OK) return r;
  }
  XGM_CUDA_TRY(cudaMemsetAsync(ctx->d_sc, 0, sizeof(Scalars), s));
  XGM_CUDA_TRY(ctx_mark(ctx, 0));
  const GView view = g.view();
  int launches = 0;
  bool tasks = k && route == CliqueRoute::kTasks;  // the task kernel ran
  if (k) {
    xgm_status r = launch_route(ctx, g, k, sp, route, &launches);
    if (r != XGM_OK) return r;
  } else if (pattern == XGM_PATTERN_DIAMOND || pattern == XGM_PATTERN_TAILED_TRIANGLE) {
    xgm_status r = launch_participation(ctx, g, sp, &tasks);
    if (r != XGM_OK) return r;
    if (pattern == XGM_PATTERN_DIAMOND)
      XGM_CUDA_TRY(launch_diamond_reduce(ctx->epart, g.ne, &ctx->d_sc->count, s));
    else if (tasks)  // one pass over the vertices (Erdos-Renyi 2^20 degree 256 33.0 -> 31.8 ms)
      XGM_CUDA_TRY(launch_tailed_reduce(view, ctx->vpart, &ctx->d_sc->count, s));
    else
      XGM_CUDA_TRY(launch_tailed_edges(view, g.ne_dag, ctx->epart, ctx->d_sc->terms, s));
    launches = 2;
  } else if (pattern == XGM_PATTERN_CYCLE4) {
    XGM_CUDA_TRY(with_room(ctx, [&] {
      return grow(&ctx->c4_lists, &ctx->c4_lists_cap, 3 * g.nv, s);
    }));
    XGM_CUDA_TRY(ctx_mark(ctx, 1));
    const C4Lists lists{ctx->c4_lists, ctx->c4_lists + g.nv, ctx->c4_lists + 2 * g.nv};
    XGM_CUDA_TRY(launch_cycle4(g, &ctx->d_sc->c4, lists, &ctx->d_sc->count, ctx->num_sms, s));
    launches = 1;
  } else {
    set_thread_error("unknown pattern");
    return XGM_ERR_INVALID;
  }
  XGM_CUDA_TRY(ctx_mark(ctx, 2));
  if (tasks)
    XGM_CUDA_TRY(cudaMemcpyAsync(ctx->d_sc->n, ctx->tb.n, sizeof(int64_t) * 8,
                                 cudaMemcpyDeviceToDevice, s));
  xgm_status r = ctx_sync_scalars(ctx);
  if (r != XGM_OK) return r;
  const float prep = ctx_ms(ctx, 0, 1), kern = ctx_ms(ctx, 1, 2);
  st.prep_ms = prep;
  st.kernel_ms = kern;
  st.device_error = ctx->h_sc->err;
  st.launches = launches;
  st.variant_tasks[XGM_VAR_WARP] = ctx->h_sc->n[2];
  st.variant_tasks[XGM_VAR_CTA] = ctx->h_sc->n[1];
  st.variant_tasks[XGM_VAR_SPLIT] = ctx->h_sc->n[0];
  st.variant_tasks[XGM_VAR_WIDE] = ctx->h_sc->n[4];
  st.variant_tasks[XGM_VAR_SEARCH] = ctx->h_sc->n[5];
  st.variant_tasks[XGM_VAR_BUCKET] = ctx->h_sc->n[6];
  st.variant_tasks[XGM_VAR_GROUP] = ctx->h_sc->n[7];
  st.tasks = ctx->h_sc->n[1] + ctx->h_sc->n[2] + ctx->h_sc->n[3] + ctx->h_sc->n[4] +
             ctx->h_sc->n[5] + ctx->h_sc->n[6] + ctx->h_sc->n[7];
  if (k && !tasks) st.tasks = g.n_roots[k - 3];
  else if (!k && !tasks && pattern != XGM_PATTERN_CYCLE4) st.tasks = g.n_roots[0];
  r = check_device_flag(ctx, ctx->h_sc->err);
  if (r != XGM_OK) return r;
  *out = pattern == XGM_PATTERN_TAILED_TRIANGLE && !tasks ? tailed_from_terms(ctx->h_sc->terms)
                                                          : ctx->h_sc->count;
  return XGM_OK;
}

// Captures the device work of one count (schedule + counting kernels) on the context
// stream into a CUDA graph and counts its kernel nodes.
xgm_status count_kernels(xgm_ctx* ctx, const DevGraph& g, int pattern, const xgm_sched& sp,
                         int* n_kernels) {
  cudaStream_t s = ctx->stream;
  XGM_CUDA_TRY(cudaSetDevice(ctx->device));
  const int k = clique_kind(pattern);
  if (!k) {
    set_thread_error("kernel counting covers the triangle / clique plans");
    return XGM_ERR_UNSUPPORTED;
  }
  CliqueRoute route = CliqueRoute::kTasks;
  xgm_status r = clique_route(ctx, g, k, sp, &route);
  if (r != XGM_OK) return r;
  ensure_clique_grid(ctx);
  XGM_CUDA_TRY(cudaStreamSynchronize(s));
  XGM_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  ctx->timed = false;
  r = launch_route(ctx, g, k, sp, route, nullptr);
  cudaGraph_t graph = nullptr;
  cudaError_t e2 = cudaStreamEndCapture(s, &graph);
  if (r != XGM_OK) {
    if (graph) cudaGraphDestroy(graph);
    return r;
  }
  XGM_CUDA_TRY(e2);
  size_t n = 0;
  cudaError_t e = cudaGraphGetNodes(graph, nullptr, &n);
  std::vector<cudaGraphNode_t> nodes(n);
  if (e == cudaSuccess && n) e = cudaGraphGetNodes(graph, nodes.data(), &n);
  int kern = 0;
  for (size_t i = 0; e == cudaSuccess && i < n; ++i) {
    cudaGraphNodeType t;
    if (cudaGraphNodeGetType(nodes[i], &t) == cudaSuccess && t == cudaGraphNodeTypeKernel) ++kern;
  }
  cudaGraphDestroy(graph);
  XGM_CUDA_TRY(e);
  *n_kernels = kern;
  return XGM_OK;
}

xgm_status algo_bytes_dispatch(xgm_ctx* ctx, const DevGraph& g, int pattern, uint64_t* out) {
  cudaStream_t s = ctx->stream;
  XGM_CUDA_TRY(cudaSetDevice(ctx->device));
  XGM_CUDA_TRY(taskbuf_reserve(ctx->tb, g.nv, s));
  XGM_CUDA_TRY(cudaMemsetAsync(ctx->d_sc, 0, sizeof(Scalars), s));
  const GView view = g.view();
  unsigned long long* acc = &ctx->d_sc->count;
  const int k = clique_kind(pattern);
  if (k > 5) {
    set_thread_error("algorithmic bytes cover the triangle, 4/5-clique and edge-induced "
                     "motif plans");
    return XGM_ERR_UNSUPPORTED;
  }
  xgm_sched heur;
  std::memset(&heur, 0, sizeof(heur));
  if (k) {
    XGM_CUDA_TRY(launch_bytes_basic(view, 0, acc, s));
    // W terms: 4 * sum over kk-cliques of d+(top member), kk = 3 .. k-1
    for (int kk = 3; kk <= k - 1; ++kk) {
      xgm_status r = schedule_tasks(ctx, g, kk, heur);
      if (r != XGM_OK) return r;
      XGM_CUDA_TRY(cudaMemsetAsync(&ctx->d_sc->q, 0, sizeof(QueueHeads), s));
      XGM_CUDA_TRY(launch_clique_weighted(kk, view, ctx->tb.lists(false), &ctx->d_sc->q,
                                          &ctx->d_sc->aux, &ctx->d_sc->err,
                                          ensure_clique_grid(ctx), s));
    }
    xgm_status r = ctx_sync_scalars(ctx);
    if (r != XGM_OK) return r;
    *out = ctx->h_sc->count + 4ull * ctx->h_sc->aux;
    return check_device_flag(ctx, ctx->h_sc->err);
  } else if (pattern == XGM_PATTERN_DIAMOND) {
    XGM_CUDA_TRY(launch_bytes_basic(view, 1, acc, s));
  } else if (pattern == XGM_PATTERN_TAILED_TRIANGLE) {
    XGM_CUDA_TRY(launch_bytes_basic(view, 2, acc, s));
  } else if (pattern == XGM_PATTERN_CYCLE4) {
    XGM_CUDA_TRY(grow(&ctx->wedges, &ctx->wedges_cap, g.nv, s));
    XGM_CUDA_TRY(launch_bytes_basic(view, 3, acc, s));
    XGM_CUDA_TRY(launch_wedge_count(view, ctx->wedges, s));
    XGM_CUDA_TRY(launch_sum_ll(ctx->wedges, g.nv, &ctx->d_sc->aux, s));
    xgm_status r2 = ctx_sync_scalars(ctx);
    if (r2 != XGM_OK) return r2;
    *out = ctx->h_sc->count + 4ull * ctx->h_sc->aux;
    return check_device_flag(ctx, ctx->h_sc->err);
  } else {
    return XGM_ERR_INVALID;
  }
  xgm_status r = ctx_sync_scalars(ctx);
  if (r != XGM_OK) return r;
  *out = ctx->h_sc->count;
  return check_device_flag(ctx, ctx->h_sc->err);
}

namespace {

// The sums of launch_motif_terms, after one triangle-participation pass when `part`.
xgm_status motif_terms(xgm_ctx* ctx, const DevGraph& g, const xgm_sched& sp, bool part,
                       uint64_t terms[6], xgm_stats& st) {
  cudaStream_t s = ctx->stream;
  XGM_CUDA_TRY(cudaSetDevice(ctx->device));
  XGM_CUDA_TRY(cudaMemsetAsync(ctx->d_sc, 0, sizeof(Scalars), s));
  XGM_CUDA_TRY(ctx_mark(ctx, 0));
  const GView view = g.view();
  bool tasks = false;  // the task kernel ran
  if (part) {
    xgm_status r = launch_participation(ctx, g, sp, &tasks);
    if (r != XGM_OK) return r;
  } else {
    XGM_CUDA_TRY(ctx_mark(ctx, 1));
  }
  XGM_CUDA_TRY(launch_motif_terms(view, part ? ctx->epart : nullptr, ctx->d_sc->terms, s));
  XGM_CUDA_TRY(ctx_mark(ctx, 2));
  if (tasks)
    XGM_CUDA_TRY(cudaMemcpyAsync(ctx->d_sc->n, ctx->tb.n, sizeof(int64_t) * 8,
                                 cudaMemcpyDeviceToDevice, s));
  xgm_status r = ctx_sync_scalars(ctx);
  if (r != XGM_OK) return r;
  const float prep = ctx_ms(ctx, 0, 1), kern = ctx_ms(ctx, 1, 2);
  std::memset(&st, 0, sizeof(st));
  st.prep_ms = prep;
  st.kernel_ms = kern;
  st.device_error = ctx->h_sc->err;
  st.launches = part ? 2 : 1;
  if (part) st.tasks = g.n_roots[0];
  if (tasks) {
    st.variant_tasks[XGM_VAR_WARP] = ctx->h_sc->n[2];
    st.variant_tasks[XGM_VAR_CTA] = ctx->h_sc->n[1];
    st.variant_tasks[XGM_VAR_SPLIT] = ctx->h_sc->n[0];
    st.variant_tasks[XGM_VAR_WIDE] = ctx->h_sc->n[4];
    st.variant_tasks[XGM_VAR_SEARCH] = ctx->h_sc->n[5];
    st.variant_tasks[XGM_VAR_BUCKET] = ctx->h_sc->n[6];
    st.variant_tasks[XGM_VAR_GROUP] = ctx->h_sc->n[7];
    st.tasks = ctx->h_sc->n[1] + ctx->h_sc->n[2] + ctx->h_sc->n[3] + ctx->h_sc->n[4] +
               ctx->h_sc->n[5] + ctx->h_sc->n[6] + ctx->h_sc->n[7];
  }
  r = check_device_flag(ctx, ctx->h_sc->err);
  if (r != XGM_OK) return r;
  for (int i = 0; i < 6; ++i) terms[i] = ctx->h_sc->terms[i];
  terms[3] = tailed_from_terms(ctx->h_sc->terms);
  return XGM_OK;
}

void add_stats(xgm_stats& acc, const xgm_stats& x) {
  acc.kernel_ms += x.kernel_ms;
  acc.prep_ms += x.prep_ms;
  acc.tasks += x.tasks;
  for (int i = 0; i < XGM_NUM_VARIANTS; ++i) acc.variant_tasks[i] += x.variant_tasks[i];
  acc.algo_bytes += x.algo_bytes;
  acc.device_error |= x.device_error;
  acc.launches += x.launches;
}

// The pieces of the 4-vertex identities (all wrapping uint64).
struct Motif4Parts {
  uint64_t k4 = 0, c4e = 0;
  uint64_t t[6] = {0, 0, 0, 0, 0, 0};  // motif_terms with participation
};

xgm_status motif4_parts(xgm_ctx* ctx, const DevGraph& g, const xgm_sched& sp, bool need_c4,
                        Motif4Parts& m, xgm_stats& st) {
  xgm_stats x;
  // open schedules, every vertex within the row capacity: rows and triangles per edge from
  // one owner pass, all parts behind one read-back (but where the task kernel wins both)
  bool rows = false;
  if (sched_is_open(sp) && g.nv > 0 && g.max_out <= kRowsCap && g.row_store_words <= kRowStoreMax &&
      !(task_kernel_wins(g, 4) && task_kernel_wins_part(g))) {
    cudaStream_t s = ctx->stream;
    XGM_CUDA_TRY(cudaSetDevice(ctx->device));
    XGM_CUDA_TRY(with_room(ctx, [&] {
      cudaError_t e = grow(&ctx->epart, &ctx->epart_cap, g.ne, s);
      if (e == cudaSuccess && need_c4) e = grow(&ctx->c4_lists, &ctx->c4_lists_cap, 3 * g.nv, s);
      return e;
    }));
    XGM_CUDA_TRY(reserve_rows(g, &ctx->rows, &ctx->rows_cap, &rows, s));
  }
  if (rows) {
    cudaStream_t s = ctx->stream;
    Scalars* sc = ctx->d_sc;
    XGM_CUDA_TRY(cudaMemsetAsync(sc, 0, sizeof(Scalars), s));
    XGM_CUDA_TRY(ctx_mark(ctx, 0));
    XGM_CUDA_TRY(cudaMemsetAsync(ctx->epart, 0, sizeof(unsigned) * (g.ne > 0 ? g.ne : 1), s));
    XGM_CUDA_TRY(ctx_mark(ctx, 1));
    XGM_CUDA_TRY(launch_owner_multi(g, ctx->rows, ctx->epart, &sc->own, ctx->num_sms, s));
    // the 4-cycles depend on nothing before them, the others on the owner kernel alone: a
    // kernel that starts in stream order after one that waits for it is past its end
    bool next = false;
    if (need_c4) {
      const C4Lists lists{ctx->c4_lists, ctx->c4_lists + g.nv, ctx->c4_lists + 2 * g.nv};
      XGM_CUDA_TRY(launch_cycle4(g, &sc->c4, lists, &sc->aux, ctx->num_sms, s, GOut{}, true));
      next = cycle4_has_cta(g);
    }
    XGM_CUDA_TRY(launch_rows_count(4, g, ctx->rows, &sc->own, &sc->count, ctx->num_sms, s, GOut{},
                                   next));
    XGM_CUDA_TRY(launch_motif_terms(g.view(), ctx->epart, sc->terms, s, true));
    XGM_CUDA_TRY(ctx_mark(ctx, 2));
    xgm_status q = ctx_sync_scalars(ctx);
    if (q != XGM_OK) return q;
    st.prep_ms = ctx_ms(ctx, 0, 1);
    st.kernel_ms = ctx_ms(ctx, 1, 2);
    st.launches = need_c4 ? 4 : 3;
    st.tasks = g.n_roots[0] + g.n_roots[1];
    st.device_error = ctx->h_sc->err;
    for (int i = 0; i < 6; ++i) m.t[i] = ctx->h_sc->terms[i];
    m.t[3] = tailed_from_terms(ctx->h_sc->terms);
    m.k4 = ctx->h_sc->count;
    m.c4e = ctx->h_sc->aux;
    return check_device_flag(ctx, ctx->h_sc->err);
  }
  xgm_status r = motif_terms(ctx, g, sp, true, m.t, x);
  if (r != XGM_OK) return r;
  add_stats(st, x);
  std::memset(&x, 0, sizeof(x));
  r = count_dispatch(ctx, g, XGM_PATTERN_CLIQUE4, sp, &m.k4, x);
  if (r != XGM_OK) return r;
  add_stats(st, x);
  if (need_c4) {
    std::memset(&x, 0, sizeof(x));
    r = count_dispatch(ctx, g, XGM_PATTERN_CYCLE4, sp, &m.c4e, x);
    if (r != XGM_OK) return r;
    add_stats(st, x);
  }
  return XGM_OK;
}

// Vertex-induced 4-vertex motifs from the edge-induced counts.  Every edge-induced
// embedding sits in exactly one induced connected 4-vertex subgraph; per 4-set:
//                3-star 4-path tailed 4-cycle diamond K4
//   3-stars        1      0      1      0       2     4      (sum_v C(d_v, 3))
//   4-paths        0      1      2      4       6    12      (3-walks - 3 x triangles)
//   tailed         .      .      1      0       4    12
//   4-cycles       .      .      0      1       1     3
//   diamonds       .      .      0      0       1     6
// The triangular system is solved from the bottom up.  The reference's formula motif
// counter (codes/GraphMiner/src/motif/omp_formula.cc:38-48 with
// cpu_kernels/automine_formula.h:20-57) derives the same six numbers from
// per-edge local counts plus enumerated 4-cycles and 4-cliques; its output order is
// [3-star, 4-path, tailed triangle, 4-cycle, diamond, 4-clique].
void motif4_solve(const Motif4Parts& m, uint64_t out[6]) {
  const uint64_t k4 = m.k4, dia_e = m.t[4], tail_e = m.t[3];
  const uint64_t star_e = m.t[1], path_e = m.t[2] - m.t[5];
  const uint64_t dia = dia_e - 6 * k4;
  const uint64_t c4 = m.c4e + 3 * k4 - dia_e;
  const uint64_t tail = tail_e - 4 * dia - 12 * k4;
  out[0] = star_e - tail - 2 * dia - 4 * k4;
  out[1] = path_e - 2 * tail - 4 * c4 - 6 * dia - 12 * k4;
  out[2] = tail;
  out[3] = c4;
  out[4] = dia;
  out[5] = k4;
}

}  // namespace

// Reference interface: MotifSolver(Graph&, int k, std::vector<uint64_t>& total, ...)
// (codes/GraphMiner/src/motif/omp_formula.cc:8, main.cc:8-31): k = 3 gives
// [wedges, triangles], k = 4 the six counts of motif4_solve, all vertex-induced.
xgm_status count_motifs(xgm_ctx* ctx, const DevGraph& g, int k, const xgm_sched& sp,
                        uint64_t* out, xgm_stats& st) {
  std::memset(&st, 0, sizeof(st));
  if (k == 3) {
    uint64_t t[6], tri = 0;
    xgm_stats x;
    if (sched_is_open(sp) && !task_kernel_wins(g, 3)) {  // both parts behind one read-back
      cudaStream_t s = ctx->stream;
      Scalars* sc = ctx->d_sc;
      XGM_CUDA_TRY(cudaSetDevice(ctx->device));
      XGM_CUDA_TRY(cudaMemsetAsync(sc, 0, sizeof(Scalars), s));
      XGM_CUDA_TRY(ctx_mark(ctx, 0));
      XGM_CUDA_TRY(ctx_mark(ctx, 1));
      XGM_CUDA_TRY(launch_motif_terms(g.view(), nullptr, sc->terms, s));
      XGM_CUDA_TRY(launch_owner_count(g, &sc->own, &sc->count, ctx->num_sms, s));
      XGM_CUDA_TRY(ctx_mark(ctx, 2));
      xgm_status q = ctx_sync_scalars(ctx);
      if (q != XGM_OK) return q;
      st.prep_ms = ctx_ms(ctx, 0, 1);
      st.kernel_ms = ctx_ms(ctx, 1, 2);
      st.launches = 2;
      st.tasks = g.n_roots[0];
      out[1] = ctx->h_sc->count;
      out[0] = ctx->h_sc->terms[0] - 3 * out[1];
      return XGM_OK;
    }
    xgm_status r = motif_terms(ctx, g, sp, false, t, x);
    if (r != XGM_OK) return r;
    add_stats(st, x);
    std::memset(&x, 0, sizeof(x));
    r = count_dispatch(ctx, g, XGM_PATTERN_TRIANGLE, sp, &tri, x);
    if (r != XGM_OK) return r;
    add_stats(st, x);
    out[0] = t[0] - 3 * tri;
    out[1] = tri;
    return XGM_OK;
  }
  if (k != 4) {
    set_thread_error("motif counting covers k = 3 and k = 4");
    return XGM_ERR_UNSUPPORTED;
  }
  Motif4Parts m;
  xgm_status r = motif4_parts(ctx, g, sp, true, m, st);
  if (r != XGM_OK) return r;
  motif4_solve(m, out);
  return XGM_OK;
}

// One plan: the clique and edge-induced motif kernels directly; wedges, 3-stars,
// 4-paths and every vertex-induced motif through the motif sums and identities.
xgm_status count_plan(xgm_ctx* ctx, const DevGraph& g, int pattern, int induced,
                      const xgm_sched& sp, uint64_t* out, xgm_stats& st) {
  const bool clique = pattern == XGM_PATTERN_TRIANGLE || pattern == XGM_PATTERN_CLIQUE4 ||
                      pattern == XGM_PATTERN_CLIQUE5 || pattern == XGM_PATTERN_CLIQUE6 ||
                      pattern == XGM_PATTERN_CLIQUE7;
  const bool kernel = pattern == XGM_PATTERN_DIAMOND || pattern == XGM_PATTERN_CYCLE4 ||
                      pattern == XGM_PATTERN_TAILED_TRIANGLE;
  if (clique || (kernel && !induced)) return count_dispatch(ctx, g, pattern, sp, out, st);
  std::memset(&st, 0, sizeof(st));
  if (pattern == XGM_PATTERN_WEDGE) {
    if (induced) {
      uint64_t m3[2];
      xgm_status r = count_motifs(ctx, g, 3, sp, m3, st);
      if (r == XGM_OK) *out = m3[0];
      return r;
    }
    uint64_t t[6];
    xgm_status r = motif_terms(ctx, g, sp, false, t, st);
    if (r == XGM_OK) *out = t[0];
    return r;
  }
  if (pattern == XGM_PATTERN_STAR3 && !induced) {
    uint64_t t[6];
    xgm_status r = motif_terms(ctx, g, sp, false, t, st);
    if (r == XGM_OK) *out = t[1];
    return r;
  }
  if (pattern == XGM_PATTERN_PATH4 && !induced) {
    uint64_t t[6];
    xgm_status r = motif_terms(ctx, g, sp, true, t, st);
    if (r == XGM_OK) *out = t[2] - t[5];
    return r;
  }
  // vertex-induced 4-vertex motifs; the 4-cycle kernel only where the identity needs it
  const bool need_c4 = pattern == XGM_PATTERN_CYCLE4 || pattern == XGM_PATTERN_PATH4;
  Motif4Parts m;
  xgm_status r = motif4_parts(ctx, g, sp, need_c4, m, st);
  if (r != XGM_OK) return r;
  uint64_t v[6];
  motif4_solve(m, v);
  switch (pattern) {
    case XGM_PATTERN_STAR3: *out = v[0]; break;
    case XGM_PATTERN_PATH4: *out = v[1]; break;
    case XGM_PATTERN_TAILED_TRIANGLE: *out = v[2]; break;
    case XGM_PATTERN_CYCLE4: *out = v[3]; break;
    case XGM_PATTERN_DIAMOND: *out = v[4]; break;
    default: set_thread_error("unknown pattern"); return XGM_ERR_INVALID;
  }
  return XGM_OK;
}

// Pattern matching of a small adjacency matrix against the builtins (edge-induced).
int match_pattern(const xgm_plan_desc* d) {
  const int n = d->num_vertices;
  if (n < 3 || n > 8) return -1;
  int deg[8] = {0}, m = 0;
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) {
      const bool a = d->adj[i][j] != 0, b = d->adj[j][i] != 0;
      if (a != b || (i == j && a)) return -1;
      if (a && i < j) ++m, ++deg[i], ++deg[j];
    }
  int sorted[8];
  for (int i = 0; i < n; ++i) sorted[i] = deg[i];
  for (int i = 0; i < n; ++i)
    for (int j = i + 1; j < n; ++j)
      if (sorted[j] < sorted[i]) { int t = sorted[i]; sorted[i] = sorted[j]; sorted[j] = t; }
  if (n == 3 && m == 3) return XGM_PATTERN_TRIANGLE;
  if (n == 4 && m == 6) return XGM_PATTERN_CLIQUE4;
  if (n == 5 && m == 10) return XGM_PATTERN_CLIQUE5;
  if (n == 6 && m == 15) return XGM_PATTERN_CLIQUE6;
  if (n == 7 && m == 21) return XGM_PATTERN_CLIQUE7;
  if (n == 4 && m == 5) return XGM_PATTERN_DIAMOND;  // K4 minus one edge
  if (n == 4 && m == 4 && sorted[0] == 2 && sorted[3] == 2) return XGM_PATTERN_CYCLE4;
  if (n == 4 && m == 4 && sorted[0] == 1 && sorted[1] == 2 && sorted[2] == 2 && sorted[3] == 3)
    return XGM_PATTERN_TAILED_TRIANGLE;
  if (n == 3 && m == 2 && sorted[0] == 1) return XGM_PATTERN_WEDGE;
  if (n == 4 && m == 3 && sorted[0] == 1 && sorted[2] == 1 && sorted[3] == 3) return XGM_PATTERN_STAR3;
  if (n == 4 && m == 3 && sorted[0] == 1 && sorted[1] == 1 && sorted[2] == 2 && sorted[3] == 2)
    return XGM_PATTERN_PATH4;
  return 0;
}

int pattern_from_name(const char* name, int* induced, uint64_t* scale) {
  const std::string s(name);
  if (induced) *induced = 0;
  if (scale) *scale = 1;
  if (s == "triangle" || s == "3-clique" || s == "clique3" || s == "tc" || s == "3-triangle")
    return XGM_PATTERN_TRIANGLE;
  if (s == "4-clique" || s == "clique4" || s == "k4") return XGM_PATTERN_CLIQUE4;
  if (s == "5-clique" || s == "clique5" || s == "k5") return XGM_PATTERN_CLIQUE5;
  if (s == "6-clique" || s == "clique6" || s == "k6") return XGM_PATTERN_CLIQUE6;
  if (s == "7-clique" || s == "clique7" || s == "k7") return XGM_PATTERN_CLIQUE7;
  if (s == "diamond" || s == "4-diamond") return XGM_PATTERN_DIAMOND;
  if (s == "rectangle" || s == "4-cycle" || s == "cycle4") return XGM_PATTERN_CYCLE4;
  if (s == "tailedtriangle" || s == "tailed-triangle" || s == "tailed_triangle" ||
      s == "4-tailed-triangle")
    return XGM_PATTERN_TAILED_TRIANGLE;
  if (s == "wedge" || s == "3-path") return XGM_PATTERN_WEDGE;
  if (s == "4-star" || s == "3-star") return XGM_PATTERN_STAR3;
  if (s == "4-path") return XGM_PATTERN_PATH4;
  // GLUMIN pattern ids (G2Miner/main.cc:13-60): vertex-induced.  P1 counts each star
  // once (GM_kernels/P1-GM.yml.cuh: leaves ordered v3 < v2 < v1); P2 walks every
  // directed edge as the diamond's shared edge (init_edgelist without symmetry
  // breaking, gpu_GM_LUT.cu:89 / common/graph.cc:296-330; P2-GM.yml.cuh), so each diamond
  // counts twice; P3 counts each tailed triangle once (v2 < v1 around the anchor v0).
  int p = 0;
  uint64_t k = 1;
  if (s == "P1") p = XGM_PATTERN_STAR3;
  else if (s == "P2") p = XGM_PATTERN_DIAMOND, k = 2;
  else if (s == "P3") p = XGM_PATTERN_TAILED_TRIANGLE;
  else if (s == "P4") p = XGM_PATTERN_CLIQUE4;
  else if (s == "P5") p = XGM_PATTERN_CLIQUE5;
  else if (s == "P23") p = XGM_PATTERN_CLIQUE6;
  else if (s == "P24") p = XGM_PATTERN_CLIQUE7;
  if (p) {
    if (induced) *induced = 1;
    if (scale) *scale = k;
  }
  return p;
}

}  // namespace xgm
