// Interpreter for set-operation programs (setprog.cuh) on the undirected CSR in
// original ids.  Tasks are the directed CSR entries (v0, v1), as GLUMIN's
// edge-parallel kernels walk the full edge list (G2Miner/gpu_GM_LUT.cu:78-95,
// GM_kernels/P*-GM.yml.cuh: `for eid ... g.get_src(eid), g.get_dst(eid)`).  Two forms:
//
// - List form (k_setprog, any degree): one warp per task.  A set operation streams
//   its first list through the warp (coalesced, 32 elements a step), tests each
//   element against the second list by binary search, and compacts the survivors with
//   a ballot into the warp's slot; a bound stops the stream at the first element at
//   or above it (the lists are sorted).  The last vertex is never enumerated: the
//   final count runs flat over every (v_{k-2}, x) pair, or, when the counted operand
//   is long, searches the short neighbour lists of the candidates in it.
// - Bitmap form for d(v0) <= 1024 (setbits.cu), for programs whose operands live in
//   N(v0) (prog_lut); others run in the list form throughout, and so do a v0 of more
//   neighbours and a graph whose stored rows do not fit.
//
// Warps of the list form claim chunks of entries from an atomic head (the row of a
// chunk's first entry by binary search over rowptr, then entry by entry).  A task whose
// estimated work passes kSplitWork queues its v2 candidates as split records of about
// kSplitWork each, run by a second k_setprog launch (each record recomputes the level-0
// slots, a few percent of its work).  A graph without a task for it launches neither.
//
// List slots live in a per-warp global scratch area ((slot count + 1) x max degree
// ints), which stays in L1/L2: a slot is written once per level and read by every
// later step.
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>

#include "api_internal.h"
#include "graph.cuh"
#include "prim.cuh"
#include "setprog.cuh"

namespace xgm {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kChunk = 8;       // CSR entries claimed per queue step
// Work of a task in lane-steps (one binary search of one lane): a task above kSplitWork
// queues its v2 candidates as records of about kSplitWork each (about a millisecond
// of one warp).
constexpr long long kSplitWork = 4096;
constexpr int64_t kSplitCap = int64_t(1) << 22;  // records (64 MB)

struct SplitRec {
  int32_t e_lo, e_hi;  // CSR entry
  int32_t lo, hi;      // v2 candidate range
};

struct ProgArgs {
  const int64_t* rowptr;
  const int32_t* col;
  int64_t nv, ne;
  int32_t* scratch;
  int64_t slot_cap;   // ints per slot
  int nslots;
  unsigned long long* heads;  // [0] entry head, [1] split tail, [2] split head
  SplitRec* split;
  int64_t split_cap;
  unsigned long long* total;
  int split_mode;
  int bits_deg;  // v0 of at most this degree run in the bitmap form
};

struct WarpState {
  int v[kProgMaxK];
  int vl[kProgMaxK];
  long long vb[kProgMaxK];
  int slen[kProgMaxSlots];
};

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Binary search for x in the sorted list b[0, len).
__device__ __forceinline__ bool member(const int32_t* b, int len, int x) {
  int lo = 0, n = len;
  while (n > 0) {
    const int h = n >> 1;
    if (__ldg(b + lo + h) < x) {
      lo += h + 1;
      n -= h + 1;
    } else {
      n = h;
    }
  }
  return lo < len && __ldg(b + lo) == x;
}

struct Operand {
  const int32_t* p;
  int n;
};

__device__ __forceinline__ Operand operand(const WarpState& w, int code, const ProgArgs& a,
                                           const int32_t* slots) {
  if (code >= kOpList) {
    const int j = code - kOpList;
    return Operand{a.col + w.vb[j], w.vl[j]};
  }
  return Operand{slots + (int64_t)code * a.slot_cap, w.slen[code]};
}

// The bound and exclusion masks of a program for K vertices name only v0..v_{K-2}
// (prog_check), so the loops over matched vertices run over K - 1 entries.
template <int K>
__device__ __forceinline__ int bound_of(const WarpState& w, unsigned mask) {
  int b = INT_MAX;
#pragma unroll
  for (int j = 0; j < K - 1; ++j)
    if ((mask >> j) & 1u) b = min(b, w.v[j]);
  return b;
}

template <int K>
struct Excl {
  int e[K - 1];
  __device__ __forceinline__ bool hit(int x) const {
    bool h = false;
#pragma unroll
    for (int j = 0; j < K - 1; ++j) h |= x == e[j];
    return h;
  }
};

template <int K>
__device__ __forceinline__ Excl<K> excl_of(const WarpState& w, unsigned mask) {
  Excl<K> r;
#pragma unroll
  for (int j = 0; j < K - 1; ++j) r.e[j] = ((mask >> j) & 1u) ? w.v[j] : -1;
  return r;
}

__device__ __forceinline__ void set_vertex(WarpState& w, int j, int x, const ProgArgs& a, int lane) {
  if (lane == 0) {
    const long long b = a.rowptr[x];
    w.v[j] = x;
    w.vb[j] = b;
    w.vl[j] = (int)(a.rowptr[x + 1] - b);
  }
  __syncwarp();
}

// out slot <- op(a, b); warp-wide.
template <int K>
__device__ void run_op(const ProgOp& o, WarpState& w, const ProgArgs& a, int32_t* slots, int lane) {
  const Operand A = operand(w, o.a, a, slots);
  const Operand B = o.kind == OP_FILTER ? Operand{nullptr, 0} : operand(w, o.b, a, slots);
  const int bnd = bound_of<K>(w, o.bound);
  const Excl<K> ex = excl_of<K>(w, o.excl);
  int32_t* out = slots + (int64_t)o.out * a.slot_cap;
  int written = 0;
  for (int base = 0; base < A.n; base += 32) {
    const int i = base + lane;
    const bool in = i < A.n;
    const int x = in ? A.p[i] : INT_MAX;
    const bool below = in && x < bnd;
    bool keep = below && !ex.hit(x);
    if (keep && o.kind != OP_FILTER) keep = member(B.p, B.n, x) == (o.kind == OP_INTERSECT);
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (keep) out[written + __popc(m & lanemask_lt())] = x;
    written += __popc(m);
    if (__ballot_sync(0xffffffffu, in && !below)) break;
  }
  if (lane == 0) w.slen[o.out] = written;
  __syncwarp();
}

// |op(a, b)| for the counted vertex; per-lane partial.
template <int K>
__device__ unsigned long long count_op(const ProgOp& o, const WarpState& w, const ProgArgs& a,
                                       const int32_t* slots, int lane) {
  const Operand A = operand(w, o.a, a, slots);
  const Operand B = o.kind == OP_FILTER ? Operand{nullptr, 0} : operand(w, o.b, a, slots);
  const int bnd = bound_of<K>(w, o.bound);
  const Excl<K> ex = excl_of<K>(w, o.excl);
  unsigned long long c = 0;
  for (int base = 0; base < A.n; base += 32) {
    const int i = base + lane;
    const bool in = i < A.n;
    const int x = in ? A.p[i] : INT_MAX;
    const bool below = in && x < bnd;
    bool keep = below && !ex.hit(x);
    if (keep && o.kind != OP_FILTER) keep = member(B.p, B.n, x) == (o.kind == OP_INTERSECT);
    c += keep ? 1 : 0;
    if (__ballot_sync(0xffffffffu, in && !below)) break;
  }
  return c;
}

// First index of sorted A[0, n) at or above x.
__device__ __forceinline__ int lower_index(const int32_t* A, int n, int x) {
  int lo = 0;
  while (n > 0) {
    const int h = n >> 1;
    if (A[lo + h] < x) {
      lo += h + 1;
      n -= h + 1;
    } else {
      n = h;
    }
  }
  return lo;
}

// One lane's count for a candidate u whose list N(u) (du entries from rb) is short
// next to A: each y in N(u) is searched in A instead of each x of A in N(u).  The
// difference count is the number of A's elements that pass the bound and the
// exclusions, minus the intersection.
template <int K>
__device__ unsigned long long count_short(const Operand& A, int u, long long rb, int du, int sbnd,
                                          bool ubnd, const Excl<K>& ex, bool uex, bool want,
                                          const int32_t* col) {
  const int bnd = ubnd ? min(sbnd, u) : sbnd;
  const int m = lower_index(A.p, A.n, bnd);
  unsigned long long inter = 0;
  for (int i = 0; i < du; ++i) {
    const int y = col[rb + i];
    if (y >= bnd) break;
    if (ex.hit(y)) continue;  // y == u cannot occur: no self-loops
    inter += member(A.p, m, y) ? 1 : 0;
  }
  if (want) return inter;
  long long pass = m;
#pragma unroll
  for (int j = 0; j < K - 1; ++j) {
    bool dup = false;
#pragma unroll
    for (int i = 0; i < j; ++i) dup |= ex.e[i] == ex.e[j];
    if (ex.e[j] >= 0 && !dup && member(A.p, m, ex.e[j])) --pass;
  }
  if (uex && !ex.hit(u) && member(A.p, m, u)) --pass;
  return (unsigned long long)(pass - (long long)inter);
}

// Final count merged with the loop over v_iv (iv = k-2) running over C[lo, hi):
// one item per (candidate u, element x of the counted operand).  When the second
// operand is N(u) and A is long, candidates with short lists are counted one per lane
// by count_short, and only the others (gathered into `big`) take the item walk.
template <int K>
__device__ unsigned long long count_flat(const ProgOp& o, const WarpState& w, int iv, Operand C,
                                         int lo, int hi, const ProgArgs& a, const int32_t* slots,
                                         int32_t* big, int lane) {
  const Operand A = operand(w, o.a, a, slots);
  const unsigned ivbit = 1u << iv;
  const int sbnd = bound_of<K>(w, o.bound & ~ivbit);
  const bool ubnd = (o.bound & ivbit) != 0;
  const Excl<K> ex = excl_of<K>(w, o.excl & ~ivbit);
  const bool uex = (o.excl & ivbit) != 0;
  const bool filter = o.kind == OP_FILTER;
  const bool b_u = !filter && o.b == kOpList + iv;
  const Operand Bf = (filter || b_u) ? Operand{nullptr, 0} : operand(w, o.b, a, slots);
  const bool want = o.kind == OP_INTERSECT;
  int n = hi - lo;
  unsigned long long c = 0;
  if (A.n == 0 || n <= 0) return 0;
  if (b_u && A.n >= 64) {
    int nbig = 0;
    for (int base = 0; base < n; base += 32) {
      const int ci = base + lane;
      const bool in = ci < n;
      const int u = in ? C.p[lo + ci] : 0;
      const long long rb = in ? a.rowptr[u] : 0;
      const int du = in ? (int)(a.rowptr[u + 1] - rb) : 0;
      const bool small = in && 4 * du <= A.n;
      if (small) c += count_short<K>(A, u, rb, du, sbnd, ubnd, ex, uex, want, a.col);
      const unsigned mb = __ballot_sync(0xffffffffu, in && !small);
      if (in && !small) big[nbig + __popc(mb & lanemask_lt())] = u;
      nbig += __popc(mb);
    }
    __syncwarp();
    C = Operand{big, nbig};
    lo = 0;
    n = nbig;
    if (n == 0) return c;
  }
  int ci = lane / A.n, ai = lane - ci * A.n;
  while (ci < n) {
    const int u = C.p[lo + ci];
    const int x = A.p[ai];
    const int bnd = ubnd ? min(sbnd, u) : sbnd;
    if (x < bnd && !ex.hit(x) && !(uex && x == u)) {
      if (filter) {
        ++c;
      } else if (b_u) {
        const long long rb = a.rowptr[u];
        c += member(a.col + rb, (int)(a.rowptr[u + 1] - rb), x) == want ? 1 : 0;
      } else {
        c += member(Bf.p, Bf.n, x) == want ? 1 : 0;
      }
    }
    ai += 32;
    while (ai >= A.n) {
      ai -= A.n;
      ++ci;
    }
  }
  return c;
}

// Operands whose lengths bound the work of one v2 step: the level-0 slots (bit = slot)
// and the lists N(v0), N(v1) (bits 16, 17) that every operand read after level 0
// descends from.
__device__ unsigned step_roots(const Prog& p) {
  bool deep[kProgMaxSlots] = {};
  int8_t from[kProgMaxSlots] = {};
  for (int l = 1; l < kProgLevels; ++l)
    for (int i = 0; i < p.nops[l]; ++i) {
      deep[p.ops[l][i].out] = true;
      from[p.ops[l][i].out] = p.ops[l][i].a;
    }
  unsigned m = 0;
  auto add = [&](int c) {
    while (c < kOpList && deep[c]) c = from[c];  // operands are defined before use
    if (c < kOpList) m |= 1u << c;
    else if (c - kOpList <= 1) m |= 1u << (16 + c - kOpList);
  };
  for (int l = 1; l < kProgLevels; ++l)
    for (int i = 0; i < p.nops[l]; ++i) add(p.ops[l][i].a);
  add(p.fin.a);
  if (p.k >= 5) add(p.cand[3]);
  if (p.k == 6) add(p.cand[4]);
  return m;
}

template <int K>
__device__ unsigned long long run_task(const Prog& p, unsigned roots, WarpState& w,
                                       const ProgArgs& a, int32_t* slots, int v0, int v1,
                                       long long e, int lo, int hi, bool may_split, int lane) {
  int32_t* big = slots + (int64_t)a.nslots * a.slot_cap;  // count_flat's long-list candidates
  set_vertex(w, 0, v0, a, lane);
  set_vertex(w, 1, v1, a, lane);
  for (int i = 0; i < p.nops[0]; ++i) run_op<K>(p.ops[0][i], w, a, slots, lane);
  if constexpr (K == 3) return count_op<K>(p.fin, w, a, slots, lane);
  const Operand C2 = operand(w, p.cand[2], a, slots);
  if (hi < 0 || hi > C2.n) hi = C2.n;
  if (may_split && C2.n > 1) {
    // lane-steps of one v2 step: the streams of the level-1 operations, then the
    // final count over (v3, x) pairs (5 vertices), over x (4 vertices), or a v3 loop
    // of such counts (6 vertices)
    int len = 0;
    for (int j = 0; j < kProgMaxSlots; ++j)
      if ((roots >> j) & 1u) len = max(len, w.slen[j]);
    if ((roots >> 16) & 1u) len = max(len, w.vl[0]);
    if ((roots >> 17) & 1u) len = max(len, w.vl[1]);
    const long long step = 1 + len / 32 + (K >= 5 ? (long long)len * len / 64 : 0) *
                                                (K == 6 ? 1 + len / 32 : 1);
    if ((long long)C2.n * step > kSplitWork) {
      // every candidate goes to the records, so a warp that claims a chunk of heavy
      // tasks only builds their level-0 slots
      const int per = (int)max(1LL, min((long long)C2.n, kSplitWork / step));
      const int nrec = (C2.n + per - 1) / per;
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(a.heads + 1, (unsigned long long)nrec);
      base = __shfl_sync(0xffffffffu, base, 0);
      const bool fits = base + nrec <= (unsigned long long)a.split_cap;
      for (int r = lane; r < nrec; r += 32) {
        // a claim that crosses the capacity leaves empty records below it; the task
        // then runs all of its candidates itself
        if (base + r >= (unsigned long long)a.split_cap) break;
        const int rlo = per * r;
        a.split[base + r] = fits ? SplitRec{(int32_t)(e & 0xffffffffLL), (int32_t)(e >> 32), rlo,
                                            min(rlo + per, C2.n)}
                                 : SplitRec{0, 0, 0, 0};
      }
      if (fits) return 0;
    }
  }
  unsigned long long c = 0;
  if constexpr (K == 4) {
    if (p.flat) return count_flat<K>(p.fin, w, 2, C2, lo, hi, a, slots, big, lane);
    for (int i2 = lo; i2 < hi; ++i2) {
      set_vertex(w, 2, C2.p[i2], a, lane);
      for (int i = 0; i < p.nops[1]; ++i) run_op<K>(p.ops[1][i], w, a, slots, lane);
      c += count_op<K>(p.fin, w, a, slots, lane);
    }
    return c;
  } else if constexpr (K == 5) {
    for (int i2 = lo; i2 < hi; ++i2) {
      set_vertex(w, 2, C2.p[i2], a, lane);
      for (int i = 0; i < p.nops[1]; ++i) run_op<K>(p.ops[1][i], w, a, slots, lane);
      const Operand C3 = operand(w, p.cand[3], a, slots);
      if (p.flat) {
        c += count_flat<K>(p.fin, w, 3, C3, 0, C3.n, a, slots, big, lane);
      } else {
        for (int i3 = 0; i3 < C3.n; ++i3) {
          set_vertex(w, 3, C3.p[i3], a, lane);
          for (int i = 0; i < p.nops[2]; ++i) run_op<K>(p.ops[2][i], w, a, slots, lane);
          c += count_op<K>(p.fin, w, a, slots, lane);
        }
      }
    }
    return c;
  } else {  // 6 vertices: one more enumerated level (v3), then as 5 vertices with v4
    for (int i2 = lo; i2 < hi; ++i2) {
      set_vertex(w, 2, C2.p[i2], a, lane);
      for (int i = 0; i < p.nops[1]; ++i) run_op<K>(p.ops[1][i], w, a, slots, lane);
      const Operand C3 = operand(w, p.cand[3], a, slots);
      for (int i3 = 0; i3 < C3.n; ++i3) {
        set_vertex(w, 3, C3.p[i3], a, lane);
        for (int i = 0; i < p.nops[2]; ++i) run_op<K>(p.ops[2][i], w, a, slots, lane);
        const Operand C4 = operand(w, p.cand[4], a, slots);
        if (p.flat) {
          c += count_flat<K>(p.fin, w, 4, C4, 0, C4.n, a, slots, big, lane);
        } else {
          for (int i4 = 0; i4 < C4.n; ++i4) {
            set_vertex(w, 4, C4.p[i4], a, lane);
            for (int i = 0; i < p.nops[3]; ++i) run_op<K>(p.ops[3][i], w, a, slots, lane);
            c += count_op<K>(p.fin, w, a, slots, lane);
          }
        }
      }
    }
    return c;
  }
}

__device__ __forceinline__ int row_of(const int64_t* rowptr, int64_t nv, long long e) {
  int64_t lo = 0, n = nv + 1;  // first index with rowptr[idx] > e, minus one
  while (n > 0) {
    const int64_t h = n >> 1;
    if (rowptr[lo + h] <= e) {
      lo += h + 1;
      n -= h + 1;
    } else {
      n = h;
    }
  }
  return (int)(lo - 1);
}

template <int K>
__global__ void __launch_bounds__(kThreads, 4) k_setprog(Prog prog, ProgArgs a) {
  __shared__ Prog p;
  __shared__ unsigned roots;
  __shared__ WarpState ws[kWarps];
  if (threadIdx.x == 0) {
    p = prog;
    roots = step_roots(prog);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  WarpState& w = ws[wib];
  int32_t* slots = a.scratch + ((int64_t)blockIdx.x * kWarps + wib) * (a.nslots + 1) * a.slot_cap;
  unsigned long long c = 0;
  if (!a.split_mode) {
    for (;;) {
      unsigned long long e0 = 0;
      if (lane == 0) e0 = atomicAdd(a.heads, (unsigned long long)kChunk);
      e0 = __shfl_sync(0xffffffffu, e0, 0);
      if ((long long)e0 >= a.ne) break;
      const long long e1 = min((long long)e0 + kChunk, (long long)a.ne);
      int v0 = 0;
      if (lane == 0) v0 = row_of(a.rowptr, a.nv, (long long)e0);
      v0 = __shfl_sync(0xffffffffu, v0, 0);
      for (long long e = (long long)e0; e < e1; ++e) {
        while (a.rowptr[v0 + 1] <= e) ++v0;
        const int v1 = a.col[e];
        if (p.v1lt && v1 >= v0) continue;
        const int d0 = (int)(a.rowptr[v0 + 1] - a.rowptr[v0]);
        if (d0 <= a.bits_deg) continue;
        c += run_task<K>(p, roots, w, a, slots, v0, v1, e, 0, -1, true, lane);
      }
    }
  } else {
    const unsigned long long nrec = min(*(volatile unsigned long long*)(a.heads + 1),
                                        (unsigned long long)a.split_cap);
    for (;;) {
      unsigned long long r = 0;
      if (lane == 0) r = atomicAdd(a.heads + 2, 1ull);
      r = __shfl_sync(0xffffffffu, r, 0);
      if (r >= nrec) break;
      const SplitRec rec = a.split[r];
      if (rec.lo >= rec.hi) continue;
      const long long e = (long long)(uint32_t)rec.e_lo | ((long long)rec.e_hi << 32);
      int v0 = 0;
      if (lane == 0) v0 = row_of(a.rowptr, a.nv, e);
      v0 = __shfl_sync(0xffffffffu, v0, 0);
      c += run_task<K>(p, roots, w, a, slots, v0, a.col[e], e, rec.lo, rec.hi, false, lane);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if (lane == 0 && c) atomicAdd(a.total, c);
}

template <int K>
cudaError_t launch_k(const Prog& p, const ProgArgs& a, int grid, cudaStream_t s) {
  ProgArgs b = a;
  b.split_mode = 0;
  k_setprog<K><<<grid, kThreads, 0, s>>>(p, b);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || K == 3) return e;
  b.split_mode = 1;
  k_setprog<K><<<grid, kThreads, 0, s>>>(p, b);
  return cudaGetLastError();
}

int occupancy(int k) {
  int n = 0;
  cudaError_t e = k == 3   ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_setprog<3>, kThreads, 0)
                  : k == 4 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_setprog<4>, kThreads, 0)
                  : k == 5 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_setprog<5>, kThreads, 0)
                           : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_setprog<6>, kThreads, 0);
  return (e == cudaSuccess && n > 0) ? n : 1;
}

}  // namespace

xgm_status count_program(xgm_ctx* ctx, const DevGraph& g, const Prog& p, uint64_t* out,
                         xgm_stats& st) {
  std::string why;
  if (!prog_check(p, &why)) {
    set_thread_error("invalid set-operation program: " + why);
    return XGM_ERR_INVALID;
  }
  cudaStream_t s = ctx->stream;
  XGM_CUDA_TRY(cudaSetDevice(ctx->device));
  XGM_CUDA_TRY(cudaMemsetAsync(ctx->d_sc, 0, sizeof(Scalars), s));
  XGM_CUDA_TRY(ctx_mark(ctx, 0));
  ProgLut lut;
  const bool bits = prog_lut(p, &lut);
  if (bits) XGM_CUDA_TRY(ensure_plan_index(g, ctx->num_sms, s));  // once per graph
  ProgArgs a{};
  a.bits_deg = bits && g.plan_deg > 0 ? g.plan_deg : 0;
  const bool lists = g.max_deg > a.bits_deg;
  int grid = 0;
  if (lists) {
    const int nslots = p.nslots > 0 ? p.nslots : 1;
    const int64_t slot_cap = g.max_deg > 0 ? g.max_deg : 1;
    // resident warps, fewer when the scratch would pass 8 GB
    grid = ctx->num_sms * occupancy(p.k);
    // per warp: the program's slots and one list of candidates for count_flat
    const int64_t per_block = (int64_t)kWarps * (nslots + 1) * slot_cap * (int64_t)sizeof(int32_t);
    const int64_t budget = int64_t(8) << 30;
    if ((int64_t)grid * per_block > budget)
      grid = (int)std::max<int64_t>(ctx->num_sms, budget / per_block);
    const int64_t need = (int64_t)grid * kWarps * (nslots + 1) * slot_cap;
    if (need > ctx->prog_scratch_cap) {
      if (ctx->prog_scratch) XGM_CUDA_TRY(cudaFreeAsync(ctx->prog_scratch, s));
      ctx->prog_scratch = nullptr;
      ctx->prog_scratch_cap = 0;
      XGM_CUDA_TRY(cudaMallocAsync((void**)&ctx->prog_scratch, sizeof(int32_t) * need, s));
      ctx->prog_scratch_cap = need;
    }
    if (!ctx->prog_split)
      XGM_CUDA_TRY(cudaMallocAsync((void**)&ctx->prog_split, sizeof(SplitRec) * kSplitCap, s));
    a.slot_cap = slot_cap;
    a.nslots = nslots;
  }
  XGM_CUDA_TRY(ctx_mark(ctx, 1));
  a.rowptr = g.rowptr_o;
  a.col = g.col_o;
  a.nv = g.nv;
  a.ne = g.ne;
  a.scratch = ctx->prog_scratch;
  a.heads = ctx->d_sc->prog + 3;
  a.split = (SplitRec*)ctx->prog_split;
  a.split_cap = kSplitCap;
  // test hook: XGM_PROG_RECORD_CAP lowers the record capacity, so the overflow path (a
  // task that cannot queue its records runs them itself) can be exercised
  if (const char* cap = std::getenv("XGM_PROG_RECORD_CAP")) {
    const long long c = std::atoll(cap);
    if (c >= 0) a.split_cap = std::min<int64_t>(a.split_cap, c);
  }
  a.total = &ctx->d_sc->count;
  a.split_mode = 0;
  int launches = 0;
  if (bits) {
    cudaError_t e = launch_bits(g, prog_terms(p, lut), ctx->d_sc->prog, &ctx->d_sc->count,
                                ctx->timed ? ctx->d_sc->n : nullptr, ctx->num_sms, s, &launches);
    if (e != cudaSuccess) return cuda_fail(e, "k_bits_cta", __FILE__, __LINE__);
  }
  if (lists) {
    cudaError_t e = p.k == 3   ? launch_k<3>(p, a, grid, s)
                    : p.k == 4 ? launch_k<4>(p, a, grid, s)
                    : p.k == 5 ? launch_k<5>(p, a, grid, s)
                               : launch_k<6>(p, a, grid, s);
    if (e != cudaSuccess) return cuda_fail(e, "k_setprog", __FILE__, __LINE__);
    launches += p.k == 3 ? 1 : 2;
  }
  XGM_CUDA_TRY(ctx_mark(ctx, 2));
  xgm_status r = ctx_sync_scalars(ctx);
  if (r != XGM_OK) return r;
  const float prep = ctx_ms(ctx, 0, 1), kern = ctx_ms(ctx, 1, 2);
  std::memset(&st, 0, sizeof(st));
  st.prep_ms = prep;
  st.kernel_ms = kern;
  st.launches = launches;
  st.tasks = g.ne;
  st.variant_tasks[XGM_VAR_SPLIT] =
      ctx->h_sc->n[0] + std::min<int64_t>((int64_t)ctx->h_sc->prog[4], a.split_cap);
  *out = ctx->h_sc->count;
  return XGM_OK;
}

xgm_status program_kernels(xgm_ctx* ctx, const DevGraph& g, const Prog& p, int* n) {
  ProgLut lut;
  const bool bits = prog_lut(p, &lut);
  if (bits) {
    XGM_CUDA_TRY(cudaSetDevice(ctx->device));
    XGM_CUDA_TRY(ensure_plan_index(g, ctx->num_sms, ctx->stream));
  }
  *n = bits ? bits_launches(g) : 0;
  if (g.max_deg > (bits && g.plan_deg > 0 ? g.plan_deg : 0)) *n += p.k == 3 ? 1 : 2;
  return XGM_OK;
}

void program_buffers_free(xgm_ctx* ctx) {
  cudaStream_t s = ctx->stream;
  if (ctx->prog_scratch) cudaFreeAsync(ctx->prog_scratch, s);
  if (ctx->prog_split) cudaFreeAsync(ctx->prog_split, s);
  ctx->prog_scratch = nullptr;
  ctx->prog_split = nullptr;
  ctx->prog_scratch_cap = 0;
}

}  // namespace xgm
