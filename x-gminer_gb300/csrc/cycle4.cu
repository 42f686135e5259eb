// Edge-induced 4-cycles on the undirected graph (rank ids), hand-written for sm_103a.
//
// Reference (the counting definition): codes/GraphMiner/src/count/omp_base.cc:5-58 with
// cpu_kernels/rectangle.h:1-46.  For every v0, the wedges v0-v1-v2 with v1 < v0 and v2 < v0
// are grouped by v2; a group of c wedges closes C(c, 2) cycles.  Any total order of the
// vertices gives the same count, so rank ids serve.
//
// The wedges of v0 are the parts below v0 of its lower neighbours' rows; what they cost is
// the counter per v2, so every counter is in shared memory:
//  - k_c4_warp, a warp per v0 of up to kWarpSegs lower neighbours: these are looked up (their
//    rows' lengths below v0); up to kWarpWedges wedges go into the warp's hash table, sized by
//    the task (clearing it costs as much as filling it); larger tasks go to the lists of
//  - k_c4_cta, two CTAs per SM: up to kHashWedges wedges in one hash table; more are counted
//    a tile of v2 ids at a time in an array of 16-bit counters, read back and cleared once
//    per tile, or, where few of them fall in a tile, a range of ids at a time in the hash table
//    (hash_passes).  Rows are sorted, so a row's part in a tile is one run: tasks
//    of up to kCursors lower neighbours keep a cursor per row and go tile by tile, from their
//    smallest v2 on (a batch's graphs begin at other ids); hubs are
//    one unit per tile (any CTA can take it) and find the run by binary search.
// Measured (GB300): Erdos-Renyi 2^20, degree 32 (331 M wedges) 14.6 -> 4.6 ms; R-MAT s19
// ef16 (2.2 G wedges) 29.4 -> 10.2 ms.  (Before: a 4096-slot table cleared by a 256-thread
// CTA per task, and counters in L2 for tasks above 2,048 wedges, at about 90 G wedges/s,
// launched in groups from the host.)  Probing a table at 3/4 load, each wedge to its end
// before the next, was 6.8 ms on the Erdos-Renyi graph (11 of 32 threads active); one
// 1024-thread CTA per SM and tiles twice as long 9.85 against 9.7 ms on R-MAT, three 512-
// thread CTAs with tiles of 28,672 ids 12.0 ms.  Bound: instruction issue and the latency of
// the row look-ups (16 warps per SM in k_c4_warp: 12 KB of table each).
#include <algorithm>
#include <atomic>

#include "motif.cuh"

namespace xgm {

namespace {

constexpr int kWarpThreads = 128;
constexpr int kWarpSlots = 2048;      // hash slots of a warp (6 bytes each)
constexpr int kWarpWedges = 1344;     // load at most 2/3
constexpr int kWarpSegs = 64;         // most lower neighbours of a warp's task
constexpr int kCtaThreads4 = 512;
constexpr int kHashSlots = 16384;     // hash slots of the CTA
constexpr int kHashWedges = 8192;
constexpr int kTileWords = 23552;     // counter words: 47,104 counters of 16 bits
constexpr int kSegs = 512;            // most lower neighbours of a task that may be hashed
constexpr int kCursors = 2048;        // largest lower degree that keeps cursors
constexpr int kPassWedges = 6144;     // wedges a hash pass aims at
// Tiles (of 2 kTileWords ids) that cost as much as a pass; a task of no more passes than
// tiles / kPassTiles is counted in passes.  1 / 2 / 4 / 8 / 16: R-MAT s19 9.5 / 9.1 / 9.9 / 9.9 /
// 9.9 ms, s21 107 / 107 / 107 / 109 / 126, Chung-Lu 2^21 103 / 100 / 98 / 101 / 106, Erdos-Renyi
// 2^20 degree 128 98 / 98 / 98 / 163 / 224, Barabasi-Albert 1 M degree 64 33 / 32 / 32 / 36 / 43.
constexpr int kPassTiles = 2;
constexpr int kRowCap = 1 << 20;      // row lengths are summed up to here

struct WarpTable {
  uint32_t key[kWarpSlots];
  uint32_t cnt[kWarpSlots / 2];  // 16-bit halves
  long long base[32];
  int32_t pre[33];
  int32_t pad[3];
};
static_assert(sizeof(WarpTable) % 16 == 0, "tables are cleared 16 bytes at a time");

// Hash part of the CTA's shared memory (the tile counters and cursors use the same bytes).
struct CtaTable {
  uint32_t key[kHashSlots];
  uint32_t cnt[kHashSlots / 2];
  long long base[kSegs];
  int32_t pre[kSegs + 4];
};
struct CtaTile {
  uint32_t ctr[kTileWords];
  int32_t cur[kCursors];
  long long base[kCtaThreads4 / 32][32];
  int32_t pre[kCtaThreads4 / 32][34];
};
constexpr int kCtaSmem4 = (int)(sizeof(CtaTable) > sizeof(CtaTile) ? sizeof(CtaTable) : sizeof(CtaTile));
static_assert(2 * (kCtaSmem4 + 2048) <= 227 * 1024, "two CTAs per SM");
static_assert(kSegs == kCtaThreads4, "a thread per lower neighbour");

__device__ __forceinline__ long long first_ge(const int32_t* col, long long lo, long long hi,
                                              int32_t x) {
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (ldg_i32(col + mid) < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ uint32_t table_slot(int32_t x, uint32_t mask) {
  return ((uint32_t)x * 2654435761u) >> 7 & mask;
}

// Adds four wedges (x[h] < 0: none) to the table of mask + 1 slots; returns how many equal
// ones came before each, summed.  One probe per turn, whichever wedge a lane is at: a warp
// takes as many turns as its slowest lane has probes, not the sum of the slowest of each.
__device__ __forceinline__ unsigned table_add4(uint32_t* key, uint32_t* cnt, uint32_t mask,
                                               int32_t (&x)[4]) {
  unsigned before = 0;
  uint32_t slot = table_slot(x[0], mask);
  while (x[0] >= 0) {  // fewer wedges than slots: an empty one exists
    const uint32_t k = atomicCAS(&key[slot], 0xFFFFFFFFu, (uint32_t)x[0]);
    if (k == (uint32_t)x[0]) {
      const int sh = (slot & 1) * 16;
      before += 1u + ((atomicAdd(&cnt[slot >> 1], 1u << sh) >> sh) & 0xFFFFu);
    }
    slot = (slot + 1) & mask;
    if (k == 0xFFFFFFFFu || k == (uint32_t)x[0]) {
      x[0] = x[1];
      x[1] = x[2];
      x[2] = x[3];
      x[3] = -1;
      slot = table_slot(x[0], mask);
    }
  }
  return before;
}

// Slots (a power of two, at most `most`) for w wedges at a load of one half.
__device__ __forceinline__ int slots_for(int w, int most) {
  const int s = w <= 128 ? 256 : 1 << (33 - __clz(w - 1));
  return s < most ? s : most;
}

template <class T>
__device__ __forceinline__ void clear_table(T& t, int slots, int tid, int nt) {
  for (int i = tid; i < slots / 4; i += nt)
    reinterpret_cast<uint4*>(t.key)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
  for (int i = tid; i < slots / 8; i += nt)
    reinterpret_cast<uint4*>(t.cnt)[i] = make_uint4(0, 0, 0, 0);
}

// Walks k = k0, k0 + step, .. < total over the runs base[i] .. (pre[] their prefix), i the
// run of k0 or before, four elements in flight (f gets four, -1 past the end).
template <class F>
__device__ __forceinline__ void walk_runs(const int32_t* col, const long long* base,
                                          const int32_t* pre, int i, int k0, int step, int total,
                                          F f) {
  if (k0 >= total) return;
  int end = pre[i + 1];
  const int32_t* run = col + (base[i] - pre[i]);  // run[k]: element k
  for (int k = k0; k < total; k += 4 * step) {
    int32_t x[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int kk = k + h * step;
      x[h] = -1;
      if (kk < total) {
        if (kk >= end) {
          do end = pre[++i + 1];
          while (kk >= end);
          run = col + (base[i] - pre[i]);
        }
        x[h] = ldg_i32(run + kk);
      }
    }
    f(x);
  }
}

__device__ __forceinline__ void c4_emit(const GOut& o, int32_t v0, unsigned long long part,
                                        unsigned long long& acc) {
  if (!o.gid) {
    acc += part;
    return;
  }
  const unsigned long long w = warp_sum_u64(part);
  if ((threadIdx.x & 31) == 0 && w) atomicAdd(&o.out[(long long)o.gid[v0] * o.stride + o.slot], w);
}

__global__ void __launch_bounds__(kWarpThreads, 4) k_c4_warp(GView g, C4Queue* q, C4Lists l,
                                                             int step, unsigned long long* out,
                                                             GOut o) {
  extern __shared__ __align__(16) char sm[];
  let_next_start();
  const int lane = threadIdx.x & 31;
  WarpTable& t = reinterpret_cast<WarpTable*>(sm)[threadIdx.x >> 5];
  unsigned long long acc = 0;
  for (;;) {
    long long vb = 0;
    if (lane == 0) vb = (long long)atomicAdd(&q->vtx, (unsigned long long)step);
    vb = __shfl_sync(kFull, vb, 0);
    if (vb >= g.nv) break;
    long long my0 = 0;  // lane: lower neighbours of one of the claimed vertices
    int mydl = 0;
    if (lane < step && vb + lane < g.nv) {
      const int64_t v = g.nv - 1 - (vb + lane);  // highest degrees first
      my0 = g.rowptr[v];
      const long long dl = g.dptr[v].x - my0;
      if (dl > kCursors) {
        l.hub[atomicAdd(&q->n_hub, 1ull)] = (int32_t)v;
      } else if (dl > kSegs) {
        l.mid[atomicAdd(&q->n_mid, 1ull)] = (int32_t)v;
      } else if (dl > kWarpSegs) {
        l.hash[atomicAdd(&q->n_hash, 1ull)] = (int32_t)v;
      } else if (dl >= 2) {
        mydl = (int)dl;
      }
    }
    for (unsigned todo = __ballot_sync(kFull, mydl > 0); todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      const int32_t v0 = (int32_t)(g.nv - 1 - (vb + src));
      const long long a0 = __shfl_sync(kFull, my0, src);
      const int dl = __shfl_sync(kFull, mydl, src);
      int w = 0, len = 0;
      long long b = 0;
      for (int i = lane; i - lane < dl; i += 32) {  // (the last batch stays in len, b)
        len = 0;
        if (i < dl) {
          const int32_t v1 = ldg_i32(g.col + a0 + i);
          b = g.rowptr[v1];
          len = (int)(first_ge(g.col, b, g.dptr[v1].y, v0) - b);
        }
        w += (int)__reduce_add_sync(kFull, (unsigned)min(len, kWarpWedges + 1));
      }
      if (w < 2) continue;
      if (w > kWarpWedges) {
        if (lane == 0) l.hash[atomicAdd(&q->n_hash, 1ull)] = v0;
        continue;
      }
      const int slots = slots_for(w, kWarpSlots);
      const uint32_t mask = (uint32_t)slots - 1u;
      clear_table(t, slots, lane, 32);
      unsigned long long part = 0;
      for (int i0 = 0; i0 < dl; i0 += 32) {
        if (dl > 32) {  // looked up again, a batch at a time
          const int i = i0 + lane;
          len = 0;
          if (i < dl) {
            const int32_t v1 = ldg_i32(g.col + a0 + i);
            b = g.rowptr[v1];
            len = (int)(first_ge(g.col, b, g.dptr[v1].y, v0) - b);
          }
        }
        int inc = len;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int y = __shfl_up_sync(kFull, inc, d);
          if (lane >= d) inc += y;
        }
        __syncwarp();
        t.base[lane] = b;
        t.pre[lane] = inc - len;
        if (lane == 31) t.pre[32] = inc;
        __syncwarp();
        walk_runs(g.col, t.base, t.pre, 0, lane, 32, t.pre[32],
                  [&](int32_t (&x)[4]) { part += table_add4(t.key, t.cnt, mask, x); });
      }
      __syncwarp();
      c4_emit(o, v0, part, acc);
    }
  }
  acc = warp_sum_u64(acc);
  if (lane == 0 && acc) atomicAdd(out, acc);
  wait_for_previous();
}

// The wedges of v0 whose v2 is in [a, a + tile), one tile of counters.  Every warp takes 32
// lower neighbours at a time, finds their rows' runs in the tile (CURSOR: from cur[] on) and
// walks the runs as one index space.  (A warp per run: 220 G wedges/s at R-MAT s19, a load's
// latency per 64 elements; eight lanes per run: 112 instructions per 32 wedges.)
template <bool CURSOR>
__device__ unsigned long long tile_wedges(const GView& g, CtaTile& t, int* next, int32_t v0,
                                          long long a0, int dl, int64_t a, bool wide) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int64_t tile = wide ? kTileWords : 2 * kTileWords;
  const int32_t limit = (int32_t)(a + tile < v0 ? a + tile : v0);
  const int32_t lo_id = (int32_t)a;
  long long* base = t.base[tid >> 5];
  int32_t* pre = t.pre[tid >> 5];
  for (;;) {
    int i0 = 0;
    if (lane == 0) i0 = atomicAdd(next, 32);
    i0 = __shfl_sync(kFull, i0, 0);
    if (i0 >= dl) break;
    long long p = 0;
    int len = 0;
    if (i0 + lane < dl) {
      const int32_t v1 = ldg_i32(g.col + a0 + i0 + lane);
      const long long b = g.rowptr[v1], e = g.dptr[v1].y;
      p = CURSOR ? b + t.cur[i0 + lane] : (a > 0 ? first_ge(g.col, b, e, lo_id) : b);
      if (p < e && ldg_i32(g.col + p) < limit) {
        const long long hi = first_ge(g.col, p + 1, e, limit);
        len = (int)(hi - p);
        if (CURSOR) t.cur[i0 + lane] = (int32_t)(hi - b);
      }
    }
    // (a run is at most a tile long: 32 of them stay below 2^31)
    int inc = len;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(kFull, inc, d);
      if (lane >= d) inc += y;
    }
    __syncwarp();
    base[lane] = p;
    pre[lane] = inc - len;
    if (lane == 31) pre[32] = inc;
    __syncwarp();
    walk_runs(g.col, base, pre, 0, lane, 32, pre[32], [&](int32_t (&x)[4]) {
#pragma unroll
      for (int h = 0; h < 4; ++h)
        if (x[h] >= 0) {
          // neighbouring ids in different words: the tile's second half is the upper half
          const uint32_t i = (uint32_t)(x[h] - lo_id);
          const bool up = i >= (uint32_t)kTileWords;
          atomicAdd(&t.ctr[up ? i - kTileWords : i], up ? 0x10000u : 1u);
        }
    });
  }
  __syncthreads();
  if (tid == 0) *next = 0;
  unsigned long long acc = 0;
  const int used = (int)(limit - a < kTileWords ? limit - a : kTileWords);
  for (int w = tid; 4 * w < used; w += kCtaThreads4) {
    uint4* c4 = reinterpret_cast<uint4*>(t.ctr) + w;
    const uint4 c = *c4;
    if (!(c.x | c.y | c.z | c.w)) continue;
    *c4 = make_uint4(0, 0, 0, 0);
    const uint32_t cs[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const unsigned long long lo = wide ? cs[h] : cs[h] & 0xFFFFu, hi = wide ? 0u : cs[h] >> 16;
      acc += lo * (lo - (lo > 0)) / 2 + hi * (hi - (hi > 0)) / 2;
    }
  }
  __syncthreads();
  return acc;
}

// Exclusive prefix of v over the CTA's threads in `before`, their sum returned.
__device__ __forceinline__ int block_scan(int v, int* wsum, int& before) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int y = __shfl_up_sync(kFull, inc, d);
    if (lane >= d) inc += y;
  }
  __syncthreads();  // (every warp has read the sums of the scan before)
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  const int ws = lane < kCtaThreads4 / 32 ? wsum[lane] : 0;
  before = (int)__reduce_add_sync(kFull, (unsigned)(lane < warp ? ws : 0)) + inc - v;
  return (int)__reduce_add_sync(kFull, (unsigned)ws);
}

// A thread's rows of a task: rows tid, tid + kCtaThreads4, ..
constexpr int kRowsPerThread = kCursors / kCtaThreads4;

// Wedges of v0 (rows beyond kRowCap counted as that many), and the smallest v2 (v0: none).
__device__ __forceinline__ int task_wedges(const GView& g, int32_t v0, long long a0, int dl,
                                           int* wsum, int* least) {
  int sum = 0, low = v0, before;
  for (int i = threadIdx.x; i < dl; i += kCtaThreads4) {
    const int32_t v1 = ldg_i32(g.col + a0 + i);
    const long long b = g.rowptr[v1], e = first_ge(g.col, b, g.dptr[v1].y, v0);
    sum += (int)(e - b < kRowCap - 1 ? e - b : kRowCap - 1);
    if (b < e) low = min(low, ldg_i32(g.col + b));
  }
  if (threadIdx.x == 0) *least = v0;
  const int w = block_scan(sum, wsum, before);
  low = __reduce_min_sync(kFull, low);
  if ((threadIdx.x & 31) == 0 && low < v0) atomicMin(least, low);
  __syncthreads();
  return w;
}

// The wedges of v0 whose v2 is in [lo, end), a range of ids at a time, each range's wedges in
// the hash table; the first range is `step` long, each next one as long as its wedges fit by the
// density of the last.  For tasks whose wedges are few for the ids they are spread over: a tile
// of counters costs its scan however few it holds.  Erdos-Renyi 2^22, degree 128 (89 tiles for
// about 10,000 wedges): 2.66 s in tiles, 0.43 s in passes (1.75 s with counters in global
// memory).  CURSOR: up to kCursors rows, their places in registers; else searched for.
template <bool CURSOR>
__device__ __noinline__ unsigned long long hash_passes(const GView& g, CtaTable& h, int* wsum,
                                                       int32_t v0, long long a0, int dl,
                                                       int64_t lo, int64_t end, int64_t step) {
  const int tid = threadIdx.x;
  int cur[kRowsPerThread] = {}, len[kRowsPerThread] = {};
  unsigned long long acc = 0;
  // row i's place at id a (with CURSOR cur, its chunk's, says it)
  auto place = [&](int i, int64_t a, int at, long long* e) {
    const int32_t v1 = ldg_i32(g.col + a0 + i);
    const long long b = g.rowptr[v1];
    *e = g.dptr[v1].y;
    return CURSOR ? b + at : first_ge(g.col, b, *e, (int32_t)a);
  };
  for (int64_t a = lo; a < end;) {
    int64_t limit = min(a + step, end);
    int total, before;
    for (;;) {  // (a range of one id has at most a wedge per row)
      int sum = 0;
      long long e;
      if constexpr (CURSOR) {
#pragma unroll
        for (int c = 0; c < kRowsPerThread; ++c) {
          const int i = tid + c * kCtaThreads4;
          if (i < dl) {
            const long long p = place(i, a, cur[c], &e);
            len[c] = (int)(first_ge(g.col, p, e, (int32_t)limit) - p);
          }
          sum += min(len[c], kHashWedges + 1);
        }
      } else {
        for (int i = tid; i < dl; i += kCtaThreads4) {
          const long long p = place(i, a, 0, &e);
          sum += (int)min(first_ge(g.col, p, e, (int32_t)limit) - p, (long long)kHashWedges);
          sum = min(sum, kHashWedges + 1);
        }
      }
      total = block_scan(sum, wsum, before);
      if (total <= kHashWedges || limit - a <= 1) break;
      limit = a + (limit - a) / 2;
    }
    // one id in more rows than the table takes
    if (total > kHashWedges && tid == 0) acc += (unsigned long long)total * (total - 1) / 2;
    if (total > 1 && total <= kHashWedges) {
      const int slots = slots_for(total, kHashSlots);
      clear_table(h, slots, tid, kCtaThreads4);
      unsigned part = 0;
      auto walk = [&](long long p, int n) {  // the chunk's runs, one a thread
        const int all = block_scan(n, wsum, before);
        h.base[tid] = p;
        h.pre[tid] = before;
        if (tid == 0) h.pre[kSegs] = all;
        __syncthreads();
        int r = 0;
        if (tid < all) {  // the run of wedge tid: largest r with pre[r] <= tid
          int hi = kSegs;
          while (hi - r > 1) {
            const int mid = (r + hi) >> 1;
            if (h.pre[mid] <= tid) r = mid; else hi = mid;
          }
        }
        walk_runs(g.col, h.base, h.pre, r, tid, kCtaThreads4, all, [&](int32_t (&x)[4]) {
          part += table_add4(h.key, h.cnt, (uint32_t)slots - 1u, x);
        });
      };
      long long e;
      if constexpr (CURSOR) {
#pragma unroll
        for (int c = 0; c < kRowsPerThread; ++c) {
          if (c * kCtaThreads4 >= dl) break;
          walk(len[c] ? place(tid + c * kCtaThreads4, a, cur[c], &e) : 0, len[c]);
        }
      } else {
        for (int i0 = 0; i0 < dl; i0 += kCtaThreads4) {
          long long p = 0;
          int n = 0;
          if (i0 + tid < dl) {
            p = place(i0 + tid, a, 0, &e);
            n = (int)(first_ge(g.col, p, e, (int32_t)limit) - p);
          }
          walk(p, n);
        }
      }
      acc += part;
    }
    if constexpr (CURSOR) {
#pragma unroll
      for (int c = 0; c < kRowsPerThread; ++c) cur[c] += len[c];
    }
    const int64_t took = limit - a;
    a = limit;
    step = max((int64_t)1, min(4 * took, took * kPassWedges / max(total, 1)));
  }
  __syncthreads();
  return acc;
}

// What k_c4_hubs says of hub h: tiles of kTileWords ids that one hash pass takes (1: tiles of
// counters) and its smallest v2.  A vertex is in one list, so the other two lists' ends are free
// for as many entries as there are hubs.
__device__ __forceinline__ int32_t& hub_tiles(const C4Lists& l, int64_t nv, long long h) {
  return l.mid[nv - 1 - h];
}
__device__ __forceinline__ int32_t& hub_least(const C4Lists& l, int64_t nv, long long h) {
  return l.hash[nv - 1 - h];
}

// A CTA a hub: its wedges by its rows' lengths (most of a lower neighbour's row lies below v0).
// R-MAT s24 ef8 (713 tiles): 2.47 s with tiles for every hub, 1.54 s.
__global__ void __launch_bounds__(kCtaThreads4) k_c4_hubs(GView g, const C4Queue* q, C4Lists l) {
  __shared__ unsigned long long sum_s;
  __shared__ int low_s;
  for (long long u = blockIdx.x; u < (long long)q->n_hub; u += gridDim.x) {
    const int32_t v0 = l.hub[u];
    const long long a0 = g.rowptr[v0], dl = g.dptr[v0].x - a0;
    __syncthreads();
    if (threadIdx.x == 0) sum_s = 0, low_s = v0;
    __syncthreads();
    unsigned long long sum = 0;
    int low = v0;
    for (long long i = threadIdx.x; i < dl; i += kCtaThreads4) {
      const int32_t v1 = ldg_i32(g.col + a0 + i);
      const long long b = g.rowptr[v1], e = g.dptr[v1].y;
      sum += (unsigned long long)(e - b);
      if (b < e) low = min(low, ldg_i32(g.col + b));
    }
    sum = warp_sum_u64(sum);
    low = __reduce_min_sync(kFull, low);
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&sum_s, sum);
      atomicMin(&low_s, low);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const long long passes = (long long)(sum_s / kPassWedges) + 1;
      const long long tiles = ((long long)v0 - low_s + kTileWords - 1) / kTileWords;
      hub_tiles(l, g.nv, u) =
          2 * kPassTiles * passes <= tiles ? (int32_t)max(2ll, tiles / passes) : 1;
      hub_least(l, g.nv, u) = low_s;
    }
  }
}

__global__ void __launch_bounds__(kCtaThreads4, 2) k_c4_cta(GView g, C4Queue* q, C4Lists l,
                                                            bool planned,
                                                            unsigned long long* out, GOut o) {
  extern __shared__ __align__(16) char sm[];
  let_next_start();
  __shared__ long long task_s;
  constexpr int kWarps = kCtaThreads4 / 32;
  __shared__ int next, wsum[kWarps], least;
  CtaTile& t = *reinterpret_cast<CtaTile*>(sm);
  CtaTable& h = *reinterpret_cast<CtaTable*>(sm);
  const int tid = threadIdx.x, lane = tid & 31;
  unsigned long long acc = 0;
  const long long n_hub = (long long)q->n_hub, n_mid = (long long)q->n_mid,
                  n_hash = (long long)q->n_hash;
  if (n_hub + n_mid > 0)
    for (int w = tid; w < kTileWords; w += kCtaThreads4) t.ctr[w] = 0u;
  if (tid == 0) next = 0;
  // a task: every thread reads task_s between two barriers
  auto claim = [&](unsigned long long* head) {
    __syncthreads();
    if (tid == 0) task_s = (long long)atomicAdd(head, 1ull);
    __syncthreads();
    return task_s;
  };
  bool zero = n_hub + n_mid > 0;  // the tile counters are
  auto clear_counters = [&] {
    if (!zero)
      for (int i = tid; i < kTileWords / 4; i += kCtaThreads4)
        reinterpret_cast<uint4*>(t.ctr)[i] = make_uint4(0, 0, 0, 0);
    zero = true;
    __syncthreads();
  };
  // a task of w wedges from id lo on: tile by tile, a cursor per row, or in hash passes
  auto ranges = [&](int32_t v0, long long a0, int dl, int lo, int w) {
    const int tiles = ((int64_t)v0 - lo + 2 * kTileWords - 1) / (2 * kTileWords);
    unsigned long long part = 0;
    if (w >= 0 && w / kPassWedges + 1 <= tiles / kPassTiles) {
      zero = false;
      return hash_passes<true>(g, h, wsum, v0, a0, dl, lo, v0,
                               max((int64_t)1, ((int64_t)v0 - lo) * kPassWedges / max(w, 1)));
    }
    clear_counters();
    for (int i = tid; i < dl; i += kCtaThreads4) t.cur[i] = 0;
    __syncthreads();
    for (int64_t a = lo; a < v0; a += 2 * kTileWords)
      part += tile_wedges<true>(g, t, &next, v0, a0, dl, a, false);
    return part;
  };
  // hubs: unit = (hub, tile of kTileWords ids); a 16-bit tile takes two of them, a hash pass as
  // many as k_c4_hubs says
  const long long tiles = (g.nv + kTileWords - 1) / kTileWords;
  for (long long u = claim(&q->h_hub); u < n_hub * tiles; u = claim(&q->h_hub)) {
    const int32_t v0 = l.hub[u / tiles];
    const long long tile = u % tiles, at = tile * kTileWords;
    if (at >= v0) continue;
    const long long a0 = g.rowptr[v0];
    const int dl = (int)(g.dptr[v0].x - a0);
    const bool wide = dl > 0xFFFF;  // a counter may pass 16 bits
    const int most = planned ? hub_tiles(l, g.nv, u / tiles) : 1;
    const int64_t lo = planned ? hub_least(l, g.nv, u / tiles) : 0;
    if (most > 1) {
      if (tile % most) continue;
      const int64_t a = max((int64_t)at, lo), end = min((int64_t)at + (int64_t)most * kTileWords, (int64_t)v0);
      if (a >= end) continue;
      zero = false;
      c4_emit(o, v0, hash_passes<false>(g, h, wsum, v0, a0, dl, a, end, end - a), acc);
      continue;
    }
    if ((!wide && (tile & 1)) || at + (wide ? 1 : 2) * kTileWords <= lo) continue;
    clear_counters();
    c4_emit(o, v0, tile_wedges<false>(g, t, &next, v0, a0, dl, at, wide), acc);
  }
  for (long long u = claim(&q->h_mid); u < n_mid; u = claim(&q->h_mid)) {
    const int32_t v0 = l.mid[u];
    const long long a0 = g.rowptr[v0];
    const int dl = (int)(g.dptr[v0].x - a0);
    // the wedges are looked up only where their number can matter: with enough tiles below v0,
    // or in a batch, whose graphs begin at other ids
    int lo = 0, w = -1;
    if (o.gid || v0 >= 4 * kPassTiles * 2 * kTileWords) {
      w = task_wedges(g, v0, a0, dl, wsum, &least);
      lo = least;
    }
    c4_emit(o, v0, ranges(v0, a0, dl, lo, w), acc);
  }
  for (long long u = claim(&q->h_hash); u < n_hash; u = claim(&q->h_hash)) {
    const int32_t v0 = l.hash[u];
    const long long a0 = g.rowptr[v0];
    const int dl = (int)(g.dptr[v0].x - a0);  // <= kSegs = the CTA's threads
    long long b = 0;
    int len = 0;
    if (tid < dl) {
      const int32_t v1 = ldg_i32(g.col + a0 + tid);
      b = g.rowptr[v1];
      len = (int)(first_ge(g.col, b, g.dptr[v1].y, v0) - b);
    }
    int before;
    const int total = block_scan(min(len, kRowCap - 1), wsum, before);
    if (total > kHashWedges) {
      if (tid == 0) least = v0;
      __syncthreads();
      const int low = __reduce_min_sync(kFull, len ? ldg_i32(g.col + b) : v0);
      if (lane == 0 && low < v0) atomicMin(&least, low);
      __syncthreads();
      c4_emit(o, v0, ranges(v0, a0, dl, least, total), acc);
      continue;
    }
    zero = false;
    h.base[tid] = b;
    h.pre[tid] = before;
    if (tid == 0) h.pre[kSegs] = total;
    const int slots = slots_for(total, kHashSlots);
    clear_table(h, slots, tid, kCtaThreads4);
    __syncthreads();
    unsigned long long part = 0;
    int i = 0;
    if (tid < total) {  // the run of wedge tid: largest i with pre[i] <= tid
      int hi = dl;
      while (hi - i > 1) {
        const int mid = (i + hi) >> 1;
        if (h.pre[mid] <= tid) i = mid; else hi = mid;
      }
    }
    walk_runs(g.col, h.base, h.pre, i, tid, kCtaThreads4, total, [&](int32_t (&x)[4]) {
      part += table_add4(h.key, h.cnt, (uint32_t)slots - 1u, x);
    });
    c4_emit(o, v0, part, acc);
  }
  acc = warp_sum_u64(acc);
  if (lane == 0 && acc) atomicAdd(out, acc);
  wait_for_previous();
}

}  // namespace

bool cycle4_has_cta(const DevGraph& g) {
  // v0 has at most max_deg lower neighbours, with rows of at most max_deg
  return g.max_deg * g.max_deg > kWarpWedges;
}

cudaError_t launch_cycle4(const DevGraph& g, C4Queue* q, const C4Lists& l,
                          unsigned long long* out, int num_sms, cudaStream_t s, const GOut& o,
                          bool next) {
  if (g.nv == 0) return cudaSuccess;
  constexpr int kWarps = kWarpThreads / 32;
  constexpr int smem = kWarps * (int)sizeof(WarpTable);
  // the shared-memory opt-ins, once per device
  static std::atomic<unsigned long long> opted{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (e == cudaSuccess && !(opted.load(std::memory_order_acquire) & bit)) {
    e = cudaFuncSetAttribute(k_c4_warp, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_c4_cta, cudaFuncAttributeMaxDynamicSharedMemorySize, kCtaSmem4);
    if (e == cudaSuccess) opted.fetch_or(bit, std::memory_order_acq_rel);
  }
  if (e != cudaSuccess) return e;
  const int64_t grid = std::min<int64_t>(4 * num_sms, (g.nv + kWarps - 1) / kWarps);
  const int step = (int)std::max<int64_t>(1, std::min<int64_t>(32, g.nv / (4 * kWarps * grid)));
  e = launch_next(!next, k_c4_warp, grid, kWarpThreads, smem, s, g.view(), q, l, step, out, o);
  if (e != cudaSuccess || !cycle4_has_cta(g)) return e;
  // hubs are looked over where their tiles can be too many (as for the other lists)
  const bool planned = g.max_deg > kCursors && (o.gid || g.nv >= 4 * kPassTiles * 2 * kTileWords);
  if (planned) {
    k_c4_hubs<<<2 * num_sms, kCtaThreads4, 0, s>>>(g.view(), q, l);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  k_c4_cta<<<2 * num_sms, kCtaThreads4, kCtaSmem4, s>>>(g.view(), q, l, planned, out, o);
  return cudaGetLastError();
}

}  // namespace xgm
