// Triangles and k-cliques from the side of the later endpoint ("owner"), hand-written for
// sm_103a.
//
// Reference kernels this replaces (same counts, different schedule):
//  - warp_edge (TC): codes/GraphMiner/src/triangle/gpu_kernels/bs_warp_edge.cuh:1-20
//  - clique4_warp_edge / clique5_warp_edge and their LUT forms: as in clique.cu
//
// Every triangle v < u < x of the degree-oriented DAG is found at its edge (v, u): x lies
// in N+(u) and in the part of N+(v) after u (its suffix).  Testing suffixes costs
// sum_v C(d+(v), 2) probes, whereas streaming N+(u) against a filter of N+(v) costs
// sum_(v,u) d+(u): at R-MAT scale 22 7.2 G against 29 G elements, because the
// out-neighbours u of a low vertex are hubs with long lists.
//
//  - big u (degree > kBigDeg, in graphs with out-lists above kShortLists): a CTA holds N+(u)
//    as a bitmap over [u + 1, V) and takes up to kOwnChunk in-neighbours v of u.  A thread
//    finds u's place in N+(v) by binary search (N+(v) is sorted); suffixes of up to kOwnShort
//    elements are tested by that thread, longer ones go to a table in shared memory, longest
//    first, and are tested by eight lanes each, a 16-byte unit per lane and step.  A hub's
//    in-neighbours are many units (u, chunk) that any CTA can take.
//  - the other u: one lane per edge (v, u) meets the suffix with N+(u) (merge_lists); both
//    are short where deg v <= deg u <= kBigDeg or no list is above kShortLists.  Longer ones
//    come here too where more vertices are above kBigDeg than the bitmap has bits, and in
//    batches: a graph with many of them is the task kernel's (task_kernel_wins, count.cu).
// Bitmaps are cleared by taking the inserted bits out again: a unit costs d+(u) stores,
// not the bitmap's size.
//
// The tests of one pair (v, u), in order, are row i of v's local DAG (u = N+(v)[i]): bit j
// iff N+(v)[j] is in N+(u).  The rows mode writes them to the row store, whole words from
// one place, no atomics; the count kernels then read a vertex's rows as one contiguous
// matrix (k = 4 .. 7).
//
// Measured (GB300, a call before -> now):
//  triangles  R-MAT s20 ef16 8.45 -> 1.42 ms; Barabasi-Albert, 3,312 vertices, 106 -> 20 us
//             (13 launches -> 1: no task lists)
//  4-cliques  R-MAT s22 65.6 -> 20.0 ms (rows 10.4, counting 9.0); s20 12.4 -> 3.5 ms
//  5-cliques  R-MAT s20 140 -> 28.6 ms; 6-cliques R-MAT s16 96 -> 10.5 ms
//  triangles per edge (diamonds), Chung-Lu 1.5 M vertices, degree 32: 9.9 -> 2.8 ms; R-MAT
//             s19 3.76 -> 1.47 ms (the hits' rank look-ups and counters: the bare count of
//             the same suffixes is 2.5 times faster)
//  4,096 Barabasi-Albert graphs, triangles + 4-cliques + diamonds each: 3.44 -> 1.17 ms
// The tests with a warp per suffix, a ballot per 32 elements: 1.86 ms (s20 triangles), 15.2
// ms (s22 rows): 145 instructions a pair, of which a third for the pair itself.
// Bound: R-MAT s22 rows, L2 and DRAM latency (2.2 G sectors, 12 GB of DRAM reads: the lists
// exceed L2) and instruction issue; counting, the tensor pipe (8.5 clocks a step: 9 of the
// 29 ms of the s20 5-clique) and the shifts and ANDs that feed it at 16 warps per SM.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <type_traits>

#include "rows.cuh"

namespace xgm {

namespace {

constexpr int kOwnThreads = 256;
constexpr int kOwnWarps = kOwnThreads / 32;
constexpr int kOwnChunk = 512;   // in-neighbours of one unit (two per thread)
constexpr int kOwnShort = 12;    // longest suffix one thread tests by itself
constexpr int kOwnLevels = 512;  // most units of one owner (host: raises the chunk above it)
constexpr int kSmallStep = 128;  // most vertices per claim of the small phase

struct OwnArgs {
  GView g;
  int64_t big0;    // first big rank
  int64_t chunk;   // in-neighbours per unit: a multiple of kOwnChunk
  int levels;      // units of the vertex of the largest degree
  int wmask;       // bitmap words - 1 (a power of two of them)
  int step;        // vertices per claim of the small phase
  const int64_t* roff = nullptr;  // rows mode: row store offset per vertex (-1: no rows)
  uint32_t* rows = nullptr;       // rows mode: the row store
  unsigned* epart = nullptr;      // participation mode: triangles per col entry
  int ranks = 0;                  // and its counters per out-neighbour of the owner
};

// kOwnPart credits every triangle (v, u, x) to its three edges, each at its lower end's col
// entry: (v, u) once per pair, (v, x) at the tested element itself, (u, x) in a shared
// counter of x's rank in N+(u), flushed once per unit.
// kOwnMulti does what kOwnRows and kOwnPart do.
enum { kOwnCount = 0, kOwnRows = 1, kOwnPart = 2, kOwnMulti = 3 };
constexpr int kOwnRanks = 4096;  // most shared counters; longer out-lists credit epart itself

// A suffix that eight lanes test: col[p .. p + len).  Rows mode: element e is bit
// i + 1 + e of row i of v's local DAG, whose word i / 32 is rows[out].
template <int MODE>
struct OwnPair {
  long long p;
  int len;
};
template <>
struct OwnPair<kOwnRows> {
  long long p, out;
  int len, i;
};
template <>
struct OwnPair<kOwnMulti> : OwnPair<kOwnRows> {};

// 32-bit mask of the bits below r (r <= 0: none, r >= 32: all).
__device__ __forceinline__ uint32_t mask_below(int r) {
  uint32_t m;
  asm("shl.b32 %0, %1, %2;" : "=r"(m) : "r"(0xFFFFFFFFu), "r"(r > 0 ? r : 0));  // clamps at 32
  return ~m;
}

// Row i of an s-vertex local DAG, built one word after the other by one thread.
struct RowWriter {
  uint32_t* out;  // word i / 32 of the row
  uint32_t bits = 0;
  int w;
  __device__ RowWriter(uint32_t* o, int i) : out(o), w(i >> 5) {}
  __device__ void upto(int q) {
    while (w < q) {
      *out++ = bits;
      bits = 0;
      ++w;
    }
  }
  __device__ void put(int j, uint32_t bit) {
    upto(j >> 5);
    bits |= bit << (j & 31);
  }
  __device__ void finish(int s) {
    upto((s - 1) >> 5);
    *out = bits;
  }
};

// Calls f(k, l) for every element the sorted ranges [a, ea) and [b, eb) of col have in common,
// at col[k] and col[l], k ascending.  Eight of b's elements at a time stay in registers and every
// one of a's up to the last of them is compared with all: the loads do not wait for one another
// as a merge's do, and lanes with lists of other lengths part less.  4,096 small graphs (5.5
// out-neighbours a vertex), the owner kernel: 1.05 ms by a merge, 0.80 with four held, 0.69 with
// six, 0.67 with eight.
constexpr int kMergeHold = 8;
template <class F>
__device__ __forceinline__ void merge_lists(const int32_t* col, long long a, long long ea,
                                            long long b, long long eb, F f) {
  if (a >= ea) return;
  for (; b < eb; b += kMergeHold) {
    int32_t y[kMergeHold];
#pragma unroll
    for (int j = 0; j < kMergeHold; ++j) y[j] = b + j < eb ? ldg_i32(col + b + j) : INT32_MAX;
    for (;;) {
      const int32_t x = ldg_i32(col + a);
      if (x > y[kMergeHold - 1]) break;
      int at = -1;
#pragma unroll
      for (int j = 0; j < kMergeHold; ++j)
        if (y[j] == x) at = j;
      if (at >= 0) f(a, b + at);
      if (++a >= ea) return;
    }
  }
}

__device__ __forceinline__ long long lower_at(const int32_t* col, long long lo, long long hi,
                                              int32_t x) {
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (ldg_i32(col + mid) < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// CTAs per SM the registers are cut for, measured per mode (the bitmap allows 5 at R-MAT s22):
// triangles s20 1.52 / 1.49 / 1.43 ms with 4 / 5 / 6, rows s22 11.9 / 13.9 / 13.5,
// participation of a 1.5 M vertex Chung-Lu graph 3.47 / 3.30 / 3.95, rows and participation
// of 4,096 small graphs 0.71 / 0.67 / 0.71 (all with 2^18-bit bitmaps from degree 65 on).
constexpr int own_ctas(int mode) {
  return mode == kOwnRows ? 4 : (mode == kOwnCount ? 6 : 5);
}

template <int MODE>
__global__ void __launch_bounds__(kOwnThreads, own_ctas(MODE)) k_owner(OwnArgs a, OwnHeads* heads,
                                                       unsigned long long* count) {
  constexpr bool ROWS = (MODE & kOwnRows) != 0, PART = (MODE & kOwnPart) != 0;
  extern __shared__ uint32_t bm[];
  let_next_start();
  // participation mode: counters per rank in N+(u), members before each bitmap word
  uint32_t* rcnt = bm + a.wmask + 1;
  uint16_t* wpre = reinterpret_cast<uint16_t*>(rcnt + a.ranks);
  __shared__ OwnPair<MODE> tab[kOwnChunk];
  __shared__ int lev[kOwnLevels + 1];  // lev[l]: units of levels above l (highest first)
  __shared__ int hist[32];  // long suffixes of the chunk by length
  __shared__ long long unit_s;
  __shared__ int wsum[2][kOwnWarps];
  const GView& g = a.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned long long acc = 0;

  if (a.big0 < g.nv) {
    for (int w = tid; w <= a.wmask; w += kOwnThreads) bm[w] = 0u;
    if (PART)
      for (int w = tid; w < a.ranks; w += kOwnThreads) rcnt[w] = 0u;
    // Units: level l holds the chunk l of every big vertex of degree > l * chunk, a prefix
    // of the descending degree order.  Levels are taken from the highest down, so the
    // last units are the small ones.
    for (int l = tid; l < a.levels; l += kOwnThreads) {
      int64_t lo = a.big0, hi = g.nv;
      while (l > 0 && lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (g.dptr[mid].y - g.rowptr[mid] > (int64_t)l * a.chunk) hi = mid; else lo = mid + 1;
      }
      lev[l] = (int)(g.nv - lo);
    }
    if (tid < 32) hist[tid] = 0;
    if (tid == 0) unit_s = (long long)atomicAdd(&heads->big, 1ull);
    __syncthreads();
    if (warp == 0) {  // suffix sums over the levels
      int run = 0;
      for (int top = a.levels; top > 0; top -= 32) {
        const int l = top - 1 - lane;
        int v = l >= 0 ? lev[l] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(kFull, v, o);
          if (lane >= o) v += y;
        }
        if (l >= 0) lev[l] = run + v;  // units of levels >= l
        run += __shfl_sync(kFull, v, 31);
      }
      if (lane == 0) lev[a.levels] = 0;
    }
    __syncthreads();
    const long long units = lev[0];
    for (;;) {
      const long long t = unit_s;
      if (t >= units) break;
      int l = 0;  // lev[l + 1] <= t < lev[l]
      {
        int lo = 0, hi = a.levels;
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (lev[mid] > t) lo = mid; else hi = mid;
        }
        l = lo;
      }
      const int64_t u = g.nv - 1 - (t - lev[l + 1]);
      const longlong2 du = ldg_ll2(g.dptr + u);
      const long long c0 = g.rowptr[u] + (long long)l * a.chunk;
      const long long c1 = c0 + a.chunk < du.x ? c0 + a.chunk : du.x;
      // (rows mode: an owner without out-neighbours still writes its empty rows)
      const bool live = (ROWS || du.x < du.y) && c0 < c1;  // uniform
      if (!live) __syncthreads();  // every thread has read unit_s
      for (long long cc = c0; live && cc < c1; cc += kOwnChunk) {
        // insert N+(u) (first pass) while the in-neighbours look u up in their lists
        if (cc == c0)
          for (long long e = du.x + tid; e < du.y; e += kOwnThreads) {
            const uint32_t off = (uint32_t)(ldg_i32(g.col + e) - (int32_t)u - 1);
            atomicOr(&bm[off >> 5], 1u << (off & 31));
          }
        long long p[2], row[2];  // list of v, row of the row store
        int ii[2], ss[2];        // u's place in it, its length
        int bin[2], slot[2];     // long suffixes: by length in words, longest first
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const long long e = cc + h * kOwnThreads + tid;
          ii[h] = ss[h] = 0;
          bin[h] = -1;
          if (e < c1) {
            const int32_t v = ldg_i32(g.col + e);
            const long long ro = ROWS ? __ldg(a.roff + v) : 0;
            const longlong2 dv = ro >= 0 ? ldg_ll2(g.dptr + v) : make_longlong2(0, 0);
            if (dv.y - dv.x >= (MODE == kOwnRows ? 3 : 2)) {
              p[h] = dv.x;
              ss[h] = (int)(dv.y - dv.x);
              ii[h] = (int)(lower_at(g.col, dv.x, dv.y, (int32_t)u) - dv.x);
              if (ROWS) row[h] = ro + tri_row_off(ii[h], (ss[h] + 31) >> 5);
              const int len = ss[h] - ii[h] - 1;
              if (len > kOwnShort) {
                bin[h] = 31 - (len < 32 * 31 ? len >> 5 : 31);
                slot[h] = atomicAdd(&hist[bin[h]], 1);
              }
            }
          }
        }
        __syncthreads();
        int nl;
        {  // start of each bin (every warp for itself), then the table
          const int c = hist[lane];
          int inc = c;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, inc, o);
            if (lane >= o) inc += y;
          }
          nl = __shfl_sync(kFull, inc, 31);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int b0 = __shfl_sync(kFull, inc - c, bin[h] & 31);
            if (bin[h] >= 0) {
              OwnPair<MODE>& x = tab[b0 + slot[h]];
              x.p = p[h] + ii[h] + 1;
              x.len = ss[h] - ii[h] - 1;
              if constexpr (ROWS) {
                x.out = row[h];
                x.i = ii[h];
              }
            }
          }
        }
        unsigned part = 0;
        const int32_t base = (int32_t)u + 1;
        // participation mode: x is the bit `off` of N+(u)
        auto credit = [&](uint32_t off) {
          const uint32_t word = bm[off >> 5];
          const int r = wpre[off >> 5] + __popc(word & ((1u << (off & 31)) - 1u));
          if (r < a.ranks) atomicAdd(&rcnt[r], 1u);
          else atomicAdd(&a.epart[du.x + r], 1u);
        };
        if (PART && cc == c0) {
          // members before each word (whole bitmap words of this owner), by a scan of 32
          // words per warp and step; the totals of the steps before in wsum
          const int words = (int)((g.nv - u + 30) >> 5);  // bits [0, V - u - 1)
          int run = 0;
          for (int w0 = 0; w0 < words; w0 += kOwnThreads) {
            const int w = w0 + tid;
            const int c = w < words ? __popc(bm[w]) : 0;
            int inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const int y = __shfl_up_sync(kFull, inc, o);
              if (lane >= o) inc += y;
            }
            if (lane == 31) wsum[(w0 / kOwnThreads) & 1][warp] = inc;
            __syncthreads();
            const int ws = lane < kOwnWarps ? wsum[(w0 / kOwnThreads) & 1][lane] : 0;
            const int before = (int)__reduce_add_sync(kFull, (unsigned)(lane < warp ? ws : 0));
            if (w < words) wpre[w] = (uint16_t)(run + before + inc - c);
            run += (int)__reduce_add_sync(kFull, (unsigned)ws);
          }
          __syncthreads();
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (bin[h] < 0 && ss[h] > 0) {
            RowWriter w(ROWS ? a.rows + row[h] : nullptr, ii[h]);
            unsigned hits = 0;
            for (int j = ii[h] + 1; j < ss[h]; ++j) {
              const uint32_t off = (uint32_t)(ldg_i32(g.col + p[h] + j) - base);
              const uint32_t bit = (bm[off >> 5] >> (off & 31)) & 1u;
              if (ROWS) w.put(j, bit);
              hits += bit;
              if (PART && bit) {
                atomicAdd(&a.epart[p[h] + j], 1u);
                credit(off);
              }
            }
            if (ROWS) w.finish(ss[h]);
            if (PART && hits) atomicAdd(&a.epart[p[h] + ii[h]], hits);
            part += hits;
          }
        __syncthreads();
        // Eight lanes per suffix, one 16-byte unit each, from the unit its first element is
        // in: 32 elements of four suffixes per step.  An element before or after the suffix
        // reads some word of the bitmap (the index wraps) and is masked by its place.
        const int l8 = lane & 7;
        for (int k0 = 4 * warp; k0 < nl; k0 += 4 * kOwnWarps) {
          const int k = k0 + (lane >> 3);
          OwnPair<MODE> t{};
          if (k < nl) t = tab[k];
          const int ph = (int)(t.p & 3);
          const int rem = t.len > 0 ? t.len + ph : 0;  // elements from the first unit on
          const int4* q = reinterpret_cast<const int4*>(g.col + (t.p - ph)) + l8;
          // rows mode: step n gives row bits from b0 + 32 n on
          int b0 = 0, steps = (rem + 31) >> 5, w0 = 0;
          uint32_t prev = 0;
          uint32_t* out = nullptr;
          if constexpr (ROWS) {
            b0 = t.i + 1 - ph;
            w0 = (b0 >> 5) - (t.i >> 5);  // of the first step, from the row's first word
            out = a.rows + t.out + w0;
            if (rem) steps = ((b0 + rem - 1) >> 5) - (b0 >> 5) + 1;
            if (l8 == 0 && w0 == 1) out[-1] = 0u;  // bits up to i: none
          }
          const int most = __reduce_max_sync(kFull, steps);
          unsigned hits = 0;
          int4 x = make_int4(0, 0, 0, 0);
          if (4 * l8 < rem) x = __ldg(q);
          for (int n = 0; n < most; ++n) {
            int4 y = make_int4(0, 0, 0, 0);
            if (32 * (n + 1) + 4 * l8 < rem) y = __ldg(q + 8 * (n + 1));
            const int32_t xs[4] = {x.x, x.y, x.z, x.w};
            uint32_t bits = 0;  // the four tests, in the top bits
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const uint32_t off = (uint32_t)(xs[h] - base);
              const uint32_t word = bm[(off >> 5) & a.wmask] >> (off & 31);
              if constexpr (PART) {
                const int e = 32 * n + 4 * l8 + h;
                if ((word & 1u) && e >= ph && e < rem) {
                  ++hits;
                  atomicAdd(&a.epart[t.p - ph + e], 1u);
                  credit(off);
                }
              }
              if constexpr (MODE != kOwnPart) bits = __funnelshift_r(bits, word, 1);
            }
            if constexpr (ROWS) {
              uint32_t word = bits >> (28 - 4 * l8);
              word |= __shfl_xor_sync(kFull, word, 1);
              word |= __shfl_xor_sync(kFull, word, 2);
              word |= __shfl_xor_sync(kFull, word, 4);
              word &= mask_below(rem - 32 * n);
              if (n == 0) word &= 0xFFFFFFFFu << ph;
              if (l8 == 0 && n < steps && w0 + n >= 0) out[n] = __funnelshift_l(prev, word, b0 & 31);
              prev = word;
            } else if constexpr (!PART) {
              uint32_t m = mask_below(rem - 32 * n - 4 * l8);
              if (n == 0 && l8 == 0) m &= 0xFFFFFFFFu << ph;
              part += __popc((bits >> 28) & m);
            }
            x = y;
          }
          if constexpr (PART) {
            hits += __shfl_xor_sync(kFull, hits, 1);
            hits += __shfl_xor_sync(kFull, hits, 2);
            hits += __shfl_xor_sync(kFull, hits, 4);
            if (l8 == 0 && hits) atomicAdd(&a.epart[t.p - 1], hits);
          }
        }
        acc += part;
        __syncthreads();
        if (tid < 32) hist[tid] = 0;
        if (cc + kOwnChunk < c1) __syncthreads();
      }
      if (tid == 0) unit_s = (long long)atomicAdd(&heads->big, 1ull);
      if (live)
        for (long long e = du.x + tid; e < du.y; e += kOwnThreads) {
          bm[(uint32_t)(ldg_i32(g.col + e) - (int32_t)u - 1) >> 5] = 0u;
          if (PART && e - du.x < a.ranks) {
            const uint32_t c = rcnt[e - du.x];
            if (c) {
              atomicAdd(&a.epart[e], c);
              rcnt[e - du.x] = 0u;
            }
          }
        }
      __syncthreads();
    }
  }

  // small u: v < u < big0, one lane per edge (v, u) with a non-empty suffix
  const long long nsm = a.big0;
  for (;;) {
    long long vb = 0;
    if (lane == 0) vb = (long long)atomicAdd(&heads->small, (unsigned long long)a.step);
    vb = __shfl_sync(kFull, vb, 0);
    if (vb >= nsm) break;
    const long long ve = vb + a.step < nsm ? vb + a.step : nsm;
    for (long long b = vb; b < ve; b += 32) {
      longlong2 d = make_longlong2(0, 0);
      long long ro = 0;
      int cnt = 0;
      if (b + lane < ve) {
        const long long v = nsm - 1 - (b + lane);  // longest lists first
        if (ROWS) ro = __ldg(a.roff + v);
        if (ro >= 0) d = ldg_ll2(g.dptr + v);
        cnt = (int)(d.y - d.x) - (ROWS ? 0 : 1);  // the last row is empty
        if (d.y - d.x < (MODE == kOwnRows ? 3 : 2)) cnt = 0;
        if (cnt > 0 && ldg_i32(g.col + d.x + cnt - 1) >= a.big0)
          cnt = (int)(lower_at(g.col, d.x, d.x + cnt, (int32_t)a.big0) - d.x);
        if (cnt < 0) cnt = 0;
      }
      int inc = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, inc, o);
        if (lane >= o) inc += y;
      }
      const int total = __shfl_sync(kFull, inc, 31);
      for (int k0 = 0; k0 < total; k0 += 32) {
        const int k = k0 + lane;
        int q = 0;  // the lane whose vertex owns edge k: first with inc > k
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const int y = __shfl_sync(kFull, inc, q + o - 1);
          if (y <= k) q += o;
        }
        q &= 31;  // k >= total runs past the last lane
        const long long base = __shfl_sync(kFull, d.x, q), end = __shfl_sync(kFull, d.y, q);
        const int ex = __shfl_sync(kFull, inc - cnt, q);
        const long long qro = ROWS ? __shfl_sync(kFull, ro, q) : 0;
        if (k < total) {
          const int i = k - ex;
          const long long at = base + i;
          const longlong2 du = ldg_ll2(g.dptr + ldg_i32(g.col + at));
          unsigned hits = 0;
          if constexpr (ROWS) {
            const int s = (int)(end - base);
            RowWriter w(a.rows + qro + tri_row_off(i, (s + 31) >> 5), i);
            merge_lists(g.col, at + 1, end, du.x, du.y, [&](long long k, long long l) {
              w.put((int)(k - base), 1u);
              if (PART) {
                ++hits;
                atomicAdd(&a.epart[k], 1u);
                atomicAdd(&a.epart[l], 1u);
              }
            });
            w.finish(s);
          } else {
            merge_lists(g.col, at + 1, end, du.x, du.y, [&](long long k, long long l) {
              ++hits;
              if (PART) {
                atomicAdd(&a.epart[k], 1u);
                atomicAdd(&a.epart[l], 1u);
              }
            });
            if (!PART) acc += hits;
          }
          if (PART && hits) atomicAdd(&a.epart[at], hits);
        }
      }
    }
  }
  if constexpr (MODE == kOwnCount) {
    acc = warp_sum_u64(acc);
    if (lane == 0 && acc) atomicAdd(count, acc);
  }
  wait_for_previous();
}

template <int MODE>
cudaError_t launch_owner(const DevGraph& g, OwnArgs a, OwnHeads* heads, unsigned long long* count,
                         int num_sms, cudaStream_t s) {
  if (g.nv == 0) return cudaSuccess;
  a.g = g.view();
  const int64_t nbig = g.max_out <= kShortLists ? 0 : std::min<int64_t>(g.n_big, own_bits((MODE & kOwnPart) != 0));
  a.big0 = g.nv - nbig;
  const int64_t per = (g.max_deg + kOwnLevels - 1) / kOwnLevels;
  a.chunk = std::max<int64_t>(kOwnChunk, (per + kOwnChunk - 1) / kOwnChunk * kOwnChunk);
  a.levels = (int)std::max<int64_t>(1, (g.max_deg + a.chunk - 1) / a.chunk);
  int words = 32;
  while (32 * (int64_t)words < nbig) words *= 2;
  a.wmask = words - 1;
  int smem = 4 * words;
  cudaError_t e = cudaSuccess;
  if constexpr ((MODE & kOwnPart) != 0) {
    a.ranks = (int)std::min<int64_t>(g.max_out, kOwnRanks);
    smem += 4 * a.ranks + 2 * words;
    // the shared-memory opt-in of the largest layout, once per device
    static std::atomic<unsigned long long> opted{0};
    int dev = 0;
    e = cudaGetDevice(&dev);
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (e == cudaSuccess && !(opted.load(std::memory_order_acquire) & bit)) {
      e = cudaFuncSetAttribute(k_owner<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(kOwnBits / 32) * 6 + 4 * kOwnRanks);
      if (e == cudaSuccess) opted.fetch_or(bit, std::memory_order_acq_rel);
    }
    if (e != cudaSuccess) return e;
  }
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_owner<MODE>, kOwnThreads, smem);
  if (e != cudaSuccess) return e;
  // no more CTAs than there is work for (small graphs would only pay for starting them),
  // and claims small enough that every warp has a few
  const int64_t want = std::max<int64_t>(nbig, (a.big0 + 4 * kOwnWarps - 1) / (4 * kOwnWarps));
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)per_sm * num_sms, want));
  a.step = (int)std::max<int64_t>(4, std::min<int64_t>(kSmallStep, a.big0 / (4 * kOwnWarps * grid)));
  k_owner<MODE><<<(unsigned)grid, kOwnThreads, smem, s>>>(a, heads, count);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ row index
// Offsets of the row store and the row tasks of a graph, by the width of their rows.
__global__ void __launch_bounds__(256) k_rows_index(const longlong2* dptr, int64_t nv,
                                                    int64_t* roff, int32_t* word_l,
                                                    int32_t* team_l, unsigned long long* rn) {
  __shared__ unsigned wsum[8], lcnt[4];
  __shared__ unsigned long long wbase, lbase[4];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int64_t b = (int64_t)blockIdx.x * 256; b < nv; b += (int64_t)gridDim.x * 256) {
    const int64_t v = b + tid;
    int s = 0;
    if (v < nv) {
      const longlong2 d = ldg_ll2(dptr + v);
      s = d.y - d.x <= kRowsCap ? (int)(d.y - d.x) : 0;
    }
    const unsigned words = row_words(s);
    const int cls = s < 3 ? 4 : (s <= 8 ? 0 : (s <= 32 ? 1 : (s <= kRowsMid ? 2 : 3)));
    if (tid < 4) lcnt[tid] = 0;
    unsigned inc = words;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    unsigned slot = 0;
    if (cls < 4) slot = atomicAdd(&lcnt[cls], 1u);
    unsigned off = inc - words, tot = 0;
    for (int w = 0; w < 8; ++w) {
      if (w < warp) off += wsum[w];
      tot += wsum[w];
    }
    __syncthreads();
    if (tid == 0) wbase = atomicAdd(&rn[0], (unsigned long long)tot);
    if (tid < 4) lbase[tid] = atomicAdd(&rn[1 + tid], (unsigned long long)lcnt[tid]);
    __syncthreads();
    if (v < nv) {
      roff[v] = words ? (int64_t)(wbase + off) : -1;
      if (cls == 0) word_l[lbase[0] + slot] = (int32_t)v;
      else if (cls == 1) word_l[nv - 1 - (int64_t)(lbase[1] + slot)] = (int32_t)v;
      else if (cls == 2) team_l[lbase[2] + slot] = (int32_t)v;
      else if (cls == 3) team_l[nv - 1 - (int64_t)(lbase[3] + slot)] = (int32_t)v;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ counting
// A task's rows are the strict upper triangle of a 0/1 matrix A (row i: words i/32 .. W-1).
// Its triangles are the sum over edges (j, l) of C_jl = (A A^T)_jl, a contraction: 32 x 32
// blocks of C on the tensor cores, f16 operands and accumulators, masked by the block of A.
//  - The operands come straight from the bit rows: the k index of a step may be permuted if
//    both operands agree, so thread t of a quad takes the bits p, p + 16 of a row's word for
//    p = t, t + 4, t + 8, t + 12.  A bit p <= 11 of a 16-bit half is an f16 power of two by
//    itself, 2^(p-24), so j's fragments are the word ANDed with a mask; l's carry 2^(14-p).
//    A product is 2^-10, and a sum of n <= 1024 of them is exact in f16.
//  - The masked sum of a block is one more contraction: C's accumulator layout is the layout
//    of a k x n operand (C^T), so the diagonal of mask x C^T gathers sum_l A_jl C_jl per row
//    j in f32.  For that the columns of a block are taken in the order that puts l and
//    l + 16 into one accumulator register, as the mask's bits lie.  Only the diagonals of
//    two accumulators count; they are read once per matrix.
// popc over row words issues 4.3 words per clock and SM partition (measured; FLO for a walk
// over members costs as much), an f16 m16n8k16 7.5 words' worth in 8.5 clocks.  e4m3
// m16n8k32 is converted to f16 on this chip (12 conversions, 2 f16 steps and 4 additions
// each; R-MAT s20 5-clique 33.5 ms with it), the 1-bit form emulated (525 clocks), u8 65
// clocks.  A tcgen05 tile has 128 rows: most matrices here are 60 to 300 wide and
// triangular, and bits would have to be spread to bytes in shared memory first.
__device__ __forceinline__ void mma_f16(uint32_t (&d)[2], uint32_t a0, uint32_t a1, uint32_t a2,
                                        uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f16.f16.f16.f16 {%0,%1}, {%2,%3,%4,%5}, {%6,%7}, {%0,%1};"
      : "+r"(d[0]), "+r"(d[1])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Rows 8 .. 15 of the left operand are zero.
__device__ __forceinline__ void mma_f32(float (&d)[4], uint32_t a0, uint32_t a2, uint32_t b0,
                                        uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1));
}
constexpr float kUnit = 17179869184.0f;  // 2^34: a mask bit is 2^-24, a common neighbour 2^-10
constexpr uint32_t kPair = 0x00010001u;  // bits p, p + 16 of a word

// First word of block q's rows; a row of the block spans W - q words.
__device__ __forceinline__ int blk_off(int q, int W) { return 16 * q * (2 * W - q + 1); }

// Row of a block that column c of its n-tile nt takes (+ 4 nt).
__device__ __forceinline__ int col_row(int c) { return (c >> 1) + 16 * (c & 1); }

// Fragments of j's words w[r] (rows 8 r + lane / 4) and of l's (rows 4 r + col_row(lane / 4)):
// four registers per word, two per k step.
__device__ __forceinline__ void frag_j(uint32_t w, int t, uint32_t (&f)[4]) {
  f[0] = w & (kPair << t);
  f[1] = w & (kPair << (t + 4));
  f[2] = w & (kPair << (t + 8));
  f[3] = (w >> 4) & (kPair << (t + 8));
}
__device__ __forceinline__ void frag_l(uint32_t w, int t, uint32_t (&f)[4]) {
  // f16 2^(14 - p) is (29 - p) << 10; the last pair is at t + 12 but j's has weight t + 8
  f[0] = ((w >> t) & kPair) * ((29u - t) << 10);
  f[1] = ((w >> (t + 4)) & kPair) * ((25u - t) << 10);
  f[2] = ((w >> (t + 8)) & kPair) * ((21u - t) << 10);
  f[3] = ((w >> (t + 12)) & kPair) * ((21u - t) << 10);
}

// One step (32 k) of a block.
__device__ __forceinline__ void block_mma(uint32_t (&c)[2][4][2], const uint32_t (&a)[4],
                                          const uint32_t (&b)[4], int t) {
  uint32_t fa[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r) frag_j(a[r], t, fa[r]);
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    uint32_t fb[4];
    frag_l(b[n], t, fb);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      mma_f16(c[m][n], fa[2 * m][0], fa[2 * m + 1][0], fa[2 * m][1], fa[2 * m + 1][1], fb[0], fb[1]);
      mma_f16(c[m][n], fa[2 * m][2], fa[2 * m + 1][2], fa[2 * m][3], fa[2 * m + 1][3], fb[2], fb[3]);
    }
  }
}

// Adds the masked sums of a block to the diagonal of d (mk[r]: the block's row 8 r + lane / 4).
__device__ __forceinline__ void block_sum(float (&d)[4], const uint32_t (&c)[2][4][2],
                                          const uint32_t (&mk)[4], int t) {
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const uint32_t w = mk[r] >> t;
#pragma unroll
    for (int h = 0; h < 2; ++h)
      mma_f32(d, (w >> (8 * h)) & kPair, (w >> (8 * h + 4)) & kPair, c[r >> 1][2 * h][r & 1],
              c[r >> 1][2 * h + 1][r & 1]);
  }
}

// The sums gathered in d, each diagonal element once (this lane's part), and d cleared.
__device__ __forceinline__ uint32_t take_diag(float (&d)[4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const float v = (g >> 1) == t ? ((g & 1) ? d[1] : d[0]) : 0.0f;
  d[0] = d[1] = d[2] = d[3] = 0.0f;
  return (uint32_t)(v * kUnit);
}

// Edges (j, l), j in block J, l in block L >= J: adds |R_j & R_l|, and with MASK (m: a row's
// words, read from J on) |R_j & R_l & m| over j, l in m, to the diagonal of d.
template <bool MASK>
__device__ __forceinline__ void tri_block(const uint32_t* M, int W, int J, int L,
                                          const uint32_t* m, float (&d)[4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int sa = W - J, sb = W - L;
  const uint32_t* A = M + blk_off(J, W) - J + g * sa;
  const uint32_t* B = M + blk_off(L, W) - L + col_row(g) * sb;
  uint32_t mk[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    mk[r] = A[8 * r * sa + L];
    if (MASK) mk[r] = (m[J] >> (8 * r + g)) & 1u ? mk[r] & m[L] : 0u;
  }
  if (!__any_sync(kFull, (mk[0] | mk[1] | mk[2] | mk[3]) != 0u)) return;
  uint32_t c[2][4][2] = {};
  for (int w = L; w < W; ++w) {
    uint32_t a[4], b[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      a[r] = A[8 * r * sa + w];
      if (MASK) a[r] &= m[w];
      b[r] = B[4 * r * sb + w];
    }
    block_mma(c, a, b, t);
  }
  block_sum(d, c, mk, t);
}

// Blocks of a matrix from block q on, dealt to nw warps (this one is wi), longest sums first.
template <bool MASK>
__device__ uint64_t tri_blocks(const uint32_t* M, int W, int q, const uint32_t* m, int wi, int nw) {
  uint64_t acc = 0;
  float d[4] = {};
  int L = 0, J = wi;  // block (q + J, q + L), J <= L, in the order L, J
  for (int done = 0;;) {
    while (J > L) J -= ++L;
    if (q + L >= W) return acc + take_diag(d);
    tri_block<MASK>(M, W, q + J, q + L, m, d);
    J += nw;
    // a block adds at most 4 rows x 32 x 1024 to an element: exact below 2^24
    if (++done % 64 == 0) acc += take_diag(d);
  }
}

// Triangles of a matrix of at most 32 vertices, row i in lane i.  Up to kPopcN vertices row by
// row (8 clocks of popc each), above that one block, its operands by shuffle (24 steps of 8.5
// clocks and as many again of fragments).
constexpr int kPopcN = 16;
__device__ __forceinline__ uint32_t tri_word(uint32_t row, int n) {
  if (n <= kPopcN) {
    uint32_t c = 0;
    for (int j = 1; j < n - 1; j += 4) {  // (rows from n on are empty)
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const uint32_t r = __shfl_sync(kFull, row, j + h);
        if ((row >> (j + h)) & 1u) c += __popc(row & r);
      }
    }
    return c;
  }
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  uint32_t a[4], b[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    a[r] = __shfl_sync(kFull, row, 8 * r + g);
    b[r] = __shfl_sync(kFull, row, 4 * r + col_row(g));
  }
  uint32_t c[2][4][2] = {};
  float d[4] = {};
  block_mma(c, a, b, t);
  block_sum(d, c, a, t);
  return take_diag(d);
}

// The matrix induced on a set of n <= 32 vertices (lane w holds word w of the set), row r in
// lane r: lane b holds member b and one ballot gives a row.  ids: 32 entries of this warp.
__device__ uint32_t small_matrix(const uint32_t* M, int W, uint32_t word, int n, uint16_t* ids) {
  const int lane = threadIdx.x & 31;
  const int cnt = __popc(word);
  int inc = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, inc, o);
    if (lane >= o) inc += y;
  }
  for (unsigned nz = __ballot_sync(kFull, word != 0u); nz; nz &= nz - 1) {
    const int w = __ffs(nz) - 1;
    const uint32_t x = __shfl_sync(kFull, word, w);
    const int e = __shfl_sync(kFull, inc - cnt, w);
    if ((x >> lane) & 1u) ids[e + __popc(x & lanemask_lt())] = (uint16_t)(32 * w + lane);
  }
  __syncwarp();
  const int id = lane < n ? (int)ids[lane] : 0;
  const uint32_t bit = lane < n ? 1u << (id & 31) : 0u;
  const int base = tri_row_off(id, W) - (id >> 5);
  const uint32_t* Mw = M + (id >> 5);
  uint32_t mine = 0;
  for (int r = 0; r < n; ++r) {
    // a word below the row's own block belongs to an earlier row: masked out below
    const uint32_t y = __ballot_sync(kFull, (Mw[__shfl_sync(kFull, base, r)] & bit) != 0u);
    if (lane == r) mine = y;
  }
  __syncwarp();
  return mine & (0xFFFFFFFEu << lane);  // members after r
}

// How the members of a row (R_i) are taken out of another row's words: per word of R_i, the
// word, the five move masks of a bit compress (Hacker's Delight, 7-4: each step moves the
// bits of its mask down by 1, 2, 4, 8, 16), and the number of members before it and in it.
struct PickWord {
  uint32_t m, mv[5];
  int pos, cnt;
};
static_assert(sizeof(PickWord) == 32, "read as two uint4");

// Word `lane` of row i of a matrix (0 outside the row).
__device__ __forceinline__ uint32_t row_word(const uint32_t* M, int W, int i) {
  const int lane = threadIdx.x & 31, q = i >> 5;
  return lane >= q && lane < W ? M[tri_row_off(i, W) + lane - q] : 0u;
}

// Prepares the members of a set of rows (lane w: word w of it): the picks (one warp of the
// team) and the ids (idx, by nw warps).  Returns their number.
__device__ int set_members(int W, uint32_t word, uint16_t* idx, PickWord* pick, int wi, int nw) {
  const int lane = threadIdx.x & 31;
  const int cnt = __popc(word);
  int inc = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, inc, o);
    if (lane >= o) inc += y;
  }
  if (wi == 0 && lane < W) {
    PickWord p;
    p.m = word;
    p.pos = inc - cnt;
    p.cnt = cnt;
    uint32_t mk = ~word << 1, m = word;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      uint32_t mp = mk ^ (mk << 1);
      mp ^= mp << 2;
      mp ^= mp << 4;
      mp ^= mp << 8;
      mp ^= mp << 16;
      p.mv[k] = mp & m;
      m = (m ^ p.mv[k]) | (p.mv[k] >> (1 << k));
      mk &= ~mp;
    }
    pick[lane] = p;
  }
  for (int w = wi; w < W; w += nw) {
    const uint32_t x = __shfl_sync(kFull, word, w);
    const int e = __shfl_sync(kFull, inc - cnt, w);
    if ((x >> lane) & 1u) idx[e + __popc(x & lanemask_lt())] = (uint16_t)(32 * w + lane);
  }
  return __shfl_sync(kFull, inc, 31);
}

// The matrix induced on R_i, in the same triangular form (C, W2 = ceil(n / 32) words), by
// nw warps: lane r of a warp takes row 32 J + r of it, compresses the words of that
// member's row by the picks and appends the bits.  (One ballot per 32 members and row, the
// lanes holding the members, cost 2.5 to 4 times as many instructions.)
__device__ void compress(const uint32_t* M, int W, const uint16_t* idx, const PickWord* pick,
                         int n, uint32_t* C, int wi, int nw) {
  const int lane = threadIdx.x & 31, W2 = (n + 31) >> 5;
  for (int J = wi; J < W2; J += nw) {
    const bool live = 32 * J + lane < n;
    const int id = live ? (int)idx[32 * J + lane] : 0;
    const int q = live ? id >> 5 : 32;  // words of the row from q on (bits after id only)
    const uint32_t* row = M + tri_row_off(id, W) - (id >> 5);
    uint32_t* out = C + blk_off(J, W2) + lane * (W2 - J);  // words J .. W2 - 1 of the row
    int w = (int)idx[32 * J] >> 5;  // the first word that holds a member of block J or later
    uint32_t bits = 0;
    int sh = pick[w].pos - 32 * J;  // < 0: members of earlier blocks, no bits of these rows
    for (; w < W; ++w) {
      const uint4 p0 = reinterpret_cast<const uint4*>(pick + w)[0];
      const uint4 p1 = reinterpret_cast<const uint4*>(pick + w)[1];
      if (p0.x == 0u) continue;
      uint32_t x = w >= q ? row[w] & p0.x : 0u, t;
      t = x & p0.y; x = (x ^ t) | (t >> 1);
      t = x & p0.z; x = (x ^ t) | (t >> 2);
      t = x & p0.w; x = (x ^ t) | (t >> 4);
      t = x & p1.x; x = (x ^ t) | (t >> 8);
      t = x & p1.y; x = (x ^ t) | (t >> 16);
      const int cnt = (int)p1.w;
      if (sh < 0) {  // first word: drop the bits before block J (all zero)
        x >>= -sh;
        sh += cnt;
        bits = x;
        continue;
      }
      bits |= x << sh;
      sh += cnt;
      if (sh >= 32) {
        *out++ = bits;
        sh -= 32;
        bits = sh ? x >> (cnt - sh) : 0u;
      }
    }
    if (sh > 0) *out = bits;
  }
}

// Cliques of D vertices in the rows' subset m of a one-word matrix.
template <int D>
__device__ uint64_t word_cliques(const uint32_t* rows, uint32_t m) {
  if constexpr (D == 1) {
    return (uint64_t)__popc(m);
  } else {
    uint64_t acc = 0;
    while (m) {
      const int l = __ffs(m) - 1;
      m &= m - 1;
      acc += word_cliques<D - 1>(rows, m & rows[l]);
    }
    return acc;
  }
}

// D-cliques (D = 3, 4, 5) among a set of n <= 32 vertices of a matrix, by one warp; tmp: 32
// words, ids: 32 entries of this warp.
template <int D>
__device__ __forceinline__ uint64_t set_cliques(const uint32_t* M, int W, uint32_t word, int n,
                                                uint16_t* ids, uint32_t* tmp) {
  const uint32_t row = small_matrix(M, W, word, n, ids);
  if constexpr (D == 3) {
    return tri_word(row, n);
  } else {
    tmp[threadIdx.x & 31] = row;
    __syncwarp();
    const uint64_t r = word_cliques<D - 1>(tmp, row);
    __syncwarp();
    return r;
  }
}

constexpr int kOwnN = 128;             // longest row one warp takes by itself
constexpr int kOwnWords = 16 * 4 * 5;  // its matrix

// Scratch of a warp: the matrix induced on a row of up to kOwnN members and what building it
// takes, 32 words of masks, ids of a small set; K >= 6: the same for a row of that matrix.
struct InduceScratch {
  PickWord pick[32];
  uint32_t mat[kOwnWords];
  uint16_t idx[kOwnN];
};
template <int LEVELS>
struct WarpScratch {
  InduceScratch level[LEVELS];
  uint32_t tmp[32];
  uint16_t ids[32];
};
static_assert(sizeof(WarpScratch<1>) % 32 == 0 && sizeof(WarpScratch<2>) % 32 == 0,
              "picks are read 16 bytes at a time");

// D-cliques (D = 3, 4, 5) of the matrix C of n vertices, by nw warps.  D = 4: for each row j
// the triangles inside it: of up to 32 members as a matrix in registers, of up to kOwnN as
// one in `in` (null: none), else as a mask over C.  D = 5: for each row j the 4-cliques
// inside it, or for each edge (j, l) the triangles inside R_j & R_l.
template <int D>
__device__ uint64_t matrix_cliques(const uint32_t* C, int n, int wi, int nw, InduceScratch* in,
                                   uint16_t* ids, uint32_t* tmp) {
  const int lane = threadIdx.x & 31, W = (n + 31) >> 5;
  if constexpr (D == 3) {
    return tri_blocks<false>(C, W, 0, nullptr, wi, nw);
  } else {
    uint64_t acc = 0;
    for (int j = wi; j + D - 1 < n; j += nw) {
      const int q = j >> 5;
      const uint32_t word = row_word(C, W, j);
      const int nj = (int)__reduce_add_sync(kFull, (unsigned)__popc(word));
      if (nj < D - 1) continue;
      if (nj <= 32) {
        acc += set_cliques<D - 1>(C, W, word, nj, ids, tmp);
      } else if (in && nj <= kOwnN) {
        set_members(W, word, in->idx, in->pick, 0, 1);
        __syncwarp();
        compress(C, W, in->idx, in->pick, nj, in->mat, 0, 1);
        __syncwarp();
        acc += matrix_cliques<D - 1>(in->mat, nj, 0, 1, nullptr, ids, tmp);
        __syncwarp();
      } else if constexpr (D == 4) {
        acc += tri_blocks<true>(C, W, q, C + tri_row_off(j, W) - q, 0, 1);
      } else {
        for (unsigned nz = __ballot_sync(kFull, word != 0u); nz; nz &= nz - 1) {
          const int ql = __ffs(nz) - 1;
          for (uint32_t bits = __shfl_sync(kFull, word, ql); bits; bits &= bits - 1) {
            const int l = 32 * ql + __ffs(bits) - 1;
            const uint32_t m2 = word & row_word(C, W, l);
            const int nl = (int)__reduce_add_sync(kFull, (unsigned)__popc(m2));
            if (nl < 3) continue;
            if (nl <= 32) {
              acc += set_cliques<3>(C, W, m2, nl, ids, tmp);
            } else {
              __syncwarp();
              tmp[lane] = m2;
              __syncwarp();
              acc += tri_blocks<true>(C, W, ql, tmp, 0, 1);
            }
          }
        }
      }
    }
    return acc;
  }
}

// Totals: one sum per thread, or (o.gid) a task's total to its graph's output.  Called by all
// lanes of a warp.
__device__ __forceinline__ void emit_rows(const GOut& o, int32_t v, uint64_t part, uint64_t& acc) {
  if (!o.gid) {
    acc += part;
    return;
  }
  const uint64_t w = warp_sum_u64(part);
  if ((threadIdx.x & 31) == 0 && w)
    atomicAdd(&o.out[(long long)o.gid[v] * o.stride + o.slot], (unsigned long long)w);
}

struct RowTasks {
  const longlong2* dptr;
  const int64_t* roff;
  const uint32_t* rows;
  const int32_t* list;  // task t: list[t], or list[-t] when `down`
  const unsigned long long* n;
  int down;
  int wcap;  // words of a row the CTA's shared memory is laid out for (word tasks: tasks
             // per claim, at most 32)
};

constexpr int kTeam = 4;                  // warps of a team
constexpr int kTeamN = 512;               // longest row a team takes
// (the 16-warp CTAs of wide tasks have no room for a second level: masks)
template <int K, int WARPS>
using TaskScratch = WarpScratch<(K >= 6 && WARPS == kTeam ? 2 : 1)>;

// Words of shared memory of a CTA of row tasks: the task's matrix; K >= 5: per team a
// matrix and ids for rows up to kTeamN (together one for the longest row) and picks, the
// list of rows too long for a warp, and each warp's scratch.
__host__ __device__ constexpr int matrix_words(int W) { return 16 * W * (W + 1); }
__host__ __device__ constexpr int team_matrix_words(int W) {
  return matrix_words(W < kTeamN / 32 ? W : kTeamN / 32);
}
template <int K, int WARPS>
constexpr int team_words(int W) {
  return K == 4 ? matrix_words(W)
                : matrix_words(W) + WARPS / kTeam * (team_matrix_words(W) + 8 * 32 + kTeamN / 2) +
                      16 * W + WARPS * (int)sizeof(TaskScratch<K, WARPS>) / 4;
}

__device__ __forceinline__ void team_sync(int team) {  // barrier 0 is __syncthreads
  asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(32 * kTeam) : "memory");
}

// Parts a task's rows are dealt to (k >= 5): a task of 256 members takes one CTA milliseconds
// at k = 6, and a graph has few of the largest.  R-MAT s16 6-clique 16.8 / 9.9 / 10.2 ms with
// 1 / 4 / 8 parts, the 16-warp tasks of the s20 5-clique 7.4 / 5.9 / 6.2 ms with 1 / 4 / 8.
constexpr int team_parts(int K, int NT) {
  return K == 4 ? 1 : (K == 5 ? (NT == 128 ? 2 : 4) : (K == 6 ? 4 : 8));
}

// CTAs per SM the registers are cut for (K = 4: 8-warp CTAs, K >= 6 spills below 168).
constexpr int team_ctas(int K, int NT) {
  return NT == 128 ? (K == 5 ? 5 : (K == 4 ? 4 : 3)) : (K == 4 ? 2 : 1);
}

// Tasks of more than 32 out-neighbours, one CTA each: the (K - 1)-cliques of the task's
// matrix.  K >= 5: the (K - 2)-cliques of the matrix induced on each row, a row of up to
// kOwnN members by one warp, of up to kTeamN by a team of four, longer ones by the CTA.
template <int K, int NT>
__global__ void __launch_bounds__(NT, team_ctas(K, NT)) k_rows_team(RowTasks t, unsigned long long* head,
                                                  unsigned long long* count, GOut o) {
  extern __shared__ __align__(16) uint32_t M[];
  __shared__ long long task_s;
  __shared__ int next_i, n_long, next_long, n_huge, team_x[NT / 32 / kTeam];
  constexpr int kWarps = NT / 32, kTeams = kWarps / kTeam;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kParts = team_parts(K, NT);
  let_next_start();
  const long long nt = (long long)*t.n;
  uint64_t total = 0;
  if (tid == 0) task_s = (long long)atomicAdd(head, 1ull);
  __syncthreads();
  for (;;) {
    const long long ti = task_s;
    if (ti >= nt * kParts) break;
    // from the list's end: its start holds the low ranks, the smallest tasks
    const long long at = nt - 1 - ti / kParts;
    const int part = (int)(ti % kParts);  // of the task's rows: part, part + kParts, ..
    const int32_t v = t.down ? t.list[-at] : t.list[at];
    uint64_t acc = 0;
    const longlong2 d = ldg_ll2(t.dptr + v);
    const int s = (int)(d.y - d.x), W = (s + 31) >> 5;
    const int used = tri_words(s), all = matrix_words(W);  // the last block padded to 32 rows
    const uint4* src = reinterpret_cast<const uint4*>(t.rows + t.roff[v]);
    for (int x = tid; 4 * x < all; x += NT) {
      uint4 y = make_uint4(0, 0, 0, 0);
      if (4 * x < used) y = __ldcs(src + x);
      if (4 * x + 1 >= used) y.y = 0;
      if (4 * x + 2 >= used) y.z = 0;
      if (4 * x + 3 >= used) y.w = 0;
      reinterpret_cast<uint4*>(M)[x] = y;
    }
    if (tid == 0) next_i = 0, n_long = 0, next_long = 0, n_huge = 0;
    __syncthreads();
    if (tid == 0) task_s = (long long)atomicAdd(head, 1ull);
    if constexpr (K == 4) {
      acc += tri_blocks<false>(M, W, 0, nullptr, warp, kWarps);
    } else {
      const int tm = team_matrix_words(t.wcap), team = warp / kTeam, tw = warp % kTeam;
      uint32_t* Cs = M + matrix_words(t.wcap);  // the teams' matrices, then their picks, ids
      PickWord* picks = reinterpret_cast<PickWord*>(Cs + kTeams * tm);
      uint16_t* idxs = reinterpret_cast<uint16_t*>(picks + kTeams * 32);
      uint16_t* longs = idxs + kTeams * kTeamN;  // rows of <= kTeamN from the front, others
      const int lcap = 32 * t.wcap;              // from the back
      using Scratch = TaskScratch<K, kWarps>;
      Scratch& ws = reinterpret_cast<Scratch*>(longs + lcap)[warp];
      InduceScratch& own = ws.level[0];
      constexpr bool kDeep = sizeof(Scratch) == sizeof(WarpScratch<2>);
      InduceScratch* deep = kDeep ? &ws.level[kDeep ? 1 : 0] : nullptr;
      for (;;) {
        int i = 0;
        if (lane == 0) i = atomicAdd(&next_i, kParts);
        i = __shfl_sync(kFull, i, 0) + part;
        if (i + K - 2 >= s) break;
        const uint32_t word = row_word(M, W, i);
        const int n = (int)__reduce_add_sync(kFull, (unsigned)__popc(word));
        if (n < K - 2) continue;
        if (n <= 32) {
          acc += set_cliques<K - 2>(M, W, word, n, ws.ids, ws.tmp);
          continue;
        }
        if (n > kOwnN) {
          if (lane == 0) {
            if (n <= kTeamN) longs[atomicAdd(&n_long, 1)] = (uint16_t)i;
            else longs[lcap - 1 - atomicAdd(&n_huge, 1)] = (uint16_t)i;
          }
          continue;
        }
        set_members(W, word, own.idx, own.pick, 0, 1);
        __syncwarp();
        compress(M, W, own.idx, own.pick, n, own.mat, 0, 1);
        __syncwarp();
        acc += matrix_cliques<K - 2>(own.mat, n, 0, 1, deep, ws.ids, ws.tmp);
        __syncwarp();
      }
      __syncthreads();
      for (;;) {
        team_sync(team);  // the team is done with its last row
        if (tw == 0 && lane == 0) team_x[team] = atomicAdd(&next_long, 1);
        team_sync(team);
        const int x = team_x[team];
        if (x >= n_long) break;
        uint32_t* C = Cs + team * tm;
        const int n = set_members(W, row_word(M, W, longs[x]), idxs + team * kTeamN,
                                  picks + 32 * team, tw, kTeam);
        team_sync(team);
        compress(M, W, idxs + team * kTeamN, picks + 32 * team, n, C, tw, kTeam);
        team_sync(team);
        acc += matrix_cliques<K - 2>(C, n, tw, kTeam, deep, ws.ids, ws.tmp);
      }
      if constexpr (kTeams * team_matrix_words(32) >= matrix_words(32)) {
        const int nh = n_huge;
        if (nh) __syncthreads();  // every team is done
        for (int x = 0; x < nh; ++x) {
          const int n = set_members(W, row_word(M, W, longs[lcap - 1 - x]), idxs, picks, warp,
                                    kWarps);
          __syncthreads();
          compress(M, W, idxs, picks, n, Cs, warp, kWarps);
          __syncthreads();
          acc += matrix_cliques<K - 2>(Cs, n, warp, kWarps, deep, ws.ids, ws.tmp);
          __syncthreads();
        }
      }
    }
    emit_rows(o, v, acc, total);
    __syncthreads();
  }
  total = warp_sum_u64(total);
  if (lane == 0 && total) atomicAdd(count, (unsigned long long)total);
  wait_for_previous();
}

// Tasks of up to 32 out-neighbours, a warp each, lane i holding row i.  K = 4: one block on
// the tensor cores, its operands by shuffle.
constexpr int kWordThreads = 256;
template <int K>
__device__ uint64_t word_tasks(const RowTasks& t, unsigned long long* head, const GOut& o,
                               uint32_t* rows_s) {
  const int lane = threadIdx.x & 31;
  uint32_t* mine = rows_s + (threadIdx.x & ~31);
  const long long nt = (long long)*t.n;
  uint64_t acc = 0;
  for (;;) {
    long long base = 0;
    if (lane == 0) base = (long long)atomicAdd(head, (unsigned long long)t.wcap);
    base = __shfl_sync(kFull, base, 0);
    if (base >= nt) break;
    const int n = nt - base < t.wcap ? (int)(nt - base) : t.wcap;
    int s = 0;
    int32_t v = 0;
    long long off = 0;
    if (lane < n) {
      v = t.down ? t.list[-(base + lane)] : t.list[base + lane];
      const longlong2 d = ldg_ll2(t.dptr + v);
      s = (int)(d.y - d.x);
      off = t.roff[v];
    }
    int sx = __shfl_sync(kFull, s, 0);
    long long ox = __shfl_sync(kFull, off, 0);
    uint32_t next = lane < sx ? __ldcs(t.rows + ox + lane) : 0u;
    for (int x = 0; x < n; ++x) {
      const uint32_t r = next;
      const int sc = sx;
      if (x + 1 < n) {  // the next task's rows are in flight while this one is counted
        sx = __shfl_sync(kFull, s, x + 1);
        ox = __shfl_sync(kFull, off, x + 1);
        next = lane < sx ? __ldcs(t.rows + ox + lane) : 0u;
      }
      if (sc < K - 1) continue;
      if constexpr (K == 4) {
        emit_rows(o, __shfl_sync(kFull, v, x), tri_word(r, sc), acc);
      } else {
        mine[lane] = r;
        __syncwarp();
        const uint64_t c = word_cliques<K - 2>(mine, r);
        __syncwarp();
        emit_rows(o, __shfl_sync(kFull, v, x), c, acc);
      }
    }
  }
  return acc;
}

// Tasks of up to 8 out-neighbours, four to a warp, lane l of a group holding row l.
template <int K>
__device__ uint64_t group_tasks(const RowTasks& t, unsigned long long* head, const GOut& o,
                                uint32_t* rows_s) {
  const int lane = threadIdx.x & 31, l8 = lane & 7, g0 = lane & 24;
  const uint32_t* mine = rows_s + (threadIdx.x & ~7);
  const long long nt = (long long)*t.n;
  uint64_t acc = 0;
  for (;;) {
    long long base = 0;
    if (lane == 0) base = (long long)atomicAdd(head, (unsigned long long)t.wcap);
    base = __shfl_sync(kFull, base, 0);
    if (base >= nt) break;
    const int n = nt - base < t.wcap ? (int)(nt - base) : t.wcap;
    int s = 0;
    int32_t v = 0;
    long long off = 0;
    if (lane < n) {
      v = t.list[base + lane];
      const longlong2 d = ldg_ll2(t.dptr + v);
      s = (int)(d.y - d.x);
      off = t.roff[v];
    }
    for (int x = 0; x < n; x += 4) {
      const int src = x + (lane >> 3);  // (lanes past n hold s = 0)
      const int sc = __shfl_sync(kFull, s, src);
      const long long ro = __shfl_sync(kFull, off, src);
      const uint32_t r = l8 < sc ? __ldcs(t.rows + ro + l8) : 0u;
      uint32_t c = 0;
      if constexpr (K == 4) {
#pragma unroll
        for (int j = 1; j < 7; ++j) {  // the last two rows hold no pair
          const uint32_t rj = __shfl_sync(kFull, r, g0 + j);
          if ((r >> j) & 1u) c += __popc(r & rj);
        }
      } else {
        rows_s[threadIdx.x] = r;
        __syncwarp();
        c = (uint32_t)word_cliques<K - 2>(mine, r);
        __syncwarp();
      }
      if (o.gid) {
        c += __shfl_xor_sync(kFull, c, 1);
        c += __shfl_xor_sync(kFull, c, 2);
        c += __shfl_xor_sync(kFull, c, 4);
        const int32_t vx = __shfl_sync(kFull, v, src);
        if (l8 == 0 && c)
          atomicAdd(&o.out[(long long)o.gid[vx] * o.stride + o.slot], (unsigned long long)c);
      } else {
        acc += c;
      }
    }
  }
  return acc;
}

// The narrow tasks: KIND 1 word tasks, 2 group tasks, 3 both in one launch.  A launch costs a
// call 3 us; with many tasks the group tasks' own 32 registers (64 warps per SM against 32)
// are worth more: 4,096 Barabasi-Albert graphs 1.52 against 1.59 ms.
template <int K, int KIND>
__global__ void __launch_bounds__(kWordThreads, KIND == 3 ? 4 : 1)
    k_rows_narrow(RowTasks word, RowTasks group, OwnHeads* heads, unsigned long long* count,
                  GOut o) {
  __shared__ uint32_t rows_s[kWordThreads];
  let_next_start();
  uint64_t acc = 0;
  if (KIND & 1) acc += word_tasks<K>(word, &heads->word, o, rows_s);
  if (KIND & 2) acc += group_tasks<K>(group, &heads->group, o, rows_s);
  acc = warp_sum_u64(acc);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd(count, (unsigned long long)acc);
  wait_for_previous();
}
constexpr int64_t kOneNarrow = int64_t(1) << 17;  // tasks up to which both kinds share a launch

// Grid of a persistent kernel: every CTA the chip holds.
template <class F>
cudaError_t full_grid(F fn, int threads, int smem, int num_sms, int* grid) {
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
  *grid = std::max(per_sm, 1) * num_sms;
  return e;
}

static_assert(4 * team_words<7, 16>(kRowsCap / 32) <= 226 * 1024, "wide tasks fit an SM");

template <int K, int NT>
cudaError_t launch_team(const DevGraph& g, RowTasks t, int cap, unsigned long long* head,
                        unsigned long long* count, int num_sms, cudaStream_t s, const GOut& o,
                        bool first) {
  t.wcap = (int)((std::min<int64_t>(g.max_out, cap) + 31) / 32);
  const int smem = 4 * team_words<K, NT / 32>(t.wcap);
  int grid = 0, dev = 0;
  // the shared-memory opt-in of the widest layout, once per device
  static std::atomic<unsigned long long> opted{0};
  cudaError_t e = cudaGetDevice(&dev);
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (e == cudaSuccess && !(opted.load(std::memory_order_acquire) & bit)) {
    e = cudaFuncSetAttribute(k_rows_team<K, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             4 * team_words<K, NT / 32>(cap / 32));
    if (e == cudaSuccess) opted.fetch_or(bit, std::memory_order_acq_rel);
  }
  if (e == cudaSuccess) e = full_grid(k_rows_team<K, NT>, NT, smem, num_sms, &grid);
  if (e != cudaSuccess) return e;
  grid = (int)std::min<int64_t>(grid, g.nv * team_parts(K, NT));
  return launch_next(first, k_rows_team<K, NT>, grid, NT, smem, s, t, head, count, o);
}

template <int K>
cudaError_t launch_rows_k(const DevGraph& g, const uint32_t* rows, OwnHeads* heads,
                          unsigned long long* count, int num_sms, cudaStream_t s, const GOut& o,
                          bool first) {
  const unsigned long long* rn = g.rn;
  cudaError_t e = cudaSuccess;
  if (g.max_out > kRowsMid) {
    const RowTasks t{g.dptr, g.roff, rows, g.rtask + 2 * g.nv - 1, rn + 4, 1, 0};
    e = launch_team<K, K == 4 ? 256 : 512>(g, t, kRowsCap, &heads->wide, count, num_sms, s, o, first);
    first = false;
  }
  if (e == cudaSuccess && g.max_out > 32) {
    const RowTasks t{g.dptr, g.roff, rows, g.rtask + g.nv, rn + 3, 0, 0};
    e = launch_team<K, 128>(g, t, kRowsMid, &heads->team, count, num_sms, s, o, first);
    first = false;
  }
  if (e != cudaSuccess) return e;
  // at most `roots` word and group tasks; claims small enough that every warp has a few
  const int64_t roots = std::max<int64_t>(g.n_roots[1], 1);
  auto narrow = [&](auto kernel, int per_warp) -> cudaError_t {
    int grid = 0;
    const cudaError_t r = full_grid(kernel, kWordThreads, 0, num_sms, &grid);
    if (r != cudaSuccess) return r;
    constexpr int kWarps = kWordThreads / 32;
    grid = (int)std::min<int64_t>(grid, (roots + kWarps * per_warp - 1) / (kWarps * per_warp));
    const int64_t claim = std::min<int64_t>(32, roots / (4 * kWarps * (int64_t)grid));
    const RowTasks word{g.dptr, g.roff, rows, g.rtask + g.nv - 1, rn + 2, 1,
                        (int)std::max<int64_t>(claim, 1)};
    const RowTasks group{g.dptr, g.roff, rows, g.rtask, rn + 1, 0, (int)std::max<int64_t>(claim, 4)};
    const bool f = first;
    first = false;
    return launch_next(f, kernel, grid, kWordThreads, 0, s, word, group, heads, count, o);
  };
  if (g.max_out <= 8) return narrow(k_rows_narrow<K, 2>, 4);
  if (roots <= kOneNarrow) return narrow(k_rows_narrow<K, 3>, 1);
  e = narrow(k_rows_narrow<K, 1>, 1);
  return e == cudaSuccess ? narrow(k_rows_narrow<K, 2>, 4) : e;
}

cudaError_t build_rows_index(const DevGraph& g, cudaStream_t s) {
  int64_t* roff = nullptr;
  int32_t* rtask = nullptr;
  unsigned long long* rn = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&roff, sizeof(int64_t) * (size_t)g.nv, s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&rtask, sizeof(int32_t) * 2 * (size_t)g.nv, s);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&rn, sizeof(*rn) * 5, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(rn, 0, sizeof(*rn) * 5, s);
  if (e == cudaSuccess) {
    const int64_t blocks = std::min<int64_t>((g.nv + 255) / 256, 65536);
    k_rows_index<<<(unsigned)blocks, 256, 0, s>>>(g.dptr, g.nv, roff, rtask, rtask + g.nv, rn);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    if (roff) cudaFreeAsync(roff, s);
    if (rtask) cudaFreeAsync(rtask, s);
    if (rn) cudaFreeAsync(rn, s);
    return e;
  }
  g.roff = roff;
  g.rtask = rtask;
  g.rn = rn;
  return cudaSuccess;
}

}  // namespace

cudaError_t launch_owner_count(const DevGraph& g, OwnHeads* heads, unsigned long long* count,
                               int num_sms, cudaStream_t s) {
  return launch_owner<kOwnCount>(g, OwnArgs{}, heads, count, num_sms, s);
}

cudaError_t launch_owner_multi(const DevGraph& g, uint32_t* rows, unsigned* epart,
                               OwnHeads* heads, int num_sms, cudaStream_t s) {
  OwnArgs a{};
  a.roff = g.roff;
  a.rows = rows;
  a.epart = epart;
  return launch_owner<kOwnMulti>(g, a, heads, nullptr, num_sms, s);
}

cudaError_t launch_owner_part(const DevGraph& g, OwnHeads* heads, unsigned* epart, int num_sms,
                              cudaStream_t s) {
  OwnArgs a{};
  a.epart = epart;
  return launch_owner<kOwnPart>(g, a, heads, nullptr, num_sms, s);
}

cudaError_t ensure_rows_index(const DevGraph& g, cudaStream_t s) {
  return build_once(
      g, s, [&] { return g.roff || g.nv == 0; }, [&] { return build_rows_index(g, s); });
}

cudaError_t reserve_rows(const DevGraph& g, uint32_t** rows, int64_t* cap, bool* fits,
                         cudaStream_t s) {
  const int64_t words = g.row_store_words + 4;
  cudaError_t e = ensure_rows_index(g, s);
  if (e == cudaSuccess && (!*rows || *cap < words)) {
    if (*rows) cudaFreeAsync(*rows, s);
    *rows = nullptr;
    *cap = 0;
    // test hook: XGM_ROW_STORE_CAP is the number of words from which there is no room
    const char* room = std::getenv("XGM_ROW_STORE_CAP");
    e = room && words > std::atoll(room) ? cudaErrorMemoryAllocation
                                         : cudaMallocAsync((void**)rows, sizeof(uint32_t) * words, s);
    if (e == cudaSuccess) *cap = words;
  }
  *fits = e == cudaSuccess;
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  return cudaSuccess;
}

cudaError_t launch_owner_rows(const DevGraph& g, uint32_t* rows, OwnHeads* heads, int num_sms,
                              cudaStream_t s) {
  OwnArgs a{};
  a.roff = g.roff;
  a.rows = rows;
  return launch_owner<kOwnRows>(g, a, heads, nullptr, num_sms, s);
}

cudaError_t launch_rows_count(int k, const DevGraph& g, const uint32_t* rows, OwnHeads* heads,
                              unsigned long long* count, int num_sms, cudaStream_t s,
                              const GOut& o, bool next) {
  if (g.nv == 0) return cudaSuccess;
  switch (k) {
    case 4: return launch_rows_k<4>(g, rows, heads, count, num_sms, s, o, !next);
    case 5: return launch_rows_k<5>(g, rows, heads, count, num_sms, s, o, !next);
    case 6: return launch_rows_k<6>(g, rows, heads, count, num_sms, s, o, !next);
    case 7: return launch_rows_k<7>(g, rows, heads, count, num_sms, s, o, !next);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace xgm
