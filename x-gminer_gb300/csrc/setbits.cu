// Bitmap form of set-operation programs (setprog.cuh): tasks whose v0 has at most 1,024
// neighbours, for programs whose operands live in N(v0) (prog_lut).
//
// GLUMIN's LUT kernels (GM_LUT_kernels/P*.yml.cuh, codegen_LUT.cuh) keep the adjacency
// among N(v0) as bit rows and run the plan on them.  Here a program is first folded to
// three terms (prog_terms): the v2 candidates, the v3 candidates and the counted set, each
// the AND of N(v0), of rows or complements of rows of v1, v2, v3, of a prefix (N(v0) is
// sorted, so a bound is an index) and of cleared bits.  A word of a term is then a handful
// of instructions whatever the program's slots, operations and levels were.
//
// The work is the steps (v0, v1, v2), and one unit of it is a part of one v0's steps, all
// of nearly the same size: plan_units deals a v0 to parts by the larger of its list sum
// (a stream program's v2 run over N(v1) \ N(v0)) and d(v0)^2.  No task is split or queued
// at run time.
//
// - k_bits_warp, d(v0) <= 32: a warp a unit, a lane a step, sets in one register each.
// - k_bits_cta, 33 <= d(v0) <= 1,024: a block a unit.  N(v0)'s rows are copied from the
//   graph's stored rows into shared memory, 16 bytes times an odd number a row, so that 32
//   lanes that each read 16 bytes of another row meet no bank twice.  Up to 128 neighbours
//   (four words) a lane still takes a step: 1.14 ms on the workload below, 1.39 ms with a
//   warp a step from 33 on.  Above, a warp takes a step: a word a lane for the terms, a v3
//   a lane for the count.  Blocks of 256 threads up to 256 neighbours, of 1,024 above, where
//   the rows leave room for one block an SM (the line at 384: 2.00 against 1.93 ms).
//
// - k_bits_map, a stream program's v0 of 33 to 256 neighbours in place of k_bits_cta, on
//   graphs with enough of them.
//
// The row of a v2 outside N(v0): up to 256 neighbours the rows of all two-hop vertices are
// built at once, by streaming the lists of N(v0)'s members into a table, whose set bits are
// the steps.  Above, where the table would not fit, or where few tasks have steps, N(v2) is
// looked up in a hash table of N(v0), a step at a time.
//
// What bounds them: instruction issue (60-80 %, the integer pipe).  P7 on R-MAT scale 12
// (5.9 M steps, 119 M v3 candidates): 6.40 ms when k_setlut and k_setprog interpreted the
// operations with binary searches in lists, 1.97 ms with a look-up of every v2's list (400 M
// look-ups), 1.05 ms with the tables; P15 on Erdos-Renyi 2^16 2.25, 1.25, 0.67 ms.
// R-MAT scale 9 P7 1.84 ms -> 0.12, where a few heavy tasks were the time; P10 on
// Erdos-Renyi 2^16 0.83 -> 0.24 ms.
#include <algorithm>
#include <atomic>

#include "api_internal.h"
#include "graph.cuh"
#include "prim.cuh"
#include "setprog.cuh"

namespace xgm {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kWarpDeg = 32;    // k_bits_warp
constexpr int kLaneDeg = 128;   // k_bits_cta: a lane a step up to here, a warp a step above
constexpr int kMidDeg = 256;    // k_bits_cta, blocks of 256 threads
constexpr int kTopDeg = 1024;   // k_bits_cta, blocks of 1,024 threads
constexpr int kTopThreads = 1024;
constexpr int kListCap = 384;   // v3 candidates a warp lists at once
constexpr int kBatch = 16;      // steps a warp decodes at once where a warp takes a step
constexpr int64_t kRowBudget = int64_t(4) << 30;  // bytes of stored rows at most

// Shared memory of a block of k_bits_cta whose v0 has at most `deg` neighbours (byte
// offsets; the rows come first).
struct CtaLayout {
  int deg, buckets;
  int n0, key, pos, rel, off, warp, per_warp, bytes;
};

struct BitArgs {
  const int64_t* rowptr;
  const int32_t* col;
  const uint32_t* rows;
  const int64_t* roff;
  const int4* units;                // {v0, part, parts, -}
  const unsigned long long* un;     // [class] units, [3] units of v0s with several
  unsigned long long* head;         // the class's next unit
  unsigned long long* total;
  int64_t* split_out;               // statistics: un[3] (or null)
  BitPlan p;
  int cls;
  int items;  // list entries a block of k_bits_map takes at a time
  CtaLayout lay;
};

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

__device__ __forceinline__ bool member(const int32_t* b, int len, int x) {
  const int i = lower_index(b, len, x);
  return i < len && b[i] == x;
}

// Row j's part of a term: r where the row is intersected, ~r where it is taken away, all
// ones where it has no part (one three-input operation).
__device__ __forceinline__ uint32_t part(const BitTerm& t, int j, uint32_t r) {
  const uint32_t off = (t.pos >> j) & 1 ? 0u : 0xffffffffu;
  const uint32_t on = (t.neg >> j) & 1 ? 0u : 0xffffffffu;
  return (r | off) & (~r | on);
}

// Bits below lim of the word that starts at lo.
__device__ __forceinline__ uint32_t below(int lim, int lo) {
  uint32_t m;
  asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(m) : "r"(max(lim - lo, 0)));
  return m;
}

// Hash table of N(v0): buckets of four keys, read by one 16-byte load.  A key lies in its
// own bucket or, with that one full, in one of the next; `probes` is the most buckets any
// key lies from its own, plus one (1 but for a few in a hundred tables: at most half a key
// a bucket on average), so that no look-up runs longer than another and lanes stay together.
struct Table {
  int32_t* key;
  uint16_t* pos;
  int mask;   // buckets - 1
  int shift;  // 32 - log2(buckets)
};

__device__ __forceinline__ uint32_t bucket_of(const Table& t, int z) {
  return ((uint32_t)z * 2654435761u) >> t.shift;
}

__device__ __forceinline__ int in_bucket(const Table& t, uint32_t h, int z, int at) {
  const int4 q = ((const int4*)t.key)[h];
  if (q.x == z) at = 4 * h;
  if (q.y == z) at = 4 * h + 1;
  if (q.z == z) at = 4 * h + 2;
  if (q.w == z) at = 4 * h + 3;
  return at;
}

// Place of z in the table (its index in N(v0) is t.pos of it), or -1.
__device__ __forceinline__ int look_up(const Table& t, int probes, int z) {
  uint32_t h = bucket_of(t, z);
  int at = in_bucket(t, h, z, -1);
  for (int k = 1; k < probes; ++k) {
    h = (h + 1) & t.mask;
    at = in_bucket(t, h, z, at);
  }
  return at;
}

// Puts z = N(v0)[i]; the buckets it took.
__device__ __forceinline__ int insert(const Table& t, int z, int i) {
  uint32_t h = bucket_of(t, z);
  for (int k = 1;; ++k, h = (h + 1) & t.mask)
    for (int q = 0; q < 4; ++q)
      if (atomicCAS(&t.key[4 * h + q], -1, z) == -1) {
        t.pos[4 * h + q] = (uint16_t)i;
        return k;
      }
}

// Start of part y of z equal parts of n.
__device__ __forceinline__ long long share(long long n, int y, int z) {
  return n / z * y + min((long long)y, n % z);
}

// n-th set bit of m (n < popc(m)).
__device__ __forceinline__ int nth_bit(uint32_t m, int n) {
  int at = 0;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const int c = __popc(m & ((1u << s) - 1u));
    if (n >= c) {
      n -= c;
      m >>= s;
      at += s;
    }
  }
  return at;
}

// Word `wi` of a term over v1 (and v2 if `two`), of the words r1 and r2 of their rows; a
// bound or exclusion by v3 is left out.
__device__ __forceinline__ uint32_t term(const BitTerm& t, uint32_t r1, uint32_t r2, int i1,
                                         int i2, int pre0, int pre2, int wi, int d0, bool two) {
  const int lo = 32 * wi;
  uint32_t m = part(t, 1, r1);
  int lim = d0;
  if (t.bound & 1) lim = min(lim, pre0);
  if (t.bound & 2) lim = min(lim, i1);
  if ((t.excl & 2) && (i1 >> 5) == wi) m &= ~(1u << (i1 & 31));
  if (two) {
    m &= part(t, 2, r2);
    if (t.bound & 4) lim = min(lim, pre2);
    if ((t.excl & 4) && i2 >= 0 && (i2 >> 5) == wi) m &= ~(1u << (i2 & 31));
  }
  return m & below(lim, lo);
}

template <int NW>
__device__ __forceinline__ void load_row(uint32_t (&x)[NW], const uint32_t* r) {
  if constexpr (NW == 1) {
    x[0] = r[0];
  } else {
#pragma unroll
    for (int k = 0; k < NW; k += 4) {
      const uint4 q = ((const uint4*)r)[k / 4];
      x[k] = q.x, x[k + 1] = q.y, x[k + 2] = q.z, x[k + 3] = q.w;
    }
  }
}

// What a warp needs of its v0.
struct Local {
  const int32_t* n0;     // N(v0)
  const uint32_t* rows;  // row i at rows + i * ld
  int ld, d0, v0, pre0;
  Table t;
  int probes;
};

// Each lane with `on` gets the row over N(v0) of the list [b, b + n).  The lists are cut
// into pieces of 16 entries, dealt to groups of eight lanes: by whole lists, four groups
// waited for the longest.  out: 32 x NW words of the warp.
template <int NW>
__device__ __forceinline__ void list_rows(const Local& w, uint32_t* out, const int32_t* col,
                                          bool on, int64_t b, int n, uint32_t (&r)[NW], int lane) {
#pragma unroll
  for (int q = 0; q < NW; ++q) out[lane * NW + q] = 0u;
  // a list far longer than N(v0): N(v0) is searched in it, an element a lane
  const bool lng = on && n > 64 + 8 * w.d0;
  int incl = on && !lng ? (n + 15) >> 4 : 0;
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, k);
    if (lane >= k) incl += y;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  const int first = incl - (on && !lng ? (n + 15) >> 4 : 0);
  const int g = lane >> 3, sub = lane & 7;
  for (int base = 0; base < total; base += 4) {
    const int item = base + g;
    int t = 0;  // the list of this piece: the first whose inclusive count passes it
#pragma unroll
    for (int h = 16; h > 0; h >>= 1)
      if (__shfl_sync(0xffffffffu, incl, t + h - 1) <= item) t += h;
    t &= 31;
    const int at = 16 * (item - __shfl_sync(0xffffffffu, first, t)) + sub;
    const int len = __shfl_sync(0xffffffffu, n, t);
    const int ln = item < total ? len : 0;
    const int32_t* l = col + __shfl_sync(0xffffffffu, b, t);
    uint32_t* o = out + t * NW;
    const int z0 = at < ln ? l[at] : -2, z1 = at + 8 < ln ? l[at + 8] : -2;
    const int p0 = look_up(w.t, w.probes, z0), p1 = look_up(w.t, w.probes, z1);
    if (p0 >= 0) {
      const int i = w.t.pos[p0];
      atomicOr(o + (NW == 1 ? 0 : i >> 5), 1u << (i & 31));
    }
    if (p1 >= 0) {
      const int i = w.t.pos[p1];
      atomicOr(o + (NW == 1 ? 0 : i >> 5), 1u << (i & 31));
    }
  }
  __syncwarp();
  for (unsigned todo = __ballot_sync(0xffffffffu, lng); todo; todo &= todo - 1) {
    const int src = __ffs(todo) - 1;
    const int ln = __shfl_sync(0xffffffffu, n, src);
    const int32_t* l = col + __shfl_sync(0xffffffffu, b, src);
#pragma unroll
    for (int q = 0; q < NW; ++q) {
      const int i = 32 * q + lane;
      const unsigned m = __ballot_sync(0xffffffffu, i < w.d0 && member(l, ln, w.n0[min(i, w.d0 - 1)]));
      if (lane == 0) out[src * NW + q] = m;
    }
  }
  __syncwarp();
  load_row<NW>(r, out + lane * NW);
  __syncwarp();
}

// v2 candidates of the task (v0, N(v0)[i]) of row words row[0, W): the entries of N(v1)
// below its bound (a stream), or the members of the set.  None where a set that needs no
// v2 is empty already.
template <int K>
__device__ __forceinline__ int task_size(const BitArgs& a, const Local& w, int i, int W) {
  const BitPlan& p = a.p;
  const int v1 = w.n0[i];
  if (p.v1lt && v1 >= w.v0) return 0;
  uint32_t any3 = K == 5 ? 0u : 1u, anyf = 0;
  int n2 = 0;
  for (int wi = 0; wi < W; ++wi) {
    const uint32_t r1 = w.rows[i * w.ld + wi];
    if (K == 5) any3 |= term(p.c3, r1, 0, i, -1, w.pre0, 0, wi, w.d0, false);
    anyf |= term(p.fin, r1, 0, i, -1, w.pre0, 0, wi, w.d0, false);
    if (!p.stream) n2 += __popc(term(p.c2, r1, 0, i, -1, w.pre0, 0, wi, w.d0, false));
  }
  if (!any3 || !anyf) return 0;
  if (!p.stream) return n2;
  const int64_t b1 = a.rowptr[v1];
  const int d1 = (int)(a.rowptr[v1 + 1] - b1);
  int ub = INT32_MAX;
  if (p.c2.bound & 1) ub = w.v0;
  if (p.c2.bound & 2) ub = min(ub, v1);
  return ub == INT32_MAX ? d1 : lower_index(a.col + b1, d1, ub);
}

// One decoded step: its task and its v2.
struct Item {
  bool on;
  int i1, i2, pre2, dy;
  int64_t by;
};

// Item `item` of the tasks' shares (rel: inclusive counts, off: item -> entry).
__device__ __forceinline__ Item decode(const BitArgs& a, const Local& w, const int32_t* rel,
                                       const int32_t* off, int W, bool on, int item) {
  const BitPlan& p = a.p;
  Item s{on, 0, -1, 0, 0, 0};
  if (!on) return s;
  s.i1 = 0;
  for (int n = w.d0; n > 0;) {  // first task whose inclusive count passes the item
    const int h = n >> 1;
    if (rel[s.i1 + h] <= item) {
      s.i1 += h + 1;
      n -= h + 1;
    } else {
      n = h;
    }
  }
  const int at = item + off[s.i1];
  if (p.stream) {
    const int y = a.col[a.rowptr[w.n0[s.i1]] + at];
    s.on = look_up(w.t, w.probes, y) < 0 && !((p.c2.excl & 1) && y == w.v0);
    if (s.on) {
      s.by = a.rowptr[y];
      s.dy = (int)(a.rowptr[y + 1] - s.by);
      if (p.bound2) s.pre2 = lower_index(w.n0, w.d0, y);
    }
  } else {
    int left = at;
    for (int wi = 0; wi < W; ++wi) {
      const uint32_t m =
          term(p.c2, w.rows[s.i1 * w.ld + wi], 0, s.i1, -1, w.pre0, 0, wi, w.d0, false);
      const int k = __popc(m);
      if (left < k) {
        s.i2 = 32 * wi + nth_bit(m, left);
        break;
      }
      left -= k;
    }
    s.pre2 = s.i2;
  }
  return s;
}

// The count of one step: v1 = N(v0)[i1], v2 with its row and places.
template <int K, int NW>
__device__ __forceinline__ unsigned count_step(const BitPlan& p, const Local& w, int i1, int i2,
                                               int pre2, const uint32_t (&r2)[NW]) {
  unsigned c = 0;
  uint32_t r1[NW], fk[NW];
  load_row<NW>(r1, w.rows + i1 * w.ld);
  uint32_t any = 0;
#pragma unroll
  for (int q = 0; q < NW; ++q) {
    fk[q] = term(p.fin, r1[q], r2[q], i1, i2, w.pre0, pre2, q, w.d0, true);
    any |= fk[q];
    if (K == 4) c += __popc(fk[q]);
  }
  if (K == 4 || !any) return c;
  const bool f_ub = (p.fin.bound >> 3) & 1, f_ux = (p.fin.excl >> 3) & 1;
  const bool f_row = ((p.fin.pos | p.fin.neg) >> 3) & 1;
  const uint32_t flip = (p.fin.neg >> 3) & 1 ? 0xffffffffu : 0u;
#pragma unroll
  for (int q = 0; q < NW; ++q) {
    for (uint32_t m = term(p.c3, r1[q], r2[q], i1, i2, w.pre0, pre2, q, w.d0, true); m;
         m &= m - 1) {
      const int b = __ffs(m) - 1;
      uint32_t r3[NW];
      if (f_row) {
        load_row<NW>(r3, w.rows + (32 * q + b) * w.ld);
      } else {
#pragma unroll
        for (int k = 0; k < NW; ++k) r3[k] = fk[k];
      }
      const uint32_t upto = f_ub ? (1u << b) - 1u : (f_ux ? ~(1u << b) : 0xffffffffu);
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        uint32_t x = fk[k] & (r3[k] ^ flip);
        if (k == q) x &= upto;
        if (k > q && f_ub) x = 0u;
        c += __popc(x);
      }
    }
  }
  return c;
}

// A lane a step: 32 items from `base`.
template <int K, int NW>
__device__ __forceinline__ unsigned lane_steps(const BitArgs& a, const Local& w,
                                               const int32_t* rel, const int32_t* off,
                                               uint32_t* out, int base, int total, int lane) {
  const Item s = decode(a, w, rel, off, NW, base + lane < total, base + lane);
  uint32_t r2[NW];
  if (a.p.stream) {
    list_rows<NW>(w, out, a.col, s.on, s.by, s.dy, r2, lane);
  } else if (s.on) {
    load_row<NW>(r2, w.rows + s.i2 * w.ld);
  }
  return s.on ? count_step<K, NW>(a.p, w, s.i1, s.i2, s.pre2, r2) : 0u;
}

// Rows over N(v0) of the vertices y outside it, by streaming the lists of N(v0)'s members
// (the graph is symmetric): y's bit i is set where y is in N(N(v0)[i]).  Every set bit of a
// finished table is a step (v0, v1, y).  Open addressing; a table takes the y whose hash_part
// lies in a range, and a range that does not fit is halved (one value of hash_part is one y).
struct YTable {
  int32_t* key;
  uint32_t* val;  // NW words a slot
  int mask, shift;
};

__device__ __forceinline__ uint32_t hash_part(int y) {
  uint32_t h = (uint32_t)y * 0x85ebca6bu;
  return h ^ (h >> 16);
}

template <int NW>
__device__ __forceinline__ bool put(const YTable& t, int y, int i) {
  uint32_t h = ((uint32_t)y * 2654435761u) >> t.shift;
  for (int k = 0; k < 64; ++k, h = (h + 1) & t.mask) {
    int at = ((volatile int32_t*)t.key)[h];
    if (at == -1) {
      at = atomicCAS(&t.key[h], -1, y);
      if (at == -1) at = y;
    }
    if (at == y) {
      atomicOr(&t.val[h * NW + (NW == 1 ? 0 : i >> 5)], 1u << (i & 31));
      return true;
    }
  }
  return false;
}

// The steps of the table's slots, 32 slots a warp at a time (from *next for a block's warps).
// queue: 64 words of the warp; steps gather there until a lane each.  live: the tasks with
// steps.
template <int K, int NW>
__device__ __forceinline__ unsigned long long table_steps(const BitPlan& p, const Local& w,
                                                          const YTable& t, const uint32_t* live,
                                                          uint32_t* queue, int* next, int lane) {
  unsigned long long c = 0;
  int qn = 0;
  auto step = [&](uint32_t e) {
    const int slot = e >> 16;
    uint32_t r2[NW];
    load_row<NW>(r2, t.val + slot * NW);
    const int pre2 = p.bound2 ? lower_index(w.n0, w.d0, t.key[slot]) : 0;
    c += count_step<K, NW>(p, w, e & 0xffff, -1, pre2, r2);
  };
  for (int base = 0;; base += 32) {
    if (next) {
      if (lane == 0) base = atomicAdd(next, 32);
      base = __shfl_sync(0xffffffffu, base, 0);
    }
    if (base > t.mask) break;
    const int slot = base + lane;
    const int y = t.key[slot];
    uint32_t m[NW];
#pragma unroll
    for (int q = 0; q < NW; ++q) m[q] = 0u;
    // the stream's bound and exclusion: y below v0, v1; not v0
    if (y >= 0 && !((p.c2.bound & 1) && y >= w.v0) && !((p.c2.excl & 1) && y == w.v0)) {
      load_row<NW>(m, t.val + slot * NW);
      const int pre = p.c2.bound & 2 ? lower_index(w.n0, w.d0, y) : 0;
#pragma unroll
      for (int q = 0; q < NW; ++q) m[q] &= live[q] & ~below(pre, 32 * q);
    }
    for (;;) {
      int i1 = -1;
#pragma unroll
      for (int q = 0; q < NW; ++q)
        if (i1 < 0 && m[q]) {
          i1 = 32 * q + __ffs(m[q]) - 1;
          m[q] &= m[q] - 1;
        }
      const unsigned b = __ballot_sync(0xffffffffu, i1 >= 0);
      if (!b) break;
      if (i1 >= 0) queue[qn + __popc(b & ((1u << lane) - 1u))] = (uint32_t)slot << 16 | i1;
      qn += __popc(b);
      __syncwarp();
      if (qn >= 32) {
        step(queue[lane]);
        const uint32_t rest = queue[32 + lane];
        __syncwarp();
        queue[lane] = rest;
        qn -= 32;
        __syncwarp();
      }
    }
  }
  if (lane < qn) step(queue[lane]);
  __syncwarp();
  return c;
}

// ---------------------------------------------------------------- d(v0) <= 32
constexpr int kSmallBuckets = 64;

constexpr int kSmallTable = 512;  // slots of a warp's table of two-hop vertices
constexpr int kSmallItems = 448;  // list entries taken to one table at first

struct SmallMap {
  int32_t key[kSmallTable];
  uint32_t val[kSmallTable];
  uint32_t queue[64];
};

struct SmallWarp {
  int32_t key[4 * kSmallBuckets];
  uint16_t pos[4 * kSmallBuckets];
  int32_t n0[32];
  uint32_t rows[32];
  uint32_t out[32];
  int32_t rel[32], off[32];
};

// The unit's share, by hash_part, of the steps whose v2 are the two-hop vertices of the lists
// [b1, b1 + d1) (a lane a list, `lists` entries in all).
template <int K>
__device__ __forceinline__ unsigned long long small_map(const BitArgs& a, const Local& w,
                                                        SmallMap& map, const int4& unit,
                                                        int64_t b1, int d1, int lists,
                                                        uint32_t live, int lane) {
  const YTable t{map.key, map.val, kSmallTable - 1, __clz(kSmallTable) + 1};
  int incl = (d1 + 15) >> 4;  // pieces of 16 entries, as in list_rows
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, k);
    if (lane >= k) incl += y;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  const int first = incl - ((d1 + 15) >> 4);
  const int g = lane >> 3, sub = lane & 7;
  const long long end = share(1LL << 32, unit.y + 1, unit.z);
  long long lo = share(1LL << 32, unit.y, unit.z);
  const int per = lists / unit.z + 1;
  long long span = (end - lo + (per + kSmallItems - 1) / kSmallItems - 1) /
                   ((per + kSmallItems - 1) / kSmallItems);
  unsigned long long c = 0;
  while (lo < end) {
    const long long hi = min(lo + span, end);
#pragma unroll
    for (int k = lane; k < kSmallTable / 4; k += 32) {
      ((int4*)map.key)[k] = make_int4(-1, -1, -1, -1);
      ((int4*)map.val)[k] = make_int4(0, 0, 0, 0);
    }
    __syncwarp();
    bool fits = true;
    for (int base = 0; base < total; base += 4) {
      const int item = base + g;
      int i = 0;  // the list of this piece
#pragma unroll
      for (int h = 16; h > 0; h >>= 1)
        if (__shfl_sync(0xffffffffu, incl, i + h - 1) <= item) i += h;
      i &= 31;
      const int at = 16 * (item - __shfl_sync(0xffffffffu, first, i)) + sub;
      const int len = __shfl_sync(0xffffffffu, d1, i);
      const int ln = item < total ? len : 0;
      const int32_t* l = a.col + __shfl_sync(0xffffffffu, b1, i);
      const int y0 = at < ln ? l[at] : -1, y1 = at + 8 < ln ? l[at + 8] : -1;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int y = k ? y1 : y0;
        const uint32_t h = hash_part(y);
        if (y >= 0 && h >= lo && h < hi && look_up(w.t, w.probes, y) < 0) fits &= put<1>(t, y, i);
      }
      __syncwarp();
    }
    if (!__all_sync(0xffffffffu, fits)) {
      span = (span + 1) / 2;
      continue;
    }
    c += table_steps<K, 1>(a.p, w, t, &live, map.queue, nullptr, lane);
    lo = hi;
  }
  return c;
}

template <int K>
__global__ void __launch_bounds__(kThreads, 4) k_bits_warp(BitArgs a) {
  extern __shared__ __align__(16) unsigned char sm[];
  let_next_start();
  const int lane = threadIdx.x & 31;
  SmallWarp& w = ((SmallWarp*)sm)[threadIdx.x >> 5];
  // (a stream program's launch only)
  SmallMap& map = ((SmallMap*)(sm + kWarps * sizeof(SmallWarp)))[threadIdx.x >> 5];
  if (blockIdx.x == 0 && threadIdx.x == 0 && a.split_out) *a.split_out = (int64_t)a.un[3];
  const int64_t n_units = (int64_t)a.un[a.cls];
  // one unit a claim, up to eight when every warp takes 64 and more
  const int64_t nw = (int64_t)gridDim.x * kWarps;
  const int chunk = (int)max((int64_t)1, min((int64_t)8, n_units / (8 * nw)));
  Local l;
  l.n0 = w.n0;
  l.rows = w.rows;
  l.ld = 1;
  l.t = Table{w.key, w.pos, kSmallBuckets - 1, __clz(kSmallBuckets) + 1};
  unsigned long long c = 0;
  for (;;) {
    int64_t u0 = 0;
    if (lane == 0) u0 = (int64_t)atomicAdd(a.head, (unsigned long long)chunk);
    u0 = __shfl_sync(0xffffffffu, u0, 0);
    if (u0 >= n_units) break;
    for (int64_t u = u0; u < min(u0 + chunk, n_units); ++u) {
      const int4 unit = a.units[u];
      l.v0 = unit.x;
      const int64_t rb = a.rowptr[l.v0];
      l.d0 = (int)(a.rowptr[l.v0 + 1] - rb);
      const bool mine = lane < l.d0;
      const int v1 = mine ? a.col[rb + lane] : 0;
#pragma unroll
      for (int k = 0; k < kSmallBuckets / 32; ++k)
        ((int4*)w.key)[32 * k + lane] = make_int4(-1, -1, -1, -1);
      if (mine) w.n0[lane] = v1;
      __syncwarp();
      int64_t b1 = 0;
      int d1 = 0, probes = 1;
      if (mine) {
        probes = insert(l.t, v1, lane);
        b1 = a.rowptr[v1];
        d1 = (int)(a.rowptr[v1 + 1] - b1);
      }
      l.probes = __reduce_max_sync(0xffffffffu, probes);
      l.pre0 = lower_index(w.n0, l.d0, l.v0);
      uint32_t row[1];
      list_rows<1>(l, w.out, a.col, mine, b1, d1, row, lane);
      w.rows[lane] = row[0];
      __syncwarp();
      // this unit's range of the v0's steps, and each task's share of it
      const int n = mine ? task_size<K>(a, l, lane, 1) : 0;
      long long incl = n;
#pragma unroll
      for (int k = 1; k < 32; k <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, incl, k);
        if (lane >= k) incl += y;
      }
      const long long all = __shfl_sync(0xffffffffu, incl, 31);
      __syncwarp();
      if (all == 0) continue;
      if (a.p.stream) {
        long long lists = d1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) lists += __shfl_xor_sync(0xffffffffu, lists, o);
        // from a table unless few tasks have steps (a table takes every list's entries, a
        // look-up form only theirs) or a pass over the lists would keep under a sixteenth
        if (2 * all >= lists && lists <= 16 * kSmallItems) {
          c += small_map<K>(a, l, map, unit, b1, d1, (int)lists,
                            __ballot_sync(0xffffffffu, n > 0), lane);
          continue;
        }
      }
      const long long lo = share(all, unit.y, unit.z), hi = share(all, unit.y + 1, unit.z);
      const int total = (int)(hi - lo);
      w.rel[lane] = (int)max(0LL, min(incl - lo, (long long)total));
      // item -> entry of the task's list; only read for tasks with items in the range
      w.off[lane] = incl - n < hi && incl > lo ? (int)(lo - (incl - n)) : 0;
      __syncwarp();
      for (int base = 0; base < total; base += 32)
        c += lane_steps<K, 1>(a, l, w.rel, w.off, w.out, base, total, lane);
      __syncwarp();
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if (lane == 0 && c) atomicAdd(a.total, c);
  wait_for_previous();
}

// ------------------------------------------------------- 33 <= d(v0) <= 1,024
// Words of a row in shared memory: 16 bytes times an odd number.
__host__ __device__ constexpr int row_stride(int W) { return 4 * (((W + 3) >> 2) | 1); }

constexpr CtaLayout cta_layout(int deg, int warps) {
  CtaLayout l{};
  l.deg = deg;
  l.buckets = 64;
  while (l.buckets < 2 * deg) l.buckets *= 2;
  if (l.buckets > 1024) l.buckets = 1024;  // a key a bucket at most
  int at = deg * 4 * row_stride((deg + 31) / 32);
  l.n0 = at;
  at += deg * 4;
  l.key = at;
  at += l.buckets * 16;
  l.pos = at;
  at += l.buckets * 8;
  l.rel = at;
  at += deg * 4;
  l.off = at;
  at += deg * 4;
  l.warp = at;
  l.per_warp = 32 * 4 + 32 * 4 + kListCap * 2;  // row of v2, counted words, v3 list
  at += l.per_warp * warps;
  l.bytes = at;
  return l;
}

static_assert(cta_layout(kTopDeg, kTopThreads / 32).bytes <= 227 * 1024, "shared memory");

// This lane's word of the row over N(v0) of a list of n entries (a warp a list).
__device__ __forceinline__ uint32_t warp_row(const Local& w, uint32_t* row, const int32_t* l,
                                             int n, int lane) {
  row[lane] = 0u;
  __syncwarp();
  if (n <= 256 + 4 * w.d0) {
    for (int t = lane; t < n; t += 32) {
      const int at = look_up(w.t, w.probes, l[t]);
      if (at >= 0) {
        const int k = w.t.pos[at];
        atomicOr(&row[k >> 5], 1u << (k & 31));
      }
    }
  } else {
    for (int b = 0; b < w.d0; b += 32) {
      const unsigned m = __ballot_sync(
          0xffffffffu, b + lane < w.d0 && member(l, n, w.n0[min(b + lane, w.d0 - 1)]));
      if (lane == 0) row[b >> 5] = m;
    }
  }
  __syncwarp();
  const uint32_t r = row[lane];
  __syncwarp();
  return r;
}

// A warp a step (d(v0) > kLaneDeg): a word a lane for the terms, a v3 a lane for the count.
template <int K>
__device__ __forceinline__ unsigned long long warp_step(const BitArgs& a, const Local& w,
                                                        uint32_t* mine, const Item& s, int W,
                                                        int lane) {
  const BitPlan& p = a.p;
  uint32_t* fk = mine + 32;
  uint16_t* list = (uint16_t*)(mine + 64);
  const bool f_ub = (p.fin.bound >> 3) & 1;
  const bool f_self = ((p.fin.excl >> 3) & 1) && !f_ub && !((p.fin.pos >> 3) & 1);
  const uint32_t r1 = lane < W ? w.rows[s.i1 * w.ld + lane] : 0u;
  uint32_t r2;
  if (p.stream) {
    r2 = warp_row(w, mine, a.col + s.by, s.dy, lane);
  } else {
    r2 = lane < W ? w.rows[s.i2 * w.ld + lane] : 0u;
  }
  const uint32_t f =
      lane < W ? term(p.fin, r1, r2, s.i1, s.i2, w.pre0, s.pre2, lane, w.d0, true) : 0u;
  if (K == 4) {
    __syncwarp();
    return __popc(f);
  }
  const uint32_t c3 =
      lane < W ? term(p.c3, r1, r2, s.i1, s.i2, w.pre0, s.pre2, lane, w.d0, true) : 0u;
  if (!__any_sync(0xffffffffu, c3) || !__any_sync(0xffffffffu, f)) return 0;
  fk[lane] = f;
  const bool f_row = ((p.fin.pos | p.fin.neg) >> 3) & 1;
  const uint32_t flip = (p.fin.neg >> 3) & 1 ? 0xffffffffu : 0u;
  unsigned long long c = 0;
  for (int wi = 0; wi < W;) {
    int n3 = 0;
    for (; wi < W && n3 + 32 <= kListCap; ++wi) {
      const uint32_t m = __shfl_sync(0xffffffffu, c3, wi);
      if ((m >> lane) & 1u)
        list[n3 + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(32 * wi + lane);
      n3 += __popc(m);
    }
    __syncwarp();
    const uint4* f4 = (const uint4*)fk;
    for (int t = lane; t < n3; t += 32) {
      const int b = list[t], bw = b >> 5;
      const uint4* r4 = f_row ? (const uint4*)(w.rows + b * w.ld) : f4;
      const int full = f_ub ? bw >> 2 : (W + 3) >> 2;  // whole 16-byte pieces
      unsigned k = 0;
      for (int q = 0; q < full; ++q) {
        const uint4 x = f4[q], r = r4[q];
        k += __popc(x.x & (r.x ^ flip)) + __popc(x.y & (r.y ^ flip)) +
             __popc(x.z & (r.z ^ flip)) + __popc(x.w & (r.w ^ flip));
      }
      if (f_ub) {  // the piece that holds v3
        const uint4 x = f4[full], r = r4[full];
        const int lim = b - 128 * full;
        k += __popc(x.x & (r.x ^ flip) & below(lim, 0)) +
             __popc(x.y & (r.y ^ flip) & below(lim, 32)) +
             __popc(x.z & (r.z ^ flip) & below(lim, 64)) +
             __popc(x.w & (r.w ^ flip) & below(lim, 96));
      }
      if (f_self) k -= (fk[bw] >> (b & 31)) & 1u;  // v3 itself is not in its own row
      c += k;
    }
    __syncwarp();
  }
  return c;
}

// N(v0), its rows and its hash table into shared memory; the row words.  A block, which
// synchronises before it reads *probes.
template <int NT>
__device__ __forceinline__ int load_v0(const BitArgs& a, Local& w, int v0, int32_t* n0,
                                       uint32_t* rows, int max_buckets, int* probes, int tid) {
  w.v0 = v0;
  const int64_t rb = a.rowptr[v0];
  const int d0 = (int)(a.rowptr[v0 + 1] - rb);
  w.d0 = d0;
  const int W = (d0 + 31) >> 5;
  w.ld = row_stride(W);
  int nb = 64;
  while (nb < 2 * d0 && nb < max_buckets) nb <<= 1;
  w.t.mask = nb - 1;
  w.t.shift = __clz(nb) + 1;
  for (int i = tid; i < nb; i += NT) ((int4*)w.t.key)[i] = make_int4(-1, -1, -1, -1);
  for (int i = tid; i < d0; i += NT) n0[i] = a.col[rb + i];
  const uint32_t* g = a.rows + a.roff[v0];
  for (int i = tid; i < d0 * w.ld; i += NT) {
    const int r = i / w.ld, wi = i - r * w.ld;
    rows[i] = wi < W ? g[(int64_t)r * W + wi] : 0u;
  }
  __syncthreads();
  for (int i = tid; i < d0; i += NT) {
    const int k = insert(w.t, n0[i], i);
    if (k > 1) atomicMax(probes, k);
  }
  w.pre0 = lower_index(n0, d0, v0);
  return W;
}

template <int K, int NT>
__global__ void __launch_bounds__(NT, NT == kThreads ? 4 : 1) k_bits_cta(BitArgs a) {
  extern __shared__ __align__(16) unsigned char sm[];
  let_next_start();
  const CtaLayout& L = a.lay;
  __shared__ int64_t s_unit;
  __shared__ int s_next, s_probes;
  __shared__ long long s_sum[NT / 32];
  uint32_t* rows = (uint32_t*)sm;
  int32_t* n0 = (int32_t*)(sm + L.n0);
  int32_t* rel = (int32_t*)(sm + L.rel);
  int32_t* off = (int32_t*)(sm + L.off);
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  uint32_t* mine = (uint32_t*)(sm + L.warp + wib * L.per_warp);
  Local w;
  w.n0 = n0;
  w.rows = rows;
  w.t.key = (int32_t*)(sm + L.key);
  w.t.pos = (uint16_t*)(sm + L.pos);
  const int64_t n_units = (int64_t)a.un[a.cls];
  unsigned long long c = 0;
  for (;;) {
    if (tid == 0) {
      s_unit = (int64_t)atomicAdd(a.head, 1ull);
      s_next = 0;
      s_probes = 1;
    }
    __syncthreads();
    const int64_t u = s_unit;
    if (u >= n_units) break;
    const int4 unit = a.units[u];
    const int W = load_v0<NT>(a, w, unit.x, n0, rows, L.buckets, &s_probes, tid);
    const int d0 = w.d0;
    // the steps of each task (v0, N(v0)[i]), this thread's run of tasks
    const int per = (d0 + NT - 1) / NT;
    const int t0 = min(tid * per, d0), t1 = min(t0 + per, d0);
    long long sum = 0;
    for (int i = t0; i < t1; ++i) {
      off[i] = task_size<K>(a, w, i, W);
      sum += off[i];
    }
    long long incl = sum;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, incl, k);
      if (lane >= k) incl += y;
    }
    if (lane == 31) s_sum[wib] = incl;
    __syncthreads();
    w.probes = s_probes;
    long long before = incl - sum, all = 0;
    for (int k = 0; k < NT / 32; ++k) {
      if (k < wib) before += s_sum[k];
      all += s_sum[k];
    }
    const long long lo = share(all, unit.y, unit.z), hi = share(all, unit.y + 1, unit.z);
    const int total = (int)(hi - lo);
    for (int i = t0; i < t1; ++i) {
      const int n = off[i];
      const long long excl = before;
      before += n;
      rel[i] = (int)max(0LL, min(before - lo, (long long)total));
      // item -> entry of the task's list; only read for tasks with items in the range
      off[i] = excl < hi && before > lo ? (int)(lo - excl) : 0;
    }
    __syncthreads();
    const bool lanes = NT == kThreads && d0 <= kLaneDeg;
    for (;;) {
      int base = 0;
      if (lane == 0) base = atomicAdd(&s_next, lanes ? 32 : kBatch);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base >= total) break;
      if (lanes) {
        c += lane_steps<K, 4>(a, w, rel, off, mine, base, total, lane);
        continue;
      }
      const Item s = decode(a, w, rel, off, W, lane < kBatch && base + lane < total, base + lane);
      for (unsigned todo = __ballot_sync(0xffffffffu, s.on); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        Item t;
        t.i1 = __shfl_sync(0xffffffffu, s.i1, src);
        t.i2 = __shfl_sync(0xffffffffu, s.i2, src);
        t.pre2 = __shfl_sync(0xffffffffu, s.pre2, src);
        t.by = __shfl_sync(0xffffffffu, s.by, src);
        t.dy = __shfl_sync(0xffffffffu, s.dy, src);
        c += warp_step<K>(a, w, mine, t, W, lane);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if (lane == 0 && c) atomicAdd(a.total, c);
  wait_for_previous();
}

// Stream programs, 33 <= d(v0) <= 256: a block takes the steps of a v0 from tables of its
// two-hop vertices, a lane a step.  3.9 steps (d(v0) <= 128) and 5.7 share a v2's row on
// R-MAT scale 12, so the lists may hold 1.5 entries a slot before a pass is cut; a step costs
// no look-ups of its v2's whole list, and the queue leaves no lane without one.  P7 there:
// 1.10 ms from k_bits_cta, 0.67 ms (blocks of 256 threads, three an SM with half the table
// 0.98, one of 1,024 with twice the table 0.88).
constexpr int kMapThreads = 512;
constexpr int kMapBlocks = 2;    // an SM
constexpr int kMapSlots = 4096;  // rows of four words; half with eight
// Work of the class, an SM, from which a stream program takes k_bits_map: below, its few large
// blocks leave SMs idle.  P7, k_bits_map against k_bits_cta, by R-MAT scale (work an SM):
// 9 (1,569) 0.190 and 0.118 ms, 10 (4,035) 0.322 and 0.260, 11 (9,472) 0.534 and 0.551,
// 12 (27,082) 1.32 and 1.78.
constexpr int kMapWork = 8192;

struct MapSmem {
  uint32_t rows[kMidDeg * row_stride(kMidDeg / 32)];
  int32_t key[4 * 2 * kMidDeg];
  uint16_t pos[4 * 2 * kMidDeg];
  int32_t n0[kMidDeg];
  int32_t rel[kMidDeg], off[kMidDeg];
  uint32_t live[kMidDeg / 32];
  uint32_t queue[kMapThreads / 32][64];
  long long sum[kMapThreads / 32], lists[kMapThreads / 32];
  int64_t unit;
  int next, probes, full, list, slot;
  // tables (key, val), or the lanes' rows
  __align__(16) uint32_t table[kMapSlots * 5];
};
static_assert(kMapBlocks * (sizeof(MapSmem) + 1024) <= 228 * 1024 &&
                  kMapSlots * 5 >= kMapThreads * 8, "shared memory");

template <int K, int NW>
__device__ __forceinline__ unsigned long long map_steps(const BitArgs& a, const Local& w,
                                                        MapSmem& m, const int4& unit,
                                                        long long lists, int tid) {
  const int lane = tid & 31, wib = tid >> 5;
  constexpr int kSlots = NW == 4 ? kMapSlots : kMapSlots / 2;
  const YTable t{(int32_t*)m.table + kSlots * NW, m.table, kSlots - 1, __clz(kSlots) + 1};
  const int target = min(a.items, kSlots * 3 / 2);
  // consecutive parts share a pass: about `target` entries of the lists each
  const int passes = (int)((lists + target - 1) / target);
  const int g = passes >= unit.z ? 1 : (unit.z + passes - 1) / passes;
  if (unit.y % g) return 0;
  const long long end = share(1LL << 32, min(unit.y + g, unit.z), unit.z);
  long long lo = share(1LL << 32, unit.y, unit.z);
  const int cut = max(1, (passes + unit.z - 1) / unit.z);
  long long span = (end - lo + cut - 1) / cut;
  unsigned long long c = 0;
  while (lo < end) {
    const long long hi = min(lo + span, end);
    for (int k = tid; k < kSlots * NW / 4; k += kMapThreads)
      ((int4*)t.val)[k] = make_int4(0, 0, 0, 0);
    for (int k = tid; k < kSlots / 4; k += kMapThreads)
      ((int4*)t.key)[k] = make_int4(-1, -1, -1, -1);
    if (tid == 0) m.full = m.list = m.slot = 0;
    __syncthreads();
    bool fits = true;
    for (;;) {
      int i = 0;
      if (lane == 0) i = atomicAdd(&m.list, 1);
      i = __shfl_sync(0xffffffffu, i, 0);
      if (i >= w.d0) break;
      const int64_t b = a.rowptr[w.n0[i]];
      const int n = (int)(a.rowptr[w.n0[i] + 1] - b);
      const int32_t* l = a.col + b;
      for (int at = lane; at < n; at += 32) {
        const int y = l[at];
        const uint32_t h = hash_part(y);
        if (h >= lo && h < hi && look_up(w.t, w.probes, y) < 0) fits &= put<NW>(t, y, i);
      }
    }
    if (!fits) m.full = 1;
    __syncthreads();
    if (m.full) {
      span = (span + 1) / 2;
      __syncthreads();
      continue;
    }
    c += table_steps<K, NW>(a.p, w, t, m.live, m.queue[wib], &m.slot, lane);
    __syncthreads();
    lo = hi;
  }
  return c;
}

template <int K>
__global__ void __launch_bounds__(kMapThreads, kMapBlocks) k_bits_map(BitArgs a) {
  extern __shared__ __align__(16) unsigned char sm[];
  let_next_start();
  MapSmem& m = *(MapSmem*)sm;
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  Local w;
  w.n0 = m.n0;
  w.rows = m.rows;
  w.t.key = m.key;
  w.t.pos = m.pos;
  const int64_t n_units = (int64_t)a.un[a.cls];
  unsigned long long c = 0;
  for (;;) {
    if (tid == 0) {
      m.unit = (int64_t)atomicAdd(a.head, 1ull);
      m.next = 0;
      m.probes = 1;
    }
    __syncthreads();
    const int64_t u = m.unit;
    if (u >= n_units) break;
    const int4 unit = a.units[u];
    const int W = load_v0<kMapThreads>(a, w, unit.x, m.n0, m.rows, 2 * kMidDeg, &m.probes, tid);
    __syncthreads();
    // a thread a task
    int n = 0, d1 = 0;
    if (tid < w.d0) {
      n = task_size<K>(a, w, tid, W);
      d1 = (int)(a.rowptr[w.n0[tid] + 1] - a.rowptr[w.n0[tid]]);
    }
    const unsigned on = __ballot_sync(0xffffffffu, n > 0);
    if (lane == 0 && wib < kMidDeg / 32) m.live[wib] = on;
    long long incl = n, lists = d1;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, incl, k);
      const long long z = __shfl_up_sync(0xffffffffu, lists, k);
      if (lane >= k) incl += y, lists += z;
    }
    if (lane == 31) m.sum[wib] = incl, m.lists[wib] = lists;
    __syncthreads();
    w.probes = m.probes;
    long long before = incl - n, all = 0;
    lists = 0;
    for (int k = 0; k < kMapThreads / 32; ++k) {
      if (k < wib) before += m.sum[k];
      all += m.sum[k];
      lists += m.lists[k];
    }
    // (the rule of k_bits_warp)
    if (2 * all >= lists && lists <= 16LL * a.items) {
      c += W <= 4 ? map_steps<K, 4>(a, w, m, unit, lists, tid)
                  : map_steps<K, 8>(a, w, m, unit, lists, tid);
      __syncthreads();
      continue;
    }
    const long long lo = share(all, unit.y, unit.z), hi = share(all, unit.y + 1, unit.z);
    const int total = (int)(hi - lo);
    if (tid < w.d0) {
      m.rel[tid] = (int)max(0LL, min(before + n - lo, (long long)total));
      m.off[tid] = before < hi && before + n > lo ? (int)(lo - before) : 0;
    }
    __syncthreads();
    uint32_t* out = m.table + wib * 32 * 8;
    for (;;) {
      int base = 0;
      if (lane == 0) base = atomicAdd(&m.next, 32);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base >= total) break;
      c += W <= 4 ? lane_steps<K, 4>(a, w, m.rel, m.off, out, base, total, lane)
                  : lane_steps<K, 8>(a, w, m.rel, m.off, out, base, total, lane);
    }
    __syncthreads();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if (lane == 0 && c) atomicAdd(a.total, c);
  wait_for_previous();
}

// --------------------------------------------------------------- per-graph index
__device__ __forceinline__ int class_of(int d) {
  return d <= 0 || d > kTopDeg ? -1 : d <= kWarpDeg ? 0 : d <= kMidDeg ? 1 : 2;
}

// sz[v] = words of v's stored rows (degree 33..1024: d(v) rows of ceil(d(v)/32)); sums[c] =
// work of the vertices of class c, sums[3 + c] their number.  A warp a vertex.
__global__ void __launch_bounds__(kThreads) k_bits_sizes(const int64_t* rowptr, const int32_t* col,
                                                         int64_t nv, int64_t* sz, int64_t* work,
                                                         unsigned long long* sums) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * kWarps;
  unsigned long long acc[6] = {0, 0, 0, 0, 0, 0};
  for (int64_t v = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5); v < nv; v += nw) {
    const int64_t rb = rowptr[v];
    const int64_t dl = rowptr[v + 1] - rb;
    const int d = (int)min(dl, (int64_t)kTopDeg + 1);
    const int cls = class_of(d);
    long long s = 0;
    if (cls >= 0)
      for (int i = lane; i < d; i += 32) {
        const int u = col[rb + i];
        s += rowptr[u + 1] - rowptr[u];
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    s = max(s, (long long)d * d);
    if (lane == 0) {
      sz[v] = cls > 0 ? (int64_t)d * ((d + 31) / 32) : 0;
      work[v] = cls >= 0 ? s : 0;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (cls == k) {
        acc[k] += (unsigned long long)s;
        acc[3 + k] += 1;
      }
  }
  if (lane == 0)
    for (int k = 0; k < 6; ++k)
      if (acc[k]) atomicAdd(sums + k, acc[k]);
}

struct UnitLists {
  int4* list[3];
  long long step[3];  // work of a unit
};

__global__ void __launch_bounds__(kThreads) k_bits_units(const int64_t* rowptr, const int64_t* work,
                                                         int64_t nv, UnitLists l,
                                                         unsigned long long* un) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * kWarps;
  for (int64_t v0 = ((int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5)) * 32; v0 < nv;
       v0 += nw * 32) {
    const int64_t v = v0 + lane;
    int cls = -1, parts = 0;
    if (v < nv) {
      cls = class_of((int)min(rowptr[v + 1] - rowptr[v], (int64_t)kTopDeg + 1));
      if (cls >= 0 && l.list[cls]) {
        const long long st = cls == 0 ? l.step[0] : cls == 1 ? l.step[1] : l.step[2];
        parts = (int)((work[v] + st - 1) / st);
      }
    }
    unsigned long long at = 0;
    if (parts) at = atomicAdd(un + cls, (unsigned long long)parts);
    if (parts > 1) atomicAdd(un + 3, (unsigned long long)parts);
    if (parts == 1) l.list[cls][at] = make_int4((int)v, 0, 1, 0);
    for (unsigned m = __ballot_sync(0xffffffffu, parts > 1); m; m &= m - 1) {
      const int src = __ffs(m) - 1;
      const int n = __shfl_sync(0xffffffffu, parts, src);
      const int cl = __shfl_sync(0xffffffffu, cls, src);
      const unsigned long long b = __shfl_sync(0xffffffffu, at, src);
      int4* out = cl == 0 ? l.list[0] : cl == 1 ? l.list[1] : l.list[2];
      for (int k = lane; k < n; k += 32) out[b + k] = make_int4((int)(v0 + src), k, n, 0);
    }
  }
}

// The stored rows: a block a unit (its share of the v0's rows), a warp a row, N(u) looked up
// in a hash table of N(v0).  R-MAT scale 12: 4.1 ms -> 32 us (a warp a vertex, a lane a
// row, binary searches).
__global__ void __launch_bounds__(kThreads) k_bits_rows(const int64_t* rowptr, const int32_t* col,
                                                        const int64_t* off, uint32_t* rows,
                                                        UnitLists l, const unsigned long long* un) {
  __shared__ __align__(16) int32_t key[4 * 1024];
  __shared__ uint16_t pos[4 * 1024];
  __shared__ int32_t n0[kTopDeg];
  __shared__ uint32_t row[kWarps][32];
  __shared__ int s_probes;
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const int64_t n1 = (int64_t)un[1], n2 = (int64_t)un[2];
  Local w;
  w.n0 = n0;
  w.t.key = key;
  w.t.pos = pos;
  for (int64_t u = blockIdx.x; u < n1 + n2; u += gridDim.x) {
    const int4 unit = u < n2 ? l.list[2][u] : l.list[1][u - n2];
    const int64_t rb = rowptr[unit.x];
    const int d0 = (int)(rowptr[unit.x + 1] - rb);
    const int r0 = (int)share(d0, unit.y, unit.z), r1 = (int)share(d0, unit.y + 1, unit.z);
    if (r0 >= r1) continue;
    const int W = (d0 + 31) >> 5;
    w.d0 = d0;
    int nb = 64;
    while (nb < 2 * d0 && nb < 1024) nb <<= 1;
    w.t.mask = nb - 1;
    w.t.shift = __clz(nb) + 1;
    __syncthreads();
    for (int i = tid; i < nb; i += kThreads) ((int4*)key)[i] = make_int4(-1, -1, -1, -1);
    for (int i = tid; i < d0; i += kThreads) n0[i] = col[rb + i];
    if (tid == 0) s_probes = 1;
    __syncthreads();
    for (int i = tid; i < d0; i += kThreads) {
      const int k = insert(w.t, n0[i], i);
      if (k > 1) atomicMax(&s_probes, k);
    }
    __syncthreads();
    w.probes = s_probes;
    uint32_t* out = rows + off[unit.x];
    for (int i = r0 + wib; i < r1; i += kWarps) {
      const int64_t b = rowptr[n0[i]];
      const uint32_t r = warp_row(w, row[wib], col + b, (int)(rowptr[n0[i] + 1] - b), lane);
      if (lane < W) out[(int64_t)i * W + lane] = r;
    }
  }
}

struct Tmp {  // freed on the stream when the build leaves
  cudaStream_t s;
  void* p = nullptr;
  ~Tmp() {
    if (p) cudaFreeAsync(p, s);
  }
};

cudaError_t build_index(const DevGraph& g, int num_sms, cudaStream_t s) {
  const int64_t nv = g.nv;
  Tmp work{s}, sums{s}, off{s}, rows{s}, units{s}, un{s};
  cudaError_t e = cudaMallocAsync(&work.p, sizeof(int64_t) * nv, s);
  if (e == cudaSuccess) e = cudaMallocAsync(&sums.p, sizeof(unsigned long long) * 6, s);
  if (e == cudaSuccess) e = cudaMallocAsync(&off.p, sizeof(int64_t) * (nv + 1), s);
  if (e == cudaSuccess) e = cudaMallocAsync(&un.p, sizeof(unsigned long long) * 4, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(sums.p, 0, sizeof(unsigned long long) * 6, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(un.p, 0, sizeof(unsigned long long) * 4, s);
  if (e != cudaSuccess) return e;
  int64_t* o = (int64_t*)off.p;
  const int wblocks = (int)std::min<int64_t>((nv + kWarps - 1) / kWarps, 65536);
  k_bits_sizes<<<wblocks, kThreads, 0, s>>>(g.rowptr_o, g.col_o, nv, o, (int64_t*)work.p,
                                            (unsigned long long*)sums.p);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = scan_excl(o, o, nv, o + nv, s);
  int64_t total = 0;
  unsigned long long h[6] = {0, 0, 0, 0, 0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(&total, o + nv, sizeof(total), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, sums.p, sizeof(h), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  // rows that do not fit leave the degrees above 32 to the list form
  bool stored = total > 0 && total * (int64_t)sizeof(uint32_t) <= kRowBudget;
  if (stored) {
    e = cudaMallocAsync(&rows.p, sizeof(uint32_t) * total, s);
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      rows.p = nullptr;
      stored = false;
    } else if (e != cudaSuccess) {
      return e;
    }
  }
  // A unit's work: enough units for every warp (block) to take several, bounded below by
  // what a unit's own set-up is worth and above by the time of one.
  UnitLists l{};
  int64_t cap[3] = {0, 0, 0};
  const long long lanes[3] = {(long long)num_sms * 40 * 4, (long long)num_sms * 4 * 4,
                              (long long)num_sms * 3};
  const long long lo[3] = {256, 256, 512}, hi[3] = {4096, 16384, 16384};
  for (int k = 0; k < 3; ++k) {
    l.step[k] = std::min(hi[k], std::max(lo[k], (long long)h[k] / lanes[k]));
    if (h[3 + k] && (k == 0 || stored)) cap[k] = (int64_t)(h[3 + k] + h[k] / l.step[k]);
  }
  e = cudaMallocAsync(&units.p, sizeof(int4) * std::max<int64_t>(1, cap[0] + cap[1] + cap[2]), s);
  if (e != cudaSuccess) return e;
  int64_t at = 0;
  for (int k = 0; k < 3; ++k) {
    l.list[k] = cap[k] ? (int4*)units.p + at : nullptr;
    g.plan_off[k] = at;
    g.plan_cap[k] = cap[k];
    at += cap[k];
  }
  k_bits_units<<<wblocks, kThreads, 0, s>>>(g.rowptr_o, (const int64_t*)work.p, nv, l,
                                            (unsigned long long*)un.p);
  e = cudaGetLastError();
  if (e == cudaSuccess && stored) {
    k_bits_rows<<<num_sms * 6, kThreads, 0, s>>>(g.rowptr_o, g.col_o, o, (uint32_t*)rows.p, l,
                                                 (const unsigned long long*)un.p);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return e;
  g.plan_items = (long long)h[1] < (long long)num_sms * kMapWork
                     ? 0
                     : (int)std::min<long long>(8192, std::max<long long>(2048, 8 * l.step[1]));
  g.plan_units = (int4*)units.p;
  g.plan_un = (unsigned long long*)un.p;
  units.p = un.p = nullptr;
  if (stored) {
    g.lut_rows = (uint32_t*)rows.p;
    g.lut_off = o;
    rows.p = off.p = nullptr;
  }
  g.plan_deg = stored || total == 0 ? kTopDeg : kWarpDeg;
  return cudaSuccess;
}

// No more blocks than there are units for: a small graph would only pay for starting them.
unsigned blocks(int most, int64_t units) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(most, units));
}

// The shared-memory opt-in of a kernel, `most` bytes, once per device.  The attribute is the
// process's: set to what each call needs, one context's launch met the smaller limit that
// another's had just set.
template <void (*KERN)(BitArgs)>
cudaError_t opt_in(int most) {
  static std::atomic<unsigned long long> opted{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (e == cudaSuccess && !(opted.load(std::memory_order_acquire) & bit)) {
    e = cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e == cudaSuccess) opted.fetch_or(bit, std::memory_order_acq_rel);
  }
  return e;
}

template <void (*KERN)(BitArgs)>
cudaError_t launch(unsigned grid, int threads, int bytes, int most, cudaStream_t s,
                   const BitArgs& a, bool first) {
  const cudaError_t e = opt_in<KERN>(most);
  return e == cudaSuccess ? launch_next(first, KERN, grid, threads, bytes, s, a) : e;
}

template <int K, int NT>
cudaError_t launch_cta(const DevGraph& g, BitArgs a, int cls, bool any, bool first,
                       unsigned long long* heads, int num_sms, cudaStream_t s) {
  constexpr int deg = NT == kThreads ? kMidDeg : kTopDeg;
  constexpr int most = cta_layout(deg, NT / 32).bytes;
  // the shared memory that the graph's own degrees need: more blocks an SM
  a.lay = cta_layout((int)std::min<int64_t>(deg, (std::max<int64_t>(g.max_deg, 1) + 127) / 128 * 128),
                     NT / 32);
  cudaError_t e = opt_in<k_bits_cta<K, NT>>(most);
  int per_sm = 1;
  if (e == cudaSuccess && any)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bits_cta<K, NT>, NT, a.lay.bytes);
  if (e != cudaSuccess) return e;
  a.cls = cls;
  a.units = g.plan_units + g.plan_off[cls];
  a.head = heads + cls;
  return launch<k_bits_cta<K, NT>>(blocks(num_sms * std::max(per_sm, 1), g.plan_cap[cls]), NT,
                                   a.lay.bytes, most, s, a, first);
}

template <int K>
cudaError_t launch_k(const DevGraph& g, BitArgs a, unsigned long long* heads, int num_sms,
                     cudaStream_t s, int* launches) {
  // the larger degrees first; each kernel's tail is the next one's beginning (P7 on R-MAT scale
  // 11 0.54 -> 0.39 ms, on scale 12 1.32 -> 1.05, against one after the other)
  bool first = true;
  if (g.plan_deg > kMidDeg && g.max_deg > kMidDeg && g.lut_rows) {
    cudaError_t e = launch_cta<K, kTopThreads>(g, a, 2, true, first, heads, num_sms, s);
    if (e != cudaSuccess) return e;
    ++*launches;
    first = false;
  }
  // launched for graphs without such a degree too (one block that finds no unit), so that
  // a plan's launches do not depend on the degrees below the list form's
  const bool any = g.max_deg > kWarpDeg;
  cudaError_t e;
  if (a.p.stream && g.plan_items) {
    a.cls = 1;
    a.units = g.plan_units + g.plan_off[1];
    a.head = heads + 1;
    a.items = g.plan_items;
    e = launch<k_bits_map<K>>(blocks(num_sms * kMapBlocks, g.plan_cap[1]), kMapThreads,
                              (int)sizeof(MapSmem), (int)sizeof(MapSmem), s, a, first);
  } else {
    e = launch_cta<K, kThreads>(g, a, 1, any, first, heads, num_sms, s);
  }
  if (e != cudaSuccess) return e;
  a.cls = 0;
  a.units = g.plan_units + g.plan_off[0];
  a.head = heads;
  constexpr int most = kWarps * (int)(sizeof(SmallWarp) + sizeof(SmallMap));
  const int bytes = a.p.stream ? most : kWarps * (int)sizeof(SmallWarp);
  e = launch<k_bits_warp<K>>(blocks(num_sms * 4, (g.plan_cap[0] + kWarps - 1) / kWarps), kThreads,
                             bytes, most, s, a, false);
  if (e != cudaSuccess) return e;
  *launches += 2;
  return cudaSuccess;
}

}  // namespace

cudaError_t ensure_plan_index(const DevGraph& g, int num_sms, cudaStream_t s) {
  auto build = [&] {
    g.plan_deg = -1;
    if (g.nv == 0 || g.ne == 0) return cudaSuccess;
    const cudaError_t e = build_index(g, num_sms, s);
    if (e == cudaErrorMemoryAllocation) {  // no room: every task stays on the list form
      cudaGetLastError();
      return cudaSuccess;
    }
    if (e != cudaSuccess) g.plan_deg = 0;
    return e;
  };
  return build_once(
      g, s, [&] { return g.plan_deg != 0; }, build);
}

int bits_launches(const DevGraph& g) {
  if (g.plan_deg <= 0) return 0;
  return g.plan_deg > kMidDeg && g.max_deg > kMidDeg && g.lut_rows ? 3 : 2;
}

cudaError_t launch_bits(const DevGraph& g, const BitPlan& p, unsigned long long* heads,
                        unsigned long long* total, int64_t* split_out, int num_sms,
                        cudaStream_t s, int* launches) {
  if (g.plan_deg <= 0) return cudaSuccess;
  BitArgs a{};
  a.rowptr = g.rowptr_o;
  a.col = g.col_o;
  a.rows = g.lut_rows;
  a.roff = g.lut_off;
  a.un = g.plan_un;
  a.total = total;
  a.split_out = split_out;
  a.p = p;
  return p.k == 4 ? launch_k<4>(g, a, heads, num_sms, s, launches)
                  : launch_k<5>(g, a, heads, num_sms, s, launches);
}

}  // namespace xgm
