// Triangles from the side of the later endpoint ("owner"), hand-written for sm_103a.
//
// Reference kernel this replaces: warp_edge (TC),
// codes/GraphMiner/src/triangle/gpu_kernels/bs_warp_edge.cuh:1-20.
//
// Every triangle v < u < x of the degree-oriented DAG is found at its edge (v, u): x lies
// in N+(u) and in the part of N+(v) after u (its suffix).  Testing suffixes costs
// sum_v C(d+(v), 2) probes, whereas streaming N+(u) against a filter of N+(v) costs
// sum_(v,u) d+(u): at R-MAT scale 22 7.2 G against 29 G elements, because the
// out-neighbours u of a low vertex are hubs with long lists.
//
//  - big u (degree > kBigDeg): a CTA holds N+(u) as a bitmap over [u + 1, V) and takes up
//    to kOwnChunk in-neighbours v of u.  A thread finds u's place in N+(v) by binary
//    search (N+(v) is sorted); suffixes of up to kOwnShort elements are tested by that
//    thread, longer ones go to a table in shared memory and are tested by whole warps,
//    32 consecutive elements at a time.  A hub's in-neighbours are many units (u, chunk)
//    that any CTA can take.
//  - the other u: one lane per edge (v, u) merges the suffix with N+(u); both are short
//    (deg v <= deg u <= kBigDeg).
// Measured (GB300): triangles of R-MAT scale 20, ef 16: 8.45 -> 2.05 ms a call; of a
// Barabasi-Albert graph of 3,312 vertices 115 -> 41 us (13 launches -> 1: no task lists).
// Bound: instruction issue (74 % active, 27 of 32 threads per instruction, L2 hit 95 %).
// Bitmaps are cleared by taking the inserted bits out again: a unit costs d+(u) stores,
// not the bitmap's size.
#include <algorithm>

#include "rows.cuh"

namespace xgm {

namespace {

constexpr int kOwnThreads = 256;
constexpr int kOwnWarps = kOwnThreads / 32;
constexpr int kOwnChunk = 512;   // in-neighbours of one unit (two per thread)
constexpr int kOwnShort = 12;    // longest suffix one thread tests by itself
constexpr int kOwnLevels = 512;  // most units of one owner (host: raises the chunk above it)
constexpr int kSmallStep = 128;  // vertices per claim of the small phase

struct OwnArgs {
  GView g;
  int64_t big0;    // first big rank
  int64_t chunk;   // in-neighbours per unit: a multiple of kOwnChunk
  int levels;      // units of the vertex of the largest degree
  int words;       // bitmap words
};

struct OwnPair {
  long long p;  // first element of the suffix
  int len;      // its length
};

// Elements two sorted ranges of col have in common.
__device__ __forceinline__ unsigned merge_count(const int32_t* col, long long a, long long ea,
                                                long long b, long long eb) {
  if (a >= ea || b >= eb) return 0u;
  unsigned acc = 0;
  int32_t x = ldg_i32(col + a), y = ldg_i32(col + b);
  for (;;) {
    const bool le = x <= y, ge = x >= y;
    acc += (le && ge) ? 1u : 0u;
    a += le;
    b += ge;
    if (a >= ea || b >= eb) return acc;
    if (le) x = ldg_i32(col + a);
    if (ge) y = ldg_i32(col + b);
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

__global__ void __launch_bounds__(kOwnThreads) k_owner_count(OwnArgs a, OwnHeads* heads,
                                                             unsigned long long* count) {
  extern __shared__ uint32_t bm[];
  __shared__ OwnPair tab[kOwnChunk];
  __shared__ int lev[kOwnLevels + 1];  // lev[l]: units of levels above l (highest first)
  __shared__ int n_long, claim;
  __shared__ long long unit_s;
  const GView& g = a.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned long long acc = 0;

  if (a.big0 < g.nv) {
    for (int w = tid; w < a.words; w += kOwnThreads) bm[w] = 0u;
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
    if (tid == 0) n_long = 0, claim = 0, unit_s = (long long)atomicAdd(&heads->big, 1ull);
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
      const bool live = du.x < du.y && c0 < c1;  // uniform
      if (!live) __syncthreads();  // every thread has read unit_s
      for (long long cc = c0; live && cc < c1; cc += kOwnChunk) {
        // insert N+(u) (first pass) while the in-neighbours look u up in their lists
        if (cc == c0)
          for (long long e = du.x + tid; e < du.y; e += kOwnThreads) {
            const uint32_t off = (uint32_t)(ldg_i32(g.col + e) - (int32_t)u - 1);
            atomicOr(&bm[off >> 5], 1u << (off & 31));
          }
        long long p[2];
        int len[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const long long e = cc + h * kOwnThreads + tid;
          len[h] = 0;
          if (e < c1) {
            const longlong2 dv = ldg_ll2(g.dptr + ldg_i32(g.col + e));
            const long long at = lower_at(g.col, dv.x, dv.y, (int32_t)u);
            p[h] = at + 1;
            len[h] = (int)(dv.y - at - 1);
            if (len[h] > kOwnShort) {
              const int k = atomicAdd(&n_long, 1);
              tab[k].p = p[h];
              tab[k].len = len[h];
            }
          }
        }
        __syncthreads();
        unsigned part = 0;
        const int32_t base = (int32_t)u + 1;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (len[h] <= kOwnShort)
            for (int k = 0; k < len[h]; ++k) {
              const uint32_t off = (uint32_t)(ldg_i32(g.col + p[h] + k) - base);
              part += (bm[off >> 5] >> (off & 31)) & 1u;
            }
        const int nl = n_long;
        for (;;) {
          int k = 0;
          if (lane == 0) k = atomicAdd(&claim, 2);
          k = __shfl_sync(kFull, k, 0);
          if (k >= nl) break;
#pragma unroll 1
          for (int k2 = k; k2 < k + 2 && k2 < nl; ++k2) {
            const int32_t* q = g.col + tab[k2].p;
            const int n = tab[k2].len;
            for (int e = lane; e < n; e += 128) {  // four independent loads per pass
              int32_t x[4];
#pragma unroll
              for (int h = 0; h < 4; ++h) x[h] = e + 32 * h < n ? ldg_i32(q + e + 32 * h) : -1;
#pragma unroll
              for (int h = 0; h < 4; ++h) {
                const uint32_t off = (uint32_t)(x[h] - base);
                if (x[h] >= 0) part += (bm[off >> 5] >> (off & 31)) & 1u;
              }
            }
          }
        }
        acc += part;
        __syncthreads();
        if (tid == 0) n_long = 0, claim = 0;
        if (cc + kOwnChunk < c1) __syncthreads();
      }
      if (tid == 0) unit_s = (long long)atomicAdd(&heads->big, 1ull);
      if (live)
        for (long long e = du.x + tid; e < du.y; e += kOwnThreads)
          bm[(uint32_t)(ldg_i32(g.col + e) - (int32_t)u - 1) >> 5] = 0u;
      __syncthreads();
    }
  }

  // small u: v < u < big0, one lane per edge (v, u) with a non-empty suffix
  const long long nsm = a.big0;
  for (;;) {
    long long vb = 0;
    if (lane == 0) vb = (long long)atomicAdd(&heads->small, (unsigned long long)kSmallStep);
    vb = __shfl_sync(kFull, vb, 0);
    if (vb >= nsm) break;
    const long long ve = vb + kSmallStep < nsm ? vb + kSmallStep : nsm;
    for (long long b = vb; b < ve; b += 32) {
      longlong2 d = make_longlong2(0, 0);
      int cnt = 0;
      if (b + lane < ve) {
        d = ldg_ll2(g.dptr + (nsm - 1 - (b + lane)));  // longest lists first
        cnt = (int)(d.y - d.x) - 1;
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
        if (k < total) {
          const long long at = base + (k - ex);
          const longlong2 du = ldg_ll2(g.dptr + ldg_i32(g.col + at));
          acc += merge_count(g.col, at + 1, end, du.x, du.y);
        }
      }
    }
  }
  acc = warp_sum_u64(acc);
  if (lane == 0 && acc) atomicAdd(count, acc);
}

}  // namespace

cudaError_t launch_owner_count(const DevGraph& g, OwnHeads* heads, unsigned long long* count,
                               int num_sms, cudaStream_t s) {
  if (g.nv == 0) return cudaSuccess;
  OwnArgs a;
  a.g = g.view();
  const int64_t nbig = std::min<int64_t>(g.n_big, kOwnBits);
  a.big0 = g.nv - nbig;
  const int64_t per = (g.max_deg + kOwnLevels - 1) / kOwnLevels;
  a.chunk = std::max<int64_t>(kOwnChunk, (per + kOwnChunk - 1) / kOwnChunk * kOwnChunk);
  a.levels = (int)std::max<int64_t>(1, (g.max_deg + a.chunk - 1) / a.chunk);
  a.words = (int)((nbig + 31) / 32);
  const int smem = 4 * std::max(a.words, 1);
  int per_sm = 0;
  cudaError_t e =
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_owner_count, kOwnThreads, smem);
  if (e != cudaSuccess) return e;
  // no more CTAs than there is work for: small graphs would only pay for starting them
  const int64_t want = std::max<int64_t>(nbig, (g.nv + kSmallStep * kOwnWarps - 1) /
                                                   (kSmallStep * kOwnWarps));
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)per_sm * num_sms, want));
  k_owner_count<<<(unsigned)grid, kOwnThreads, smem, s>>>(a, heads, count);
  return cudaGetLastError();
}

}  // namespace xgm
