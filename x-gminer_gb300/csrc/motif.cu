// Edge-induced 4-vertex motif plans on the undirected graph (rank ids).
//
// Reference (CPU, the counting definitions): codes/GraphMiner/src/count/omp_base.cc:5-58
// with cpu_kernels/diamond.h:1-8, rectangle.h:1-46 and tailedtriangle.h:1-12; GPU
// analogues codes/GraphMiner/src/count/gpu_base.cu:1-104.
//
//  diamond        = sum over undirected edges e of C(n_e, 2), n_e = |N(u) & N(v)| =
//                   number of triangles containing e.
//  tailed triangle = sum over v with deg(v) > 2 of t(v) * (deg(v) - 2), t(v) = number
//                   of triangles containing v = half the sum of n_e over v's edges.
//  4-cycle        = for every v0, wedges v0-v1-v2 with v1 < v0 and v2 < v0 grouped by
//                   v2; a group of c wedges closes C(c, 2) cycles.
// n_e and t(v) come from one triangle-participation pass of the DAG kernels
// (clique.cu); the 4-cycle plan has its own kernels (cycle4.cu).
#include "clique.cuh"
#include "motif.cuh"

namespace xgm {

namespace {

constexpr int kThreads = 256;
constexpr unsigned kReduceBlocks = 152 * 8;  // of a reduction: every SM full, once

// Sum of C(n, 2) over all entries (16 bytes a load; entries of lower neighbours are zero).
__global__ void __launch_bounds__(kThreads) k_diamond_reduce(const unsigned* epart, int64_t ne,
                                                             unsigned long long* out) {
  unsigned long long acc = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t n4 = ne >> 2;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n4; e += stride) {
    const uint4 c = __ldcs(reinterpret_cast<const uint4*>(epart) + e);
    if (!(c.x | c.y | c.z | c.w)) continue;
    const unsigned cs[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const unsigned long long n = cs[h];
      acc += n * (n - (n > 0)) / 2;
    }
  }
  for (int64_t e = 4 * n4 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < ne; e += stride) {
    const unsigned long long n = epart[e];
    acc += n * (n - (n > 0)) / 2;
  }
  acc = warp_sum_u64(acc);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd(out, acc);
}

// C(d, 3) in wrapping uint64 arithmetic without an intermediate overflow for d < 2^32:
// 3 divides one of d, d-1, d-2; when it does not divide x = d(d-1)/2 it divides d-2.
__device__ __forceinline__ unsigned long long choose3(unsigned long long d) {
  if (d < 3) return 0;
  const unsigned long long x = d * (d - 1) / 2;
  return x % 3 == 0 ? (x / 3) * (d - 2) : x * ((d - 2) / 3);
}

// The sums behind the motif identities, one warp per vertex (lane 0: vertex terms;
// lanes stride the out-neighbours for the edge terms), wrapping uint64:
//   out[0] = sum_v C(d_v, 2)                 edge-induced wedges
//   out[1] = sum_v C(d_v, 3)                 edge-induced 3-stars
//   out[2] = sum_{uv in E} (d_u-1)(d_v-1)    3-edge walks x-u-v-y, x != v, y != u
//   out[3] = 2 sum_v t_v (d_v - 2)           twice the edge-induced tailed triangles, as
//   out[6]                                   the sum of low and of high 32-bit halves
//   out[4] = sum_{uv in E} C(t_uv, 2)        edge-induced diamonds
//   out[5] = sum_{uv in E} t_uv              3 x triangles
// t_uv are the triangle-participation counters (epart, null for the 3-vertex census: out[3..6]
// stay 0); t_v is half the sum of t over v's edges, so out[3] is sum t_uv (d_u + d_v - 4).
// Few blocks: a sum costs one atomic per warp and term.
__global__ void __launch_bounds__(kThreads) k_motif_terms(GView g, const unsigned* epart,
                                                          unsigned long long* out) {
  const int lane = threadIdx.x & 31;
  unsigned long long acc[7] = {0, 0, 0, 0, 0, 0, 0};
  const int64_t nwarps = (int64_t)gridDim.x * (kThreads / 32);
  for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < g.nv; r += nwarps) {
    const unsigned long long d = (unsigned long long)(g.rowptr[r + 1] - g.rowptr[r]);
    if (lane == 0) {
      acc[0] += d * (d - (d > 0)) / 2;
      acc[1] += choose3(d);
    }
    const longlong2 p = g.dptr[r];
    for (long long j = p.x + lane; j < p.y; j += 32) {
      const int32_t v = ldg_i32(g.col + j);
      const unsigned long long dv = (unsigned long long)(g.rowptr[v + 1] - g.rowptr[v]);
      acc[2] += (d - 1) * (dv - 1);
      if (epart) {
        const unsigned long long n = epart[j];
        if (n) {  // both ends have degree >= 2; n < 2^31, degrees < 2^31
          acc[4] += n * (n - 1) / 2;
          acc[5] += n;
          const unsigned long long t = n * (d + dv - 4);
          acc[3] += t & 0xFFFFFFFFull;
          acc[6] += t >> 32;
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    const unsigned long long w = warp_sum_u64(acc[i]);
    if (lane == 0 && w) atomicAdd(out + i, w);
  }
}

// Entries of row v1 below v0: col[rowptr[v1] .. first index with col >= v0).
__device__ __forceinline__ long long lower_end(const GView& g, int32_t v1, int32_t v0) {
  long long lo = g.rowptr[v1], hi = g.dptr[v1].y;
  while (lo < hi) {
    long long mid = (lo + hi) >> 1;
    if (ldg_i32(g.col + mid) < v0) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// wedges[r] = number of wedges r-v1-v2 with v1, v2 < r.  Warp per vertex.
__global__ void k_wedge_count(GView g, long long* wedges) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < g.nv; r += warps) {
    const long long a0 = g.rowptr[r], a1 = g.dptr[r].x;  // lower neighbours
    long long w = 0;
    for (long long e = a0 + lane; e < a1; e += 32) {
      const int32_t v1 = ldg_i32(g.col + e);
      w += lower_end(g, v1, (int32_t)r) - g.rowptr[v1];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w += __shfl_down_sync(kFull, w, o);
    if (lane == 0) wedges[r] = w;
  }
}

// Per-graph diamond / tailed-triangle totals from the participation counters: block
// of consecutive rank ids (graphs are contiguous in rank order), shared-memory
// aggregation by graph id, then one atomic per (block, graph).
__global__ void k_part_reduce_graphs(GView g, const int32_t* gid,
                                     const unsigned long long* vpart, const unsigned* epart,
                                     unsigned long long* out, int stride, int slot_d, int slot_t) {
  __shared__ unsigned long long sd[kThreads], st[kThreads];
  __shared__ int32_t gfirst;
  for (int64_t base = (int64_t)blockIdx.x * kThreads; base < g.nv;
       base += (int64_t)gridDim.x * kThreads) {
    sd[threadIdx.x] = 0;
    st[threadIdx.x] = 0;
    if (threadIdx.x == 0) gfirst = gid[base];
    __syncthreads();
    const int64_t r = base + threadIdx.x;
    if (r < g.nv) {
      const longlong2 d = g.dptr[r];
      const long long deg = d.y - g.rowptr[r];
      unsigned long long dia = 0;
      if (slot_d >= 0)
        for (long long e = d.x; e < d.y; ++e) {
          const unsigned long long c = epart[e];
          dia += c * (c - (c > 0)) / 2;
        }
      const unsigned long long tt = (slot_t >= 0 && deg > 2) ? vpart[r] * (unsigned long long)(deg - 2) : 0;
      const int k = gid[r] - gfirst;  // < kThreads: ids are non-decreasing in rank order
      if (dia) atomicAdd(&sd[k], dia);
      if (tt) atomicAdd(&st[k], tt);
    }
    __syncthreads();
    const long long gg = (long long)gfirst + threadIdx.x;
    if (slot_d >= 0 && sd[threadIdx.x]) atomicAdd(&out[gg * stride + slot_d], sd[threadIdx.x]);
    if (slot_t >= 0 && st[threadIdx.x]) atomicAdd(&out[gg * stride + slot_t], st[threadIdx.x]);
    __syncthreads();
  }
}

inline unsigned grid_for(int64_t n) {
  int64_t b = (n + kThreads - 1) / kThreads;
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(b, int64_t(1) << 20));
}

}  // namespace

cudaError_t launch_diamond_reduce(const unsigned* epart, int64_t ne, unsigned long long* out,
                                  cudaStream_t s) {
  k_diamond_reduce<<<std::min(grid_for((ne + 3) / 4), kReduceBlocks), kThreads, 0, s>>>(epart, ne,
                                                                                       out);
  return cudaGetLastError();
}

cudaError_t launch_motif_terms(const GView& g, const unsigned* epart, unsigned long long* out,
                               cudaStream_t s) {
  if (g.nv == 0) return cudaSuccess;
  k_motif_terms<<<std::min(grid_for(g.nv * 32), kReduceBlocks), kThreads, 0, s>>>(g, epart, out);
  return cudaGetLastError();
}

uint64_t tailed_from_terms(const unsigned long long* terms) {
  const unsigned __int128 twice = ((unsigned __int128)terms[6] << 32) + terms[3];
  return (uint64_t)(twice >> 1);
}

cudaError_t launch_wedge_count(const GView& g, long long* wedges, cudaStream_t s) {
  if (g.nv == 0) return cudaSuccess;
  k_wedge_count<<<grid_for(g.nv * 32), kThreads, 0, s>>>(g, wedges);
  return cudaGetLastError();
}

cudaError_t launch_part_reduce_graphs(const GView& g, const int32_t* gid,
                                      const unsigned long long* vpart, const unsigned* epart,
                                      unsigned long long* out, int stride, int slot_d, int slot_t,
                                      cudaStream_t s) {
  if (g.nv == 0) return cudaSuccess;
  k_part_reduce_graphs<<<grid_for(g.nv), kThreads, 0, s>>>(g, gid, vpart, epart, out, stride,
                                                           slot_d, slot_t);
  return cudaGetLastError();
}

}  // namespace xgm
