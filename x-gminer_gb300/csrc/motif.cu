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

// Sum of t(v) (deg(v) - 2), t(v) the triangles of v (the task kernel's; the owner kernel counts
// them per edge, k_motif_terms).
__global__ void __launch_bounds__(kThreads) k_tailed_reduce(GView g, const unsigned long long* vpart,
                                                            unsigned long long* out) {
  unsigned long long acc = 0;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < g.nv;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t d = g.rowptr[r + 1] - g.rowptr[r];
    if (d > 2) acc += vpart[r] * (unsigned long long)(d - 2);
  }
  acc = warp_sum_u64(acc);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd(out, acc);
}

// out[3], out[6] of k_motif_terms alone (tailed triangles), LANES lanes per vertex: only edges
// in a triangle look their ends up.  A call on Erdos-Renyi 2^20, degree 32 (few such edges) 1.71
// ms with all of k_motif_terms' sums, 1.37 (16 lanes 1.41; 1.47 from triangles per vertex, the
// task kernel); R-MAT s22 21.7 -> 20.5.
template <int LANES>
__global__ void __launch_bounds__(kThreads) k_tailed_edges(GView g, const unsigned* epart,
                                                           unsigned long long* out) {
  const int l = threadIdx.x & (LANES - 1);
  const int64_t groups = (int64_t)gridDim.x * (kThreads / LANES);
  unsigned long long lo = 0, hi = 0;
  for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / LANES; r < g.nv; r += groups) {
    const longlong2 p = g.dptr[r];
    for (long long j = p.x + l; j < p.y; j += LANES) {
      const unsigned long long n = epart[j];
      if (!n) continue;  // (else both ends have degree >= 2)
      const int32_t v = ldg_i32(g.col + j);
      const long long d = p.y - g.rowptr[r], dv = g.dptr[v].y - g.rowptr[v];
      const unsigned long long t = n * (unsigned long long)(d + dv - 4);
      lo += t & 0xFFFFFFFFull;
      hi += t >> 32;
    }
  }
  lo = warp_sum_u64(lo);
  hi = warp_sum_u64(hi);
  if ((threadIdx.x & 31) == 0) {
    if (lo) atomicAdd(out + 3, lo);
    if (hi) atomicAdd(out + 6, hi);
  }
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
  let_next_start();
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
  wait_for_previous();
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

// Per-graph sums from the triangles per edge (batched graphs): diamonds to out, three times
// the triangles and (TAIL) twice the tailed triangles (low and high 32-bit halves) to
// sums[3 gid].  A warp streams the rows of 32 consecutive ranks, 16 bytes a lane (entries of
// lower neighbours are zero); graphs are contiguous in rank order, so most blocks belong to
// one graph and end in one atomic per sum.  (A thread per vertex walking its out-list: 368
// us on 5.2 M vertices.)
template <bool TAIL>
__global__ void __launch_bounds__(kThreads) k_graph_terms(GView g, const int32_t* gid,
                                                          const unsigned* epart,
                                                          unsigned long long* out, int stride,
                                                          int slot_d, unsigned long long* sums) {
  __shared__ int64_t row_s[kThreads / 32][33];
  let_next_start();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t* row = row_s[warp];
  const int64_t nwarps = (int64_t)gridDim.x * (kThreads / 32);
  for (int64_t r0 = 32 * ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5); r0 < g.nv;
       r0 += 32 * nwarps) {
    const int64_t r1 = r0 + 32 < g.nv ? r0 + 32 : g.nv;
    __syncwarp();
    row[lane] = g.rowptr[r0 + lane < r1 ? r0 + lane : r1];
    if (lane == 0) row[32] = g.rowptr[r1];
    __syncwarp();
    const int64_t e0 = row[0], e1 = row[32];
    const int32_t first = gid[r0];
    const bool one = gid[r1 - 1] == first;  // one graph
    unsigned long long dia = 0, tri = 0, lo = 0, hi = 0;
    for (int64_t q = (e0 >> 2) + lane; 4 * q < e1; q += 32) {
      // (epart holds whole 16-byte units; a unit may begin or end in a neighbouring row)
      const uint4 c4 = __ldcs(reinterpret_cast<const uint4*>(epart) + q);
      if (!(c4.x | c4.y | c4.z | c4.w)) continue;
      const unsigned cs[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int64_t e = 4 * q + h;
        const unsigned long long n = cs[h];
        if (!n || e < e0 || e >= e1) continue;
        if (!TAIL && one) {
          dia += n * (n - 1) / 2;
          tri += n;
          continue;
        }
        int r = 0;  // the entry's row: largest with row[r] <= e
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
          if (row[r + d] <= e) r += d;
        unsigned long long t = 0;
        if (TAIL) {
          const int32_t v = ldg_i32(g.col + e);
          t = n * (unsigned long long)(row[r + 1] - row[r] + (g.dptr[v].y - g.rowptr[v]) - 4);
        }
        if (one) {
          dia += n * (n - 1) / 2;
          tri += n;
          lo += t & 0xFFFFFFFFull;
          hi += t >> 32;
        } else {
          const int64_t gg = gid[r0 + r];
          if (slot_d >= 0 && n > 1) atomicAdd(&out[gg * stride + slot_d], n * (n - 1) / 2);
          atomicAdd(&sums[3 * gg], n);
          if (TAIL) {
            atomicAdd(&sums[3 * gg + 1], t & 0xFFFFFFFFull);
            if (t >> 32) atomicAdd(&sums[3 * gg + 2], t >> 32);
          }
        }
      }
    }
    if (!one) continue;
    dia = warp_sum_u64(dia);
    tri = warp_sum_u64(tri);
    if (TAIL) lo = warp_sum_u64(lo), hi = warp_sum_u64(hi);
    if (lane == 0 && tri) {
      if (slot_d >= 0 && dia) atomicAdd(&out[(int64_t)first * stride + slot_d], dia);
      atomicAdd(&sums[3 * (int64_t)first], tri);
      if (TAIL) {
        atomicAdd(&sums[3 * (int64_t)first + 1], lo);
        if (hi) atomicAdd(&sums[3 * (int64_t)first + 2], hi);
      }
    }
  }
  wait_for_previous();
}

// Triangles and tailed triangles per graph from the sums (a slot < 0 is skipped).
__global__ void k_graph_finish(const unsigned long long* sums, int graphs, unsigned long long* out,
                               int stride, int slot_tri, int slot_t) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < graphs;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (slot_tri >= 0) out[i * stride + slot_tri] = sums[3 * i] / 3;
    if (slot_t >= 0) {  // (high half << 32 + low half) / 2
      const unsigned long long lo = sums[3 * i + 1], hi = sums[3 * i + 2];
      const unsigned long long low = lo + (hi << 32), carry = low < lo;
      out[i * stride + slot_t] = (low >> 1) | (((hi >> 32) + carry) << 63);
    }
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

cudaError_t launch_tailed_reduce(const GView& g, const unsigned long long* vpart,
                                 unsigned long long* out, cudaStream_t s) {
  if (g.nv == 0) return cudaSuccess;
  k_tailed_reduce<<<std::min(grid_for(g.nv), kReduceBlocks), kThreads, 0, s>>>(g, vpart, out);
  return cudaGetLastError();
}

cudaError_t launch_tailed_edges(const GView& g, int64_t ne_dag, const unsigned* epart,
                                unsigned long long* out, cudaStream_t s) {
  if (g.nv == 0) return cudaSuccess;
  // eight lanes up to 32 out-neighbours a vertex on average
  const bool narrow = ne_dag <= 32 * g.nv;
  const unsigned grid = std::min(grid_for(g.nv * (narrow ? 8 : 32)), kReduceBlocks);
  if (narrow) k_tailed_edges<8><<<grid, kThreads, 0, s>>>(g, epart, out);
  else k_tailed_edges<32><<<grid, kThreads, 0, s>>>(g, epart, out);
  return cudaGetLastError();
}

cudaError_t launch_motif_terms(const GView& g, const unsigned* epart, unsigned long long* out,
                               cudaStream_t s, bool next) {
  if (g.nv == 0) return cudaSuccess;
  return launch_next(!next, k_motif_terms, std::min(grid_for(g.nv * 32), kReduceBlocks), kThreads,
                     0, s, g, epart, out);
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

cudaError_t launch_graph_terms(const GView& g, const int32_t* gid, int graphs,
                               const unsigned* epart, unsigned long long* sums,
                               unsigned long long* out, int stride, int slot_tri, int slot_d,
                               int slot_t, cudaStream_t s, bool next) {
  if (g.nv == 0) return cudaSuccess;
  const unsigned grid = std::min(grid_for(g.nv), kReduceBlocks);
  const cudaError_t e = launch_next(!next, slot_t >= 0 ? k_graph_terms<true> : k_graph_terms<false>,
                                    grid, kThreads, 0, s, g, gid, epart, out, stride, slot_d, sums);
  if (e != cudaSuccess) return e;
  k_graph_finish<<<grid_for(graphs), kThreads, 0, s>>>(sums, graphs, out, stride, slot_tri, slot_t);
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
