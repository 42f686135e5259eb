// Device-wide primitives used by the CSR build and the scheduler: exclusive scan and
// LSD radix sort of 64-bit keys.  Written for this engine; no library sort or scan is
// on the path.
#include <algorithm>
#include <utility>

#include "prim.cuh"

namespace xgm {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048

template <class T>
__device__ __forceinline__ int64_t as_i64(T v) { return (int64_t)v; }

// Block-wide exclusive scan of one int64 per thread; returns the block total too.
__device__ __forceinline__ int64_t block_excl_scan(int64_t v, int64_t* total) {
  __shared__ int64_t warp_tot[kScanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int64_t y = __shfl_up_sync(kFull, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) warp_tot[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int64_t w = lane < kScanThreads / 32 ? warp_tot[lane] : 0;
    int64_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int64_t y = __shfl_up_sync(kFull, wi, o);
      if (lane >= o) wi += y;
    }
    if (lane < kScanThreads / 32) warp_tot[lane] = wi - w;  // exclusive
    if (lane == kScanThreads / 32 - 1) *total = wi;
  }
  __syncthreads();
  int64_t r = warp_tot[warp] + inc - v;
  __syncthreads();
  return r;
}

template <class T>
__global__ void __launch_bounds__(kScanThreads) k_tile_reduce(const T* in, int64_t n,
                                                              int64_t* partial) {
  __shared__ int64_t red[kScanThreads / 32];
  int64_t base = (int64_t)blockIdx.x * kScanTile;
  int64_t s = 0;
#pragma unroll
  for (int t = 0; t < kScanItems; ++t) {
    int64_t i = base + t * kScanThreads + threadIdx.x;
    if (i < n) s += as_i64(in[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(kFull, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    int64_t t = 0;
    for (int w = 0; w < kScanThreads / 32; ++w) t += red[w];
    partial[blockIdx.x] = t;
  }
}

// out[i] = offset(tile) + exclusive prefix within the tile.  in and out may alias.
template <class T>
__global__ void __launch_bounds__(kScanThreads) k_tile_scan(const T* in, int64_t* out, int64_t n,
                                                            const int64_t* tile_off,
                                                            int64_t* total) {
  __shared__ int64_t buf[kScanTile];
  __shared__ int64_t btotal;
  int64_t base = (int64_t)blockIdx.x * kScanTile;
#pragma unroll
  for (int t = 0; t < kScanItems; ++t) {
    int64_t i = base + t * kScanThreads + threadIdx.x;
    buf[t * kScanThreads + threadIdx.x] = i < n ? as_i64(in[i]) : 0;
  }
  __syncthreads();
  int64_t v[kScanItems];
  int64_t s = 0;
#pragma unroll
  for (int t = 0; t < kScanItems; ++t) {
    v[t] = buf[threadIdx.x * kScanItems + t];
    s += v[t];
  }
  int64_t off = block_excl_scan(s, &btotal) + (tile_off ? tile_off[blockIdx.x] : 0);
#pragma unroll
  for (int t = 0; t < kScanItems; ++t) {
    buf[threadIdx.x * kScanItems + t] = off;
    off += v[t];
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < kScanItems; ++t) {
    int64_t i = base + t * kScanThreads + threadIdx.x;
    if (i < n) out[i] = buf[t * kScanThreads + threadIdx.x];
  }
  if (total && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
    *total = (tile_off ? tile_off[blockIdx.x] : 0) + btotal;
}

template <class T>
cudaError_t scan_impl(const T* in, int64_t* out, int64_t n, int64_t* total, cudaStream_t st) {
  if (n <= 0) {
    if (total) return cudaMemsetAsync(total, 0, sizeof(int64_t), st);
    return cudaSuccess;
  }
  int64_t tiles = (n + kScanTile - 1) / kScanTile;
  if (tiles == 1) {
    k_tile_scan<T><<<1, kScanThreads, 0, st>>>(in, out, n, nullptr, total);
    return cudaGetLastError();
  }
  int64_t* partial = nullptr;
  cudaError_t e = cudaMallocAsync(&partial, sizeof(int64_t) * tiles, st);
  if (e != cudaSuccess) return e;
  k_tile_reduce<T><<<(unsigned)tiles, kScanThreads, 0, st>>>(in, n, partial);
  e = scan_impl<int64_t>(partial, partial, tiles, nullptr, st);
  if (e == cudaSuccess) {
    k_tile_scan<T><<<(unsigned)tiles, kScanThreads, 0, st>>>(in, out, n, partial, total);
    e = cudaGetLastError();
  }
  cudaFreeAsync(partial, st);
  return e;
}

// ------------------------------------------------------------------ radix sort
constexpr int kSortWarps = 8;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortWarps * 32 * kSortItems;  // 2048 keys
constexpr int kRadix = 256;

__global__ void __launch_bounds__(kSortWarps * 32) k_radix_hist(const uint64_t* keys, int64_t n,
                                                               int shift, int digits,
                                                               int64_t* counts, int64_t tiles) {
  __shared__ uint32_t h[kRadix];
  for (int d = threadIdx.x; d < digits; d += blockDim.x) h[d] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kSortTile + threadIdx.x;
  uint64_t k[kSortItems];
#pragma unroll
  for (int t = 0; t < kSortItems; ++t) {
    const int64_t i = base + t * kSortWarps * 32;
    k[t] = i < n ? keys[i] : 0ull;
  }
#pragma unroll
  for (int t = 0; t < kSortItems; ++t)
    if (base + t * kSortWarps * 32 < n) atomicAdd(&h[(k[t] >> shift) & (digits - 1)], 1u);
  __syncthreads();
  for (int d = threadIdx.x; d < digits; d += blockDim.x) counts[(int64_t)d * tiles + blockIdx.x] = h[d];
}

// Stable scatter: warp w of the tile owns keys [w*256, (w+1)*256) of the tile and
// walks them in 8 rounds of 32; a ballot per digit bit groups equal digits inside a round
// so each key gets its rank among equal digits in tile order.  The keys are then
// placed in digit order in shared memory and written out in that order, so every
// digit's run reaches global memory as contiguous, coalesced stores.
// LOW: only the low 32 bits under `mask` are written.
// 31 M keys, 7-bit digits: 0.25 ms a pass with the loads inside the rounds and __match_any_sync,
// 0.23 with the loads first, 0.17 with ballots (copying the keys takes 0.07).
template <bool LOW>
__global__ void __launch_bounds__(kSortWarps * 32) k_radix_scatter(const uint64_t* in, void* out,
                                                                  int64_t n, int shift, int digits,
                                                                  uint32_t mask,
                                                                  const int64_t* offs,
                                                                  int64_t tiles) {
  __shared__ uint64_t sk[kSortTile];
  __shared__ uint32_t wcnt[kSortWarps][kRadix];
  __shared__ uint32_t dstart[kRadix];
  __shared__ uint32_t wsum[kSortWarps];
  __shared__ int64_t gbase[kRadix];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int d = tid; d < digits; d += blockDim.x) gbase[d] = offs[(int64_t)d * tiles + blockIdx.x];
  for (int i = tid; i < kSortWarps * kRadix; i += blockDim.x) (&wcnt[0][0])[i] = 0;
  __syncthreads();
  const int64_t tile0 = (int64_t)blockIdx.x * kSortTile;
  const int tn = (int)min((int64_t)kSortTile, n - tile0);
  const int64_t base = tile0 + warp * (32 * kSortItems);
  uint64_t k[kSortItems];
  uint32_t rk[kSortItems];
#pragma unroll
  for (int t = 0; t < kSortItems; ++t) {  // every load in flight before the first is ranked
    const int64_t i = base + t * 32 + lane;
    k[t] = i < n ? in[i] : 0ull;
  }
#pragma unroll
  for (int t = 0; t < kSortItems; ++t) {
    const bool valid = base + t * 32 + lane < n;
    const int d = valid ? (int)((k[t] >> shift) & (digits - 1)) : kRadix;
    unsigned peers = __ballot_sync(kFull, valid);
    if (!valid) peers = ~peers;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if ((1 << q) >= digits) break;
      const unsigned set = __ballot_sync(kFull, (d >> q) & 1);
      peers &= (d >> q) & 1 ? set : ~set;
    }
    const uint32_t before = valid ? wcnt[warp][d] : 0u;
    rk[t] = before + __popc(peers & lanemask_lt());
    __syncwarp();
    if (valid && lane == __ffs(peers) - 1) wcnt[warp][d] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // per digit: exclusive prefix over the warps, then the tile-local start of each digit
  uint32_t tot = 0;
  if (tid < kRadix) {
    for (int w = 0; w < kSortWarps; ++w) {
      const uint32_t c = wcnt[w][tid];
      wcnt[w][tid] = tot;
      tot += c;
    }
  }
  uint32_t incl = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (tid < kRadix) {
    uint32_t off = 0;
    for (int w = 0; w < warp; ++w) off += wsum[w];
    dstart[tid] = off + incl - tot;
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < kSortItems; ++t) {
    const int64_t i = base + t * 32 + lane;
    if (i < n) {
      const int d = (int)((k[t] >> shift) & (digits - 1));
      sk[dstart[d] + wcnt[warp][d] + rk[t]] = k[t];
    }
  }
  __syncthreads();
  for (int i = tid; i < tn; i += blockDim.x) {
    const uint64_t key = sk[i];
    const int d = (int)((key >> shift) & (digits - 1));
    const int64_t at = gbase[d] + (i - (int)dstart[d]);
    if (LOW) ((uint32_t*)out)[at] = (uint32_t)key & mask;
    else ((uint64_t*)out)[at] = key;
  }
}

}  // namespace

cudaError_t scan_excl(const int64_t* in, int64_t* out, int64_t n, int64_t* total, cudaStream_t s) {
  return scan_impl<int64_t>(in, out, n, total, s);
}
cudaError_t scan_excl(const int32_t* in, int64_t* out, int64_t n, int64_t* total, cudaStream_t s) {
  return scan_impl<int32_t>(in, out, n, total, s);
}
cudaError_t scan_excl(const uint8_t* in, int64_t* out, int64_t n, int64_t* total, cudaStream_t s) {
  return scan_impl<uint8_t>(in, out, n, total, s);
}

cudaError_t radix_sort_u64(uint64_t* keys, uint64_t* tmp, int64_t n, int bits, cudaStream_t st,
                           int shift0, int32_t* low, uint32_t mask) {
  if (n <= 0) return cudaSuccess;
  // passes of nearly equal digits: fewer bins, so longer runs and fewer counts to scan.  One
  // pass at least where only the low bits are wanted.
  const int passes = bits > 0 ? (bits + 7) / 8 : (low ? 1 : 0);
  const int per = passes ? (bits + passes - 1) / passes : 0;
  int64_t tiles = (n + kSortTile - 1) / kSortTile;
  int64_t* counts = nullptr;
  cudaError_t e = cudaMallocAsync(&counts, sizeof(int64_t) * (int64_t(1) << per) * tiles, st);
  if (e != cudaSuccess) return e;
  uint64_t *a = keys, *b = tmp;
  for (int p = 0; p < passes && e == cudaSuccess; ++p) {
    const int shift = shift0 + p * per, digits = 1 << std::min(per, bits - p * per);
    k_radix_hist<<<(unsigned)tiles, kSortWarps * 32, 0, st>>>(a, n, shift, digits, counts, tiles);
    e = scan_impl<int64_t>(counts, counts, digits * tiles, nullptr, st);
    if (e != cudaSuccess) break;
    if (low && p == passes - 1)
      k_radix_scatter<true><<<(unsigned)tiles, kSortWarps * 32, 0, st>>>(a, low, n, shift, digits,
                                                                         mask, counts, tiles);
    else
      k_radix_scatter<false><<<(unsigned)tiles, kSortWarps * 32, 0, st>>>(a, b, n, shift, digits,
                                                                          0u, counts, tiles);
    e = cudaGetLastError();
    std::swap(a, b);
  }
  if (e == cudaSuccess && !low && a != keys)
    e = cudaMemcpyAsync(keys, a, sizeof(uint64_t) * n, cudaMemcpyDeviceToDevice, st);
  cudaFreeAsync(counts, st);
  return e;
}

}  // namespace xgm
