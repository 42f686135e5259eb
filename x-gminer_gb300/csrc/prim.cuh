// Device-wide scan and radix sort (prim.cu).
#pragma once
#include "common.cuh"

namespace xgm {

// Exclusive prefix sum into int64 (in and out may alias).  `total` (device, optional)
// receives the sum of all n inputs.
cudaError_t scan_excl(const int64_t* in, int64_t* out, int64_t n, int64_t* total, cudaStream_t s);
cudaError_t scan_excl(const int32_t* in, int64_t* out, int64_t n, int64_t* total, cudaStream_t s);
cudaError_t scan_excl(const uint8_t* in, int64_t* out, int64_t n, int64_t* total, cudaStream_t s);

// Stable LSD radix sort of keys[0..n) over bits [shift0, shift0 + bits), at most 8 bits
// per pass; tmp must hold n keys.  The result is left in keys; or, when `low` is given,
// only its low 32 bits under `mask` are written, to low[0..n), by the last pass (keys and
// tmp are then scratch).
cudaError_t radix_sort_u64(uint64_t* keys, uint64_t* tmp, int64_t n, int bits, cudaStream_t s,
                           int shift0 = 0, int32_t* low = nullptr, uint32_t mask = 0);

}  // namespace xgm
