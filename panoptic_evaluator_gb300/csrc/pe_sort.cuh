// Block-wide sorting of (score, index) records by falling score, equal scores by index.
#pragma once

#include "pe_common.cuh"

namespace pe {

// Sort key of a score: an unsigned integer that orders like the score descending (-0.0 taken as 0.0, so
// equal scores give equal keys; NaN last, as the reference's argsort puts it), compared with integers
// instead of FP64 (GB300's FP64 pipe runs at 1/64 of the FP32 rate). Ties sort by record index, which
// makes the sort stable.
__device__ __forceinline__ u64 score_key(double score) {
  if (score != score) return ~0ull;
  u64 b = (u64)__double_as_longlong(score == 0.0 ? 0.0 : score);
  b = (b >> 63) ? ~b : (b | 0x8000000000000000ull);  // ascending in the score
  return ~b;                                           // descending
}

__device__ __forceinline__ bool before_in_order(u64 ka, int ia, u64 kb, int ib) {
  return ka < kb || (ka == kb && ia < ib);
}

// Bitonic sort of n (key, index) pairs, n padded to a power of two with
// sentinels that sort last. `global` arrays need a fence before each barrier.
template <bool kGlobal>
__device__ void bitonic_sort(u64* key, int* idx, int n, int padded) {
  for (int i = n + threadIdx.x; i < padded; i += blockDim.x) {
    key[i] = ~0ull;
    idx[i] = INT_MAX;
  }
  __syncthreads();
  for (int size = 2; size <= padded; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < padded; i += blockDim.x) {
        const int j = i ^ stride;
        if (j > i) {
          const bool ascending = (i & size) == 0;
          const u64 ki = key[i], kj = key[j];
          const int ii = idx[i], ij = idx[j];
          const bool swap = ascending ? before_in_order(kj, ij, ki, ii) : before_in_order(ki, ii, kj, ij);
          if (swap) { key[i] = kj; key[j] = ki; idx[i] = ij; idx[j] = ii; }
        }
      }
      if constexpr (kGlobal) __threadfence_block();
      __syncthreads();
    }
  }
}

// Up to kEach records per thread: each record's place is the number of records before it, one pass over
// the others instead of a barrier per stage of the network (100 records: 1 pass, against 28 barriers).
// idx is left in order, the keys as they were. Synchronises the block.
template <int kEach = 1>
__device__ __forceinline__ void rank_sort(const u64* key, int* idx, int n) {
  int place[kEach], mine[kEach];
  u64 own[kEach];
#pragma unroll
  for (int e = 0; e < kEach; ++e) {
    const int i = threadIdx.x + e * blockDim.x;
    own[e] = i < n ? key[i] : 0;
    mine[e] = i < n ? idx[i] : 0;
    place[e] = 0;
  }
  if ((int)threadIdx.x < n) {
#pragma unroll 4
    for (int j = 0; j < n; ++j) {
      const u64 k = key[j];
      const int i = idx[j];
#pragma unroll
      for (int e = 0; e < kEach; ++e) place[e] += before_in_order(k, i, own[e], mine[e]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < kEach; ++e)
    if ((int)(threadIdx.x + e * blockDim.x) < n) idx[place[e]] = mine[e];
  __syncthreads();
}

}  // namespace pe
