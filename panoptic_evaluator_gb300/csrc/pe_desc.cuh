// Per-image descriptor table shared by the batched kernels: kDescFields int64
// values per image, built on the host (panoptic_evaluator_gb300/_batch.py).
#pragma once

#include "pe_common.cuh"
#include "pe_fields.h"

namespace pe {

__device__ __forceinline__ const int64_t* desc_of(const int64_t* descs, int64_t b) { return descs + b * kDescFields; }

// Image owning chunk `chunk` (binary search over kChunkBegin).
__device__ __forceinline__ int64_t image_of_chunk(const int64_t* descs, int64_t B, int64_t chunk) {
  int64_t lo = 0, hi = B - 1;
  while (lo < hi) {
    const int64_t mid = (lo + hi + 1) >> 1;
    if (descs[mid * kDescFields + kChunkBegin] <= chunk) lo = mid; else hi = mid - 1;
  }
  return lo;
}

}  // namespace pe
