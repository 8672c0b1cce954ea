// What the two ways to count mask intersections share: the choice between them, made on the device.
#pragma once
#include "pe_common.cuh"

namespace pe {

constexpr int kSampleParts = 8;  // CTAs that sample one image

// The sample's estimate of the time that streaming would take (sample_image in pe_pairs.cu: picoseconds, a few entries
// per image) and the limit up to which it is the faster way. Both kernels read it, so exactly one of them does the work.
struct Choice {
  const u64* costs;  // null: the contraction runs whatever the masks hold
  int64_t entries, limit;
};

// Whole-block call at a kernel's start: does the batch stay below the limit?
__device__ __forceinline__ bool streams(const Choice& choice) {
  if (!choice.costs) return false;
  __shared__ u64 total;
  if (threadIdx.x < 32) {
    u64 sum = 0;
    for (int64_t i = threadIdx.x; i < choice.entries; i += 32) sum += choice.costs[i];
    for (int k = 16; k; k >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, k);
    if (threadIdx.x == 0) total = sum;
  }
  __syncthreads();
  return (int64_t)total <= choice.limit;
}

// The contraction's launch, outputs zeroed before (pe_contract.cu).
int launch_contract(const int64_t* descs, const int64_t* blocks, int64_t n_blocks, int64_t total_chunks,
                    const int64_t* cta_bounds, int64_t ctas, const int64_t* order, uint32_t* inter, uint64_t* pa,
                    uint64_t* ga, const void* maps, Choice choice, int32_t* error, cudaStream_t stream);

}  // namespace pe
