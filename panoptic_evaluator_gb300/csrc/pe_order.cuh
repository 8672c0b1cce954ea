// What an update does to each image's metadata first: the given fields into flat arrays, and the score order of its
// detections. One block per image; the kernels that call these do both for one launch where they can.
#pragma once

#include "pe_desc.cuh"
#include "pe_sort.cuh"

namespace pe {

// Per-image metadata of an instance update gathered into flat arrays at each image's detection / slot
// offsets (one launch instead of a host-side concatenation per field). fields: one row of
// kGatherFields int64 per image: device pointers of its prediction classes, scores, target classes,
// crowd flags and annotation areas (0: absent), then element sizes (bit 0: prediction classes int64,
// bit 1: scores float64, bit 2: target classes int64, bit 4: areas float64; else int32 / float32).
constexpr int kGatherFields = 6;
struct FieldGather {
  const int64_t* fields;
  int* pc;
  double* scores;
  int* gc;
  uint8_t* crowd;
  double* areas;
};

__device__ __forceinline__ void gather_image(const int64_t* d, int64_t image, const FieldGather& a) {
  const int64_t* f = a.fields + image * kGatherFields;
  const int D = (int)d[kD], G = (int)d[kG];
  const int64_t db = d[kDetBegin], sb = d[kSlotBegin], bits = f[5];
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    a.pc[db + i] = (bits & 1) ? (int)reinterpret_cast<const int64_t*>(f[0])[i] : reinterpret_cast<const int*>(f[0])[i];
    a.scores[db + i] = (bits & 2) ? reinterpret_cast<const double*>(f[1])[i]
                                  : (double)reinterpret_cast<const float*>(f[1])[i];
  }
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    a.gc[sb + g] = (bits & 4) ? (int)reinterpret_cast<const int64_t*>(f[2])[g] : reinterpret_cast<const int*>(f[2])[g];
    a.crowd[sb + g] = f[3] ? reinterpret_cast<const uint8_t*>(f[3])[g] : 0;
    if (a.areas && f[4])
      a.areas[sb + g] = (bits & 16) ? reinterpret_cast<const double*>(f[4])[g]
                                    : (double)reinterpret_cast<const float*>(f[4])[g];
  }
}

// The image's classes for the matching, after gather_image and a block barrier: those of its targets, and of its
// detections, of which one outside [0, C) marks class 0. class_bits: ceil(C / 32) words per image.
__device__ __forceinline__ void mark_classes(const int64_t* d, int64_t image, const FieldGather& a, int C,
                                             u32* class_bits) {
  const int D = (int)d[kD], G = (int)d[kG], words = (C + 31) / 32;
  u32* bits = class_bits + image * words;
  for (int w = threadIdx.x; w < words; w += blockDim.x) bits[w] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    const int c = a.pc[d[kDetBegin] + i], k = c >= 0 && c < C ? c : 0;
    atomicOr(bits + (k >> 5), 1u << (k & 31));
  }
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    const int c = a.gc[d[kSlotBegin] + g];
    if (c >= 0 && c < C) atomicOr(bits + (c >> 5), 1u << (c & 31));
  }
}

// Per-image stable descending score order (NaN scores last). Latency bounds it: 32 images of 100
// detections took 10.6 us, 8 of 256 15.8, with a bitonic network over FP64 keys; 4.5 and 8.5 now.
constexpr int kSortThreads = 256;
constexpr int kOrderCap = 4096;  // detections of an image sorted in shared memory, at most
struct ScoreOrder {
  const double* scores;
  const int* classes;
  int64_t* order;
  double* sorted_scores;
  int* sorted_classes;
  u64* ws_key;  // two entries per detection of the batch
  int* ws_idx;
  int cap;      // entries of the launch's shared memory, a power of two
};

inline size_t sort_bytes(int cap) { return (sizeof(u64) + sizeof(int)) * (size_t)cap; }

inline ScoreOrder score_order(const double* scores, const int* classes, int64_t detections, int64_t* order,
                              double* sorted_scores, int* sorted_classes, void* workspace) {
  int cap = 32;
  while (cap < kOrderCap && cap < detections) cap <<= 1;
  u64* key = static_cast<u64*>(workspace);
  return ScoreOrder{scores, classes, order, sorted_scores, sorted_classes, key,
                    reinterpret_cast<int*>(key + 2 * round_up(detections + 1, 64)), cap};
}

__device__ __forceinline__ void sort_image(const int64_t* d, const ScoreOrder& a, unsigned char* smem_raw) {
  const int D = (int)d[kD];
  const int64_t base = d[kDetBegin];
  if (D == 0) return;
  int padded = 1;
  while (padded < D) padded <<= 1;
  const bool in_smem = padded <= a.cap;
  u64* key = in_smem ? reinterpret_cast<u64*>(smem_raw) : a.ws_key + 2 * base;
  int* idx = in_smem ? reinterpret_cast<int*>(smem_raw + sizeof(u64) * a.cap) : a.ws_idx + 2 * base;
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    key[i] = score_key(a.scores[base + i]);
    idx[i] = i;
  }
  __syncthreads();
  if (D <= (int)blockDim.x) rank_sort(key, idx, D);
  else if (in_smem) bitonic_sort<false>(key, idx, D, padded);
  else bitonic_sort<true>(key, idx, D, padded);
  for (int r = threadIdx.x; r < D; r += blockDim.x) {
    const int i = idx[r];
    a.order[base + r] = i;
    a.sorted_scores[base + r] = a.scores[base + i];
    a.sorted_classes[base + r] = a.classes[base + i];
  }
}

}  // namespace pe
