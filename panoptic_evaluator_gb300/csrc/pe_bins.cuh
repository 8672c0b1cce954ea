// Per-lane pixel loads and (mask, slot) binning shared by the fused passes.
#pragma once

#include "pe_common.cuh"

namespace pe {

// Sixteen neighbouring map pixels; pixels past `end` read as -1. Images of odd pixel counts start anywhere
// on the 16-byte grid: their pixels come out of the five aligned words that hold them (p + x has the same
// offset for every lane), since sixteen single loads per lane touch each line sixteen times.
__device__ __forceinline__ void load16_maps(const int* __restrict__ p, int64_t x, int64_t end, bool vec, int v[16]) {
  if (!vec && x + 16 <= end) {
    const int shift = (int)((reinterpret_cast<uintptr_t>(p + x) >> 2) & 3);
    const int4* q = reinterpret_cast<const int4*>(p + x - shift);
    int w[20];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const int4 u = k < 4 || shift ? __ldg(q + k) : make_int4(0, 0, 0, 0);
      w[4 * k] = u.x; w[4 * k + 1] = u.y; w[4 * k + 2] = u.z; w[4 * k + 3] = u.w;
    }
    const bool s2 = shift & 2, s1 = shift & 1;
#pragma unroll
    for (int k = 0; k < 18; ++k) w[k] = s2 ? w[k + 2] : w[k];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = s1 ? w[k + 1] : w[k];
    return;
  }
  if (vec && x + 16 <= end) {
    const int4* q = reinterpret_cast<const int4*>(p + x);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int4 w = __ldg(q + k);
      v[4 * k] = w.x; v[4 * k + 1] = w.y; v[4 * k + 2] = w.z; v[4 * k + 3] = w.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = x + j < end ? __ldg(p + x + j) : -1;
  }
}

__device__ __forceinline__ uint4 load16_mask(const uint8_t* __restrict__ p, int64_t x, int64_t end, bool vec) {
  if (vec && x + 16 <= end) return __ldg(reinterpret_cast<const uint4*>(p + x));
  uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
  for (int j = 0; j < 16; ++j)
    if (x + j < end) w[j >> 2] |= (uint32_t)(__ldg(p + x + j) != 0) << (8 * (j & 3));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Streaming (evict-first) 16-byte load of 16 mask bytes; bytes past `end` read as 0.
__device__ __forceinline__ uint4 load16_stream(const uint8_t* __restrict__ p, int64_t x, int64_t end, bool vec) {
  if (vec && x + 16 <= end) return __ldcs(reinterpret_cast<const uint4*>(p + x));
  return load16_mask(p, x, end, vec);
}

// Counts go straight to global memory with reductions whose result is unused
// (fire-and-forget), so no lane waits on a shared-memory table. What they must
// not do is meet: a few bins of an image (void, its large segments) take a count
// from nearly every lane, and reductions on one address are served one after
// another. Lanes of a warp that add to the same bin are therefore summed first
// wherever many of them can. (Fused pass of 64 uneven images 359 -> 309 us, of 8
// images with 256 detections 231 -> 205; prefix pass of 16 images 231 -> 151, and
// 382 with no grouping at all.)
constexpr u32 kEmpty = 0xffffffffu;
constexpr int kGroupLanes = 16;  // lanes with a count from which they are grouped by bin (8: 2 % slower, 3: 6 %)

// Adds `count` of each lane to row[bin]: one reduction per distinct bin of the warp when at least
// kGroupLanes lanes have a count (kGrouped: always), else one per lane. Called by every lane.
template <bool kGrouped = false>
__device__ __forceinline__ void add_lanes(u32* row, u32 bin, u32 count) {
  if (kGrouped || __popc(__ballot_sync(0xffffffffu, count != 0)) >= kGroupLanes) {
    const u32 peers = __match_any_sync(0xffffffffu, count ? bin : kEmpty);
    const u32 sum = __reduce_add_sync(peers, count);
    if ((threadIdx.x & 31) != (u32)(__ffs(peers) - 1)) count = 0;
    else if (count) count = sum;
  }
  if (count) atomicAdd(row + bin, count);
}

// The same for a bin common to the warp.
__device__ __forceinline__ void add_common(u32* bin, u32 count) {
  const u32 sum = __reduce_add_sync(0xffffffffu, count);
  if ((threadIdx.x & 31) == 0 && sum) atomicAdd(bin, sum);
}

// Per-lane view of its 16 target slots, fixed for every mask of a step: pixel
// bit masks of "on the first pixel's slot", "on the last's (if different)", "on
// void (if neither is)" and "on any other valid slot". Invalid slots and pixels
// past the image are in none; an invalid slot inside the image sets `bad`.
struct LaneSlots {
  u32 e1, e2, e0, emid;
  int s1, s2;
  __device__ __forceinline__ u32 valid() const { return e1 | e2 | e0 | emid; }
};

__device__ __forceinline__ u32 inside_bits(int64_t x, int64_t pixels) {
  return x + 16 <= pixels ? 0xffffu : (x < pixels ? (1u << (pixels - x)) - 1u : 0u);
}

__device__ __forceinline__ LaneSlots lane_slots(const int (&t)[16], int64_t x, int64_t pixels, int G, bool& bad) {
  LaneSlots ls;
  ls.s1 = t[0];
  ls.s2 = t[15];
  const u32 inside = inside_bits(x, pixels);
  u32 ok = 0, e1 = 0, e2 = 0, e0 = 0;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    ok |= (u32)((u32)t[j] < (u32)G) << j;
    e1 |= (u32)(t[j] == ls.s1) << j;
    e2 |= (u32)(t[j] == ls.s2) << j;
    e0 |= (u32)(t[j] == 0) << j;
  }
  bad |= (inside & ~ok) != 0;
  ok &= inside;
  ls.e1 = e1 & ok;
  ls.e2 = e2 & ok & ~e1;
  ls.e0 = e0 & ok & ~e1 & ~e2;
  ls.emid = ok & ~(e1 | e2 | e0);
  return ls;
}

// Adds the pixels m of each lane to row[slot]. Called by every lane of the warp.
template <bool kGrouped = false>
__device__ __forceinline__ void add_slots(const int (&t)[16], const LaneSlots& ls, u32 m, u32* row) {
  add_lanes<kGrouped>(row, (u32)ls.s1, __popc(m & ls.e1));
  add_lanes<kGrouped>(row, (u32)ls.s2, __popc(m & ls.e2));
  add_common(row, __popc(m & ls.e0));
  const u32 mid = m & ls.emid;  // another slot inside 16 pixels: rare
  if (mid) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if ((mid >> j) & 1u) atomicAdd(row + t[j], 1u);
  }
}

// Adds each lane's 16 (target, prediction) pairs to pairs[t * P + p]: those equal to the first pixel's
// pair, to the last's, void on void, and the others one by one. Called by every lane of the warp.
__device__ __forceinline__ void add_pairs(const int (&t)[16], const int (&p)[16], int64_t x, int64_t pixels, int G,
                                          int P, u32* pairs, bool& bad) {
  const u32 inside = inside_bits(x, pixels);
  u32 key[16], ok = 0;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const bool in = (u32)t[j] < (u32)G && (u32)p[j] < (u32)P && ((inside >> j) & 1u);
    ok |= (u32)in << j;
    key[j] = in ? (u32)(t[j] * P + p[j]) : kEmpty;
  }
  bad |= (inside & ~ok) != 0;
  const u32 first = key[0], last = key[15];
  u32 n_first = 0, n_last = 0, n_void = 0;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const bool in = key[j] != kEmpty, a = key[j] == first, b = key[j] == last, v = key[j] == 0;
    n_first += in && a;
    n_last += in && !a && b;
    n_void += in && !a && !b && v;
    if (in && !a && !b && !v) atomicAdd(pairs + key[j], 1u);
  }
  add_lanes<true>(pairs, first, n_first);
  add_lanes(pairs, last, n_last);
  add_common(pairs, n_void);
}

// 16 bytes of 0/1 -> 16 bits, byte j -> bit j.
__device__ __forceinline__ u32 pack16(uint4 w) {
  const auto pack4 = [](u32 v) { return ((v & 0x01010101u) * 0x01020408u) >> 24; };
  return pack4(w.x) | pack4(w.y) << 4 | pack4(w.z) << 8 | pack4(w.w) << 12;
}

}  // namespace pe
