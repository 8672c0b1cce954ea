// Generation-order prefix evaluation (segmentation_prefixes) for many images.
//
// The reference draws masks one launch at a time and scores each step with a
// single CTA (prefix_kernel.cu:142-199: 2N+1 launches per image). Here every
// batch is five launches, whatever the number of images or masks:
//   1. prefix_pass   one read of the target map and of every mask byte. Each
//                    lane tracks the visible owner of its 16 pixels (the last
//                    mask drawn over them) and, at every requested checkpoint,
//                    emits the owner transitions since the previous checkpoint
//                    into per-checkpoint delta histograms [Q][G][N+1]. The same
//                    pass counts target areas and the raw mask x slot
//                    intersections used by instance matching.
//   2. prefix_scan   running sums over checkpoints turn deltas into the canvas
//                    pair histograms (column 0 starts with the target areas).
//   3. prefix_rows   one CTA per (image, checkpoint): canvas PQ / confusion with
//                    active labels (segments with visible pixels), shared with
//                    the panoptic evaluator's scoring code; beside them one CTA
//                    or more per image: greedy generation-order matching
//                    (prefix.py:106-118), a chain per (threshold, class), its
//                    counts, precision and recall at the checkpoints.
//   4. pe_compute    per-checkpoint PQ/SQ/RQ/IoU summaries.
#include "pe_common.cuh"
#include "pe_fields.h"
#include "pe_score.cuh"
#include "pe_bins.cuh"

namespace pe {
namespace {

constexpr int kPxThreads = 256;
constexpr int kPxChunk = kPxThreads * 16;
constexpr int kPxWindow = 4;  // masks whose 16-byte words each lane loads before processing them

__device__ __forceinline__ const int64_t* pdesc(const int64_t* descs, int64_t b) { return descs + b * kPrefixFields; }

__device__ __forceinline__ int64_t find_image(const int64_t* descs, int64_t B, int field, int64_t value) {
  int64_t lo = 0, hi = B - 1;
  while (lo < hi) {
    const int64_t mid = (lo + hi + 1) >> 1;
    if (descs[mid * kPrefixFields + field] <= value) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Visible owner (1-based mask index, 0 = none) of one lane's 16 pixels, now and at the previous
// checkpoint: one byte per pixel when every image of the batch has at most 255 masks (kBytes), else
// 16 bits per pixel. Drawing a mask is a byte (or half-word) select per register, so its cost does not
// depend on how many of the 16 pixels it covers. Pixels outside the image or on an invalid slot are
// drawn too and skipped when transitions are emitted.
template <bool kBytes>
struct Owners {
  static constexpr int kWords = kBytes ? 4 : 8;
  u32 now[kWords], prev[kWords];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int k = 0; k < kWords; ++k) now[k] = prev[k] = 0;
  }
  // lsb: the lane's 16 mask bytes reduced to 0/1; covered pixels take owner `value`.
  __device__ __forceinline__ void draw(const u32 (&lsb)[4], u32 value) {
    if constexpr (kBytes) {
      const u32 fill = value * 0x01010101u;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const u32 m = lsb[k] * 0xffu;  // 0x00 / 0xff per byte (no carries: bytes are 0 or 1)
        now[k] = (now[k] & ~m) | (fill & m);
      }
    } else {
      const u32 fill = value * 0x00010001u;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const u32 lo = __byte_perm(lsb[k], 0u, 0x4140) * 0xffffu, hi = __byte_perm(lsb[k], 0u, 0x4342) * 0xffffu;
        now[2 * k] = (now[2 * k] & ~lo) | (fill & lo);
        now[2 * k + 1] = (now[2 * k + 1] & ~hi) | (fill & hi);
      }
    }
  }
  __device__ __forceinline__ static int at(const u32 (&v)[kWords], int j) {
    if constexpr (kBytes) return (int)((v[j >> 2] >> (8 * (j & 3))) & 0xffu);
    else return (int)((v[j >> 1] >> (16 * (j & 1))) & 0xffffu);
  }
  __device__ __forceinline__ bool changed() const {
    u32 d = 0;
#pragma unroll
    for (int k = 0; k < kWords; ++k) d |= now[k] ^ prev[k];
    return d != 0;
  }
};

// Draw mask i (its 16 bytes for this lane in w) over the lane's pixels: the raw mask x slot
// intersections raw_row[slot] and the new owners. Called by every lane of the warp.
template <bool kBytes>
__device__ __forceinline__ void draw_mask(int i, uint4 w, const int (&t)[16], const LaneSlots& ls, u32* raw_row,
                                          Owners<kBytes>& s) {
  const u32 lsb[4] = {w.x & 0x01010101u, w.y & 0x01010101u, w.z & 0x01010101u, w.w & 0x01010101u};
  const auto pack4 = [](u32 v) { return (v * 0x01020408u) >> 24; };
  const u32 m = pack4(lsb[0]) | pack4(lsb[1]) << 4 | pack4(lsb[2]) << 8 | pack4(lsb[3]) << 12;
  add_slots(t, ls, m & ls.valid(), raw_row);
  s.draw(lsb, (u32)(i + 1));
}

// At a requested checkpoint: the owner transitions of the lane's valid pixels since the previous
// checkpoint into that checkpoint's delta histogram dq [G][N + 1] (run-combined), then the owners
// become the previous ones. Called by every lane when any lane of the warp changed.
// Bytes of four words that differ from the byte before them (byte j against byte j - 1 across the words;
// byte 0 against `before`), as 16 bits.
__device__ __forceinline__ u32 byte_changes(const u32 (&v)[4]) {
  u32 bits = 0, carry = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    u32 x = v[k] ^ ((v[k] << 8) | carry);
    carry = v[k] >> 24;
    x |= x >> 4;
    x |= x >> 2;
    x |= x >> 1;
    bits |= (((x & 0x01010101u) * 0x01020408u) >> 24) << (4 * k);
  }
  return bits;
}

// Bytes where two sets of four words differ, as 16 bits.
__device__ __forceinline__ u32 byte_differs(const u32 (&a)[4], const u32 (&b)[4]) {
  u32 bits = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    u32 x = a[k] ^ b[k];
    x |= x >> 4;
    x |= x >> 2;
    x |= x >> 1;
    bits |= (((x & 0x01010101u) * 0x01020408u) >> 24) << (4 * k);
  }
  return bits;
}

// Byte j of four words (j uniform or not: three selects, no local memory).
__device__ __forceinline__ int byte_at(const u32 (&v)[4], int j) {
  const int k = j >> 2;
  const u32 w = k == 0 ? v[0] : (k == 1 ? v[1] : (k == 2 ? v[2] : v[3]));
  return (int)((w >> (8 * (j & 3))) & 0xffu);
}

// The lanes' first runs of equal (slot, old owner, new owner): summed over the lanes of the warp that share
// one when many have a run (inside a large region every lane has the same transition), else lane by lane.
__device__ __forceinline__ void add_first_run(int g, int o, int n, int count, int* dq, int N) {
  if (__popc(__ballot_sync(0xffffffffu, count != 0)) >= kGroupLanes) {
    // Owners are below 65536 (N < 65535), so (slot, old, new) packs into 64 bits.
    const unsigned long long key =
        count ? ((unsigned long long)(u32)g << 32) | ((unsigned long long)o << 16) | (unsigned long long)n : ~0ull;
    const u32 peers = __match_any_sync(0xffffffffu, key);
    const int total = (int)__reduce_add_sync(peers, (u32)count);
    if ((threadIdx.x & 31) != (int)(__ffs(peers) - 1)) count = 0;
    else if (count) count = total;
  }
  if (count) {
    atomicAdd(dq + (int64_t)g * (N + 1) + o, -count);
    atomicAdd(dq + (int64_t)g * (N + 1) + n, count);
  }
}

// Slot changes between neighbouring pixels of a lane (bit j: pixel j's slot differs from pixel j - 1's).
__device__ __forceinline__ u32 slot_changes(const int (&t)[16]) {
  u32 bits = 1u;
#pragma unroll
  for (int j = 1; j < 16; ++j) bits |= (u32)(t[j] != t[j - 1]) << j;
  return bits;
}

// Byte-owner transitions of a lane, run by run rather than pixel by pixel: the changed valid pixels
// (cv) split into runs wherever the slot (gchg, fixed for the chunk), the old owner or the new owner
// changes from one pixel to the next; a lane usually has one to three runs. The first run is summed
// over the warp's lanes that share it, later runs go to memory directly.
__device__ __forceinline__ void emit_transitions_bytes(const int (&t)[16], const LaneSlots& ls, int* dq, int N,
                                                       Owners<true>& s) {
  const u32 cv = byte_differs(s.now, s.prev) & ls.valid();
  const u32 kchg = slot_changes(t) | byte_changes(s.now) | byte_changes(s.prev) | 1u;
  u32 starts = cv & (~(cv << 1) | kchg);
  int fg = -1, fo = 0, fn = 0, fcnt = 0;
  while (starts) {
    const int j = __ffs(starts) - 1;
    starts &= starts - 1;
    const int end = starts ? __ffs(starts) - 1 : 16;
    const int cnt = __popc(cv & ((end == 16 ? 0xffffu : (1u << end) - 1u) & ~((1u << j) - 1u)));
    int g;
    if ((ls.e1 >> j) & 1u) {
      g = ls.s1;
    } else if ((ls.e2 >> j) & 1u) {
      g = ls.s2;
    } else if ((ls.e0 >> j) & 1u) {
      g = 0;
    } else {  // another slot inside the lane: rare
      g = t[0];
#pragma unroll
      for (int k = 1; k < 16; ++k) g = k == j ? t[k] : g;
    }
    const int o = byte_at(s.prev, j), n = byte_at(s.now, j);
    if (fcnt == 0) {
      fg = g; fo = o; fn = n; fcnt = cnt;
    } else {
      atomicAdd(dq + (int64_t)g * (N + 1) + o, -cnt);
      atomicAdd(dq + (int64_t)g * (N + 1) + n, cnt);
    }
  }
  add_first_run(fg, fo, fn, fcnt, dq, N);
#pragma unroll
  for (int k = 0; k < 4; ++k) s.prev[k] = s.now[k];
}

// Later runs, at region borders, go to memory directly.
template <bool kBytes>
__device__ __forceinline__ void emit_transitions(const int (&t)[16], u32 valid, int* dq, int N, Owners<kBytes>& s) {
  int rg = -1, ro = -1, rn = -1, cnt = 0;
  int fg = -1, fo = 0, fn = 0, fcnt = 0;  // the lane's first run
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const int o = Owners<kBytes>::at(s.prev, j), n = Owners<kBytes>::at(s.now, j);
    if (!((valid >> j) & 1u) || o == n) continue;
    const int g = t[j];
    if (g == rg && o == ro && n == rn) {
      ++cnt;
    } else {
      if (cnt) {
        if (fcnt == 0) {
          fg = rg; fo = ro; fn = rn; fcnt = cnt;
        } else {
          atomicAdd(dq + (int64_t)rg * (N + 1) + ro, -cnt);
          atomicAdd(dq + (int64_t)rg * (N + 1) + rn, cnt);
        }
      }
      rg = g; ro = o; rn = n; cnt = 1;
    }
  }
  if (cnt) {
    if (fcnt == 0) {
      fg = rg; fo = ro; fn = rn; fcnt = cnt;
    } else {
      atomicAdd(dq + (int64_t)rg * (N + 1) + ro, -cnt);
      atomicAdd(dq + (int64_t)rg * (N + 1) + rn, cnt);
    }
  }
  add_first_run(fg, fo, fn, fcnt, dq, N);
#pragma unroll
  for (int k = 0; k < Owners<kBytes>::kWords; ++k) s.prev[k] = s.now[k];
}

// Transitions at a checkpoint: the run form for byte owners, the pixel loop for 16-bit owners.
template <bool kBytes>
__device__ __forceinline__ void emit_at_checkpoint(const int (&t)[16], const LaneSlots& ls, int* dq, int N,
                                                   Owners<kBytes>& s) {
  if constexpr (kBytes) emit_transitions_bytes(t, ls, dq, N, s);
  else emit_transitions<false>(t, ls.valid(), dq, N, s);
}

// One CTA per 4096-pixel chunk, masks read with plain loads (rows at any alignment).
template <bool kBytes>
__global__ void __launch_bounds__(kPxThreads, 2)
prefix_pass_kernel(const int64_t* __restrict__ descs, int64_t B, const int* __restrict__ step_q, u32* __restrict__ ga,
                   u32* __restrict__ raw, int* __restrict__ delta, int* __restrict__ error) {
  wait_for_earlier_kernels();
  const int64_t b = find_image(descs, B, kPrefixChunkBegin, blockIdx.x);
  const int64_t* d = pdesc(descs, b);
  const int64_t pixels = d[kPrefixPixels];
  const int64_t x = (blockIdx.x - d[kPrefixChunkBegin]) * (int64_t)kPxChunk + (int64_t)threadIdx.x * 16;
  const int N = (int)d[kPrefixN], G = (int)d[kPrefixG];
  const int* target = reinterpret_cast<const int*>(d[kPrefixTarget]);
  const uint8_t* masks = reinterpret_cast<const uint8_t*>(d[kPrefixMasks]);
  const int64_t stride = d[kPrefixStride];
  const bool vec_map = d[kPrefixFlags] & 1, vec_masks = d[kPrefixFlags] & 2;
  const int* steps = step_q + d[kPrefixStepBegin];
  int* delta_img = delta + d[kPrefixPairBegin];
  u32* raw_img = raw + d[kPrefixRawBegin];
  const int64_t plane = (int64_t)G * (N + 1);
  const int lane = threadIdx.x & 31;

  int t[16];
  load16_maps(target, x, pixels, vec_map, t);
  bool bad = false;
  const LaneSlots ls = lane_slots(t, x, pixels, G, bad);
  add_slots<true>(t, ls, ls.valid(), ga + d[kPrefixSlotBegin]);
  Owners<kBytes> s;
  s.clear();
  const int64_t xm = x < pixels ? x : pixels;
  uint4 window[kPxWindow];
  for (int i = 0; i < N; ++i) {
    if (i % kPxWindow == 0) {  // the next kPxWindow masks' words are all in flight before any is used
#pragma unroll
      for (int k = 0; k < kPxWindow; ++k)
        window[k] = i + k < N ? load16_mask(masks + (int64_t)(i + k) * stride, xm, pixels, vec_masks)
                              : make_uint4(0, 0, 0, 0);
    }
    uint4 w = window[0];
#pragma unroll
    for (int k = 1; k < kPxWindow; ++k)
      if (i % kPxWindow == k) w = window[k];
    if (__any_sync(0xffffffffu, (w.x | w.y | w.z | w.w) != 0))
      draw_mask<kBytes>(i, w, t, ls, raw_img + (int64_t)i * G, s);
    const int q = steps[i + 1];  // uniform across the CTA
    if (q >= 0 && __any_sync(0xffffffffu, s.changed()))
      emit_at_checkpoint<kBytes>(t, ls, delta_img + q * plane, N, s);
  }
  if (bad) atomicOr(error, 1);
}

// Persistent form: a producer warp streams every mask's segment of the current 4096-pixel chunk into a
// shared-memory ring with cp.async.bulk (one copy per mask row and chunk: the 16-byte-aligned words
// covering the segment, since rows may start at any byte; completion on the stage's mbarrier) while
// 8 consumer warps draw the masks in order from shared memory. What bounds them is instructions: most
// masks leave most warps' 512 pixels alone, so a stage of four masks costs a warp four loads, one
// warp-wide OR of "has a pixel here" and a barrier, and only masks with a pixel (a superset: the staged
// words as they lie) are re-aligned and drawn; checkpoints are a bit mask read 32 masks at a time, and
// only warps drawn to since the last one look for transitions. 16 images of 845 x 845 with 64 masks:
// 151 us (308 with a test, a step lookup and two loads per mask and one reduction per lane and slot for
// the target areas: those met on the bins of void and of large segments), 45 for one of 256 x 384 (69). Each
// wait is bounded; a timeout sets bit 30 of *error, the producer waits (bounded) for its copies in
// flight, and every role returns.
constexpr int kPbConsumers = kPxThreads;
constexpr int kPbThreads = kPbConsumers + 32;
constexpr int kPbStage = 4;  // mask rows per ring stage
constexpr int kPbRing = 6;   // stages in flight per CTA
constexpr long long kPbWaitLimit = 4000000000ll;  // about two seconds of SM clock
constexpr int kPbTimeoutBit = 1 << 30;

constexpr int kPbSlot = kPxChunk + 16;  // staged bytes per mask row and chunk (aligned words covering it)

constexpr int kPbChunkRing = 4;  // published chunks in flight per CTA

struct PrefixShared {
  unsigned char ring[kPbRing][kPbStage][kPbSlot];
  int64_t x0[kPbChunkRing];     // first pixel of the chunk published to the consumers
  int64_t image[kPbChunkRing];  // its image; -1 ends the CTA's work
  uint64_t full[kPbRing];
  uint64_t empty[kPbRing];
  uint64_t chunk_full[kPbChunkRing];
  uint64_t chunk_empty[kPbChunkRing];
  int abort;
};

template <bool kBytes>
__global__ void __launch_bounds__(kPbThreads, 2)
prefix_pass_bulk_kernel(const int64_t* __restrict__ descs, int64_t B, int64_t total_chunks,
                        unsigned long long* __restrict__ schedule, const int* __restrict__ step_q,
                        u32* __restrict__ ga, u32* __restrict__ raw, int* __restrict__ delta,
                        int* __restrict__ error) {
  wait_for_earlier_kernels();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PrefixShared& sm = *reinterpret_cast<PrefixShared*>(smem_raw);
  // Without a counter: contiguous chunk ranges whose sizes differ by at most one chunk.
  const int64_t c_begin = (int64_t)blockIdx.x * total_chunks / gridDim.x;
  const int64_t c_end = (int64_t)(blockIdx.x + 1) * total_chunks / gridDim.x;
  if (!schedule && c_begin >= c_end) return;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kPbRing; ++i) {
      mbar_init(&sm.full[i], 1);
      mbar_init(&sm.empty[i], kPbConsumers / 32);
    }
    for (int i = 0; i < kPbChunkRing; ++i) {
      mbar_init(&sm.chunk_full[i], 1);
      mbar_init(&sm.chunk_empty[i], kPbConsumers / 32);
    }
    sm.abort = 0;
    mbar_fence_init();
  }
  __syncthreads();
  volatile int* abort = &sm.abort;

  if (threadIdx.x >= kPbConsumers) {
    // ---- producer ----------------------------------------------------------
    if (threadIdx.x != kPbConsumers) return;
    int64_t seq = 0, published = 0, next = c_begin;
    bool ok = true;
    // Publish a chunk to the consumers (image -1: no more work); false when the wait for a free entry fails.
    auto publish = [&](int64_t image, int64_t x0) {
      const int e = (int)(published % kPbChunkRing);
      const int64_t use = published / kPbChunkRing;
      if ((use > 0 && !mbar_wait(&sm.chunk_empty[e], (uint32_t)((use - 1) & 1), kPbWaitLimit)) || *abort)
        return false;
      sm.x0[e] = x0;
      sm.image[e] = image;
      mbar_arrive(&sm.chunk_full[e]);  // release: the entry is visible to consumers that see the phase
      ++published;
      return true;
    };
    while (ok) {
      const int64_t chunk = schedule ? (int64_t)atomicAdd(schedule, 1ull) : (next < c_end ? next++ : total_chunks);
      if (chunk >= total_chunks) break;
      const int64_t image = find_image(descs, B, kPrefixChunkBegin, chunk);
      const int64_t* d = pdesc(descs, image);
      const int64_t pixels = d[kPrefixPixels];
      const int64_t x0 = (chunk - d[kPrefixChunkBegin]) * (int64_t)kPxChunk;
      if (!publish(image, x0)) {
        ok = false;
        break;
      }
      const int64_t len = min((int64_t)kPxChunk, pixels - x0);
      const int N = (int)d[kPrefixN];
      const uint8_t* masks = reinterpret_cast<const uint8_t*>(d[kPrefixMasks]);
      const int64_t stride = d[kPrefixStride];
      const int* target = reinterpret_cast<const int*>(d[kPrefixTarget]);
      const uint32_t map_bytes = (uint32_t)((len * 4) & ~15ll);
      if ((d[kPrefixFlags] & 1) && map_bytes) bulk_prefetch_l2(target + x0, map_bytes);
      for (int r0 = 0; r0 < N; r0 += kPbStage) {
        const int slot = (int)(seq % kPbRing);
        const int64_t use = seq / kPbRing;
        if ((use > 0 && !mbar_wait(&sm.empty[slot], (uint32_t)((use - 1) & 1), kPbWaitLimit)) || *abort) {
          ok = false;
          break;
        }
        const int n = min(kPbStage, N - r0);
        uint32_t sizes[kPbStage], total = 0;
#pragma unroll
        for (int k = 0; k < kPbStage; ++k) {
          // Aligned words from the one holding pixel x0 to the one holding the segment's last byte.
          const int o = (int)(reinterpret_cast<uintptr_t>(masks + (int64_t)(r0 + k) * stride) & 15);
          sizes[k] = k < n ? (uint32_t)round_up(len + o, 16) : 0u;
          total += sizes[k];
        }
        mbar_arrive_expect_tx(&sm.full[slot], total);
        for (int k = 0; k < n; ++k) {
          const uint8_t* row = masks + (int64_t)(r0 + k) * stride;
          const int o = (int)(reinterpret_cast<uintptr_t>(row) & 15);
          bulk_copy_g2s(sm.ring[slot][k], row + x0 - o, sizes[k], &sm.full[slot]);
        }
        ++seq;
      }
    }
    if (ok) ok = publish(-1, 0);
    if (!ok) {
      *abort = 1;
      atomicOr(error, kPbTimeoutBit);
    }
    for (int64_t q = seq > kPbRing ? seq - kPbRing : 0; q < seq; ++q)  // copies still in flight land first
      mbar_wait(&sm.full[q % kPbRing], (uint32_t)((q / kPbRing) & 1), kPbWaitLimit);
    return;
  }

  // ---- consumers -----------------------------------------------------------
  const int lane = threadIdx.x & 31;
  int64_t seq = 0, taken = 0;
  bool ok = true, bad = false;
  while (ok) {
    const int e = (int)(taken % kPbChunkRing);
    const bool ready = mbar_wait(&sm.chunk_full[e], (uint32_t)((taken / kPbChunkRing) & 1), kPbWaitLimit);
    if (!__all_sync(0xffffffffu, ready && !*abort)) {
      ok = false;
      break;
    }
    const int64_t image = sm.image[e], x0 = sm.x0[e];
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.chunk_empty[e]);
    ++taken;
    if (image < 0) break;
    const int64_t* d = pdesc(descs, image);
    const int64_t pixels = d[kPrefixPixels];
    const int64_t x = x0 + (int64_t)threadIdx.x * 16;
    const int N = (int)d[kPrefixN], G = (int)d[kPrefixG];
    const int* steps = step_q + d[kPrefixStepBegin];
    const int64_t plane = (int64_t)G * (N + 1);
    const int64_t stride = d[kPrefixStride];
    // Row r of the chunk starts (first + r * stride) mod 16 bytes into its first staged word.
    const uint32_t first = (uint32_t)d[kPrefixMasks] & 15u, o_step = (uint32_t)stride & 15u;
    int* delta_img = delta + d[kPrefixPairBegin];
    u32* raw_img = raw + d[kPrefixRawBegin];
    int t[16];
    load16_maps(reinterpret_cast<const int*>(d[kPrefixTarget]), x, pixels, d[kPrefixFlags] & 1, t);
    // Pixels past the image end are not valid: stale staged bytes under them are ignored.
    const LaneSlots ls = lane_slots(t, x, pixels, G, bad);
    add_slots<true>(t, ls, ls.valid(), ga + d[kPrefixSlotBegin]);
    Owners<kBytes> s;
    s.clear();
    u32 checks = 0;      // bit k: a checkpoint follows mask 32 (r0 / 32) + k
    bool drawn = false;  // since the last checkpoint, anywhere in the warp
    for (int r0 = 0; r0 < N; r0 += kPbStage) {
      if ((r0 & 31) == 0) checks = __ballot_sync(0xffffffffu, r0 + lane < N && steps[r0 + 1 + lane] >= 0);
      const int slot = (int)(seq % kPbRing);
      const bool got = mbar_wait(&sm.full[slot], (uint32_t)((seq / kPbRing) & 1), kPbWaitLimit);
      if (!__all_sync(0xffffffffu, got && !*abort)) {  // warp-uniform decision
        ok = false;
        break;
      }
      const uint4* words = reinterpret_cast<const uint4*>(&sm.ring[slot][0][threadIdx.x * 16]);
      u32 hit = 0;
#pragma unroll
      for (int k = 0; k < kPbStage; ++k) {
        const uint4 a = words[k * (kPbSlot / 16)];
        u32 any = a.x | a.y | a.z | a.w;
        if (lane == 31 && ((first + (r0 + k) * o_step) & 15u)) {  // the warp's pixels end in the next word
          const uint4 b = words[k * (kPbSlot / 16) + 1];
          any |= b.x | b.y | b.z | b.w;
        }
        hit |= (u32)(any != 0) << k;
      }
      const u32 present = (1u << min(kPbStage, N - r0)) - 1u;
      hit = __reduce_or_sync(0xffffffffu, hit) & present;
      const u32 check = (checks >> (r0 & 31)) & present;
      // One mask at a time, not unrolled: the drawing code is large and unrolled copies of it missed the
      // instruction cache.
#pragma unroll 1
      for (u32 todo = hit | check; todo; todo &= todo - 1) {
        const int k = __ffs(todo) - 1, i = r0 + k;
        if ((hit >> k) & 1u) {
          const int o = (int)((first + i * o_step) & 15u);
          const uint4 a = words[k * (kPbSlot / 16)];
          draw_mask<kBytes>(i, o ? realign16(a, words[k * (kPbSlot / 16) + 1], o) : a, t, ls,
                            raw_img + (int64_t)i * G, s);
          drawn = true;
        }
        if (drawn && ((check >> k) & 1u)) {
          drawn = false;
          if (__any_sync(0xffffffffu, s.changed()))
            emit_at_checkpoint<kBytes>(t, ls, delta_img + (int64_t)steps[i + 1] * plane, N, s);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.empty[slot]);
      ++seq;
    }
  }
  if (!ok) {
    *abort = 1;
    if (lane == 0) atomicOr(error, kPbTimeoutBit);
  }
  if (bad) atomicOr(error, 1);
}

// Running sums over checkpoints: delta[q] -> pairs[q] in place.
__global__ void prefix_scan_kernel(const int64_t* __restrict__ descs, const u32* __restrict__ ga,
                                   int* __restrict__ delta) {
  wait_for_earlier_kernels();
  const int64_t* d = pdesc(descs, blockIdx.y);
  const int N = (int)d[kPrefixN], G = (int)d[kPrefixG], Q = (int)d[kPrefixQ];
  const int64_t plane = (int64_t)G * (N + 1);
  const int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= plane) return;
  int* base = delta + d[kPrefixPairBegin] + cell;
  const int g = (int)(cell / (N + 1)), j = (int)(cell % (N + 1));
  int v = j == 0 ? (int)ga[d[kPrefixSlotBegin] + g] : 0;
  for (int q = 0; q < Q; ++q) {
    v += base[(int64_t)q * plane];
    base[(int64_t)q * plane] = v;
  }
}

__host__ __device__ inline size_t label_bytes(int64_t P) { return ((size_t)P * sizeof(int) + 15) & ~size_t{15}; }

// Canvas PQ of one (image, checkpoint) row, scored in one pass (pe_score.cuh). smem: dynamic shared memory of
// the launch (labels, then tables and entry list); rows whose tables do not fit it are scored in place.
__device__ __forceinline__ void score_row(const int64_t* descs, int64_t B, int64_t row, const int* pairs,
                                          const int* classes, const int* gc, const uint8_t* crowd, int C, int64_t* tp,
                                          int64_t* fp, int64_t* fn, double* sums, int64_t* confusion,
                                          unsigned char* smem_raw, int smem) {
  const int64_t b = find_image(descs, B, kPrefixQBegin, row);
  const int64_t* d = pdesc(descs, b);
  const int N = (int)d[kPrefixN], G = (int)d[kPrefixG], P = N + 1;
  const int q = (int)(row - d[kPrefixQBegin]);
  const u32* pq = reinterpret_cast<const u32*>(pairs + d[kPrefixPairBegin] + (int64_t)q * G * P);
  gc += d[kPrefixSlotBegin];
  crowd += d[kPrefixSlotBegin];
  classes += d[kPrefixDetBegin];
  ScoreOut out{reinterpret_cast<u64*>(tp + row * C), reinterpret_cast<u64*>(fp + row * C),
               reinterpret_cast<u64*>(fn + row * C), sums + row * C,
               reinterpret_cast<u64*>(confusion + row * C * (int64_t)(C + 1))};
  int* labels = reinterpret_cast<int*>(smem_raw);
  const size_t tables_at = label_bytes(P);
  // Active labels: a mask's class while it has visible pixels (prefix.py:82).
  if (tables_at + ScoreTables::base_bytes(G, P, C) <= (size_t)smem) {
    const ScoreTables t = ScoreTables::at(smem_raw + tables_at, G, P, C, smem - tables_at);
    score_totals(pq, t, gc, crowd, G, P, C);
    for (int p = threadIdx.x; p < P; p += blockDim.x) labels[p] = (p > 0 && t.col[p] > 0) ? classes[p - 1] : -1;
    __syncthreads();
    score_matches<u32, false>(pq, t, labels, G, P, C, out);
    return;
  }
  u64* areas = reinterpret_cast<u64*>(smem_raw + tables_at);
  int* matched = reinterpret_cast<int*>(areas + G + P);
  unsigned char* staging = reinterpret_cast<unsigned char*>(matched + G);
  staging += (16 - reinterpret_cast<uintptr_t>(staging) % 16) % 16;
  score_areas<u32, false>(pq, gc, labels, crowd, areas, G, P, C, false);
  __syncthreads();
  for (int p = threadIdx.x; p < P; p += blockDim.x) labels[p] = (p > 0 && areas[G + p] > 0) ? classes[p - 1] : -1;
  __syncthreads();
  score_accumulate<u32, false>(pq, gc, labels, crowd, areas, matched, G, P, C, out, staging);
}

// Greedy generation-order matching (prefix.py:106-118) and the validation of an image's metadata. Only masks and
// targets of one class meet, so every (IoU threshold, class) is a chain of its own: the masks of the class in
// generation order, each taking the free target of the largest IoU (the first slot on ties), the counts written at
// every checkpoint. `splits` CTAs share an image's classes. A CTA groups its classes' slots and masks, takes the
// IoU of every pair once into shared memory (where `smem` has room for them) and then walks one chain per thread.
// Error bits: 2 empty prediction mask, 4 bad target class / slot 0 not void, 8 target areas vs metadata, 16 bad
// prediction class.
//
// The chains are latency: one warp per threshold walking all masks of an image took 40.8 us for 16 images of 64
// masks, 101 slots and 133 classes on 16 SMs, and 6.0 us more for the ratios in a launch of their own.
constexpr int kSerialSlots = 8;      // a thread alone walks chains of up to 8 slots a class ...
constexpr int kSerialPairs = 128;    // ... or 128 pairs in all (a warp step costs about as much as 8 slots)
constexpr int kMatchClasses = 16;    // classes per CTA, at least, while an image's classes are shared

__host__ __device__ inline size_t prefix_match_bytes(int64_t N, int64_t G, int64_t T, int64_t C) {
  const int64_t ints = 3 * N + 1 + 2 * G + 4 * C + 3 + T * ((G + 31) / 32);
  return sizeof(u64) * N + sizeof(int) * ints + G + 16;
}

struct PrefixMatch {
  const int64_t* descs;
  const u32* ga;
  const u32* raw;
  const int* classes;
  const int* gc;
  const uint8_t* crowd;
  const uint8_t* isthing;
  const double* thresholds;
  int T, C;
  const int* step_q;
  int64_t *itp, *ifp, *ifn;
  double *precision, *recall;
  int validate;
  int* error;
};

__device__ __forceinline__ int warp_exclusive_sum(int v, int lane, int* total) {
  int sum = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, sum, off);
    if (lane >= off) sum += u;
  }
  *total = __shfl_sync(0xffffffffu, sum, 31);
  return sum - v;
}

__device__ __forceinline__ void match_classes(const PrefixMatch& a, int64_t image, int split, int splits,
                                              unsigned char* smem_raw, int smem) {
  const int64_t* d = pdesc(a.descs, image);
  const int N = (int)d[kPrefixN], G = (int)d[kPrefixG], T = a.T, C = a.C;
  const int64_t first_row = d[kPrefixQBegin];
  const int* steps = a.step_q + d[kPrefixStepBegin];
  const u32* ga = a.ga + d[kPrefixSlotBegin];
  const int* gc = a.gc + d[kPrefixSlotBegin];
  const uint8_t* crowd = a.crowd + d[kPrefixSlotBegin];
  const int* classes = a.classes + d[kPrefixDetBegin];
  const u32* raw = a.raw + d[kPrefixRawBegin];
  const int per = (C + splits - 1) / splits;
  const int c0 = min(C, split * per), nc = min(C, c0 + per) - c0;  // this CTA's classes: c0 and the nc - 1 after it
  const int words = (G + 31) / 32;

  u64* areas = reinterpret_cast<u64*>(smem_raw);             // N: mask areas on valid slots
  u32* checks = reinterpret_cast<u32*>(areas + N);           // N + 1: checkpoints by prefix, prefix << 16 | row
  int* mask_class = reinterpret_cast<int*>(checks + N + 1);  // N: the mask's class here if a thing, else -1
  int* by_mask = mask_class + N;                             // N: masks by class, in generation order
  int* slot_class = by_mask + N;                             // G
  int* by_slot = slot_class + G;                             // G: slots by class, in slot order
  int* slot_start = by_slot + G;                             // nc + 1
  int* mask_start = slot_start + nc + 1;                     // nc + 1
  int* pair_start = mask_start + nc + 1;                     // nc + 1
  int* positives = pair_start + nc + 1;                      // nc
  u32* used = reinterpret_cast<u32*>(positives + nc);        // T x words: targets taken, by position in by_slot
  uint8_t* crowd_s = reinterpret_cast<uint8_t*>(used + T * words);
  const size_t at = (prefix_match_bytes(N, G, T, C) + 7) & ~size_t{7};
  long long* ious = reinterpret_cast<long long*>(smem_raw + at);  // IoU bit patterns: per class, mask major
  const int room = (size_t)smem > at ? (int)(((size_t)smem - at) / sizeof(long long)) : 0;
  __shared__ int s_err, s_checks;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = (int)(blockDim.x >> 5);

  if (tid == 0) s_err = 0;
  for (int k = tid; k <= nc; k += blockDim.x) slot_start[k] = mask_start[k] = 0;
  for (int k = tid; k < nc; k += blockDim.x) positives[k] = 0;
  for (int k = tid; k < T * words; k += blockDim.x) used[k] = 0;
  __syncthreads();
  int err = 0;
  for (int g = tid; g < G; g += blockDim.x) {
    const int c = gc[g];
    const bool ignored = crowd[g];
    const bool here = c >= c0 && c < c0 + nc && a.isthing[c];
    crowd_s[g] = ignored;
    slot_class[g] = here ? c - c0 : -1;
    if (here) {
      atomicAdd(slot_start + c - c0, 1);
      if (!ignored) atomicAdd(positives + c - c0, 1);
    }
    if (a.validate && split == 0) {
      if (c < -1 || c >= C || (g == 0 && (c != -1 || ignored))) err |= 4;
      if (g > 0 && ((ga[g] > 0) != (c >= 0))) err |= 8;
    }
  }
  for (int i = tid; i < N; i += blockDim.x) {
    const int c = classes[i];
    const bool here = c >= c0 && c < c0 + nc && a.isthing[c];
    mask_class[i] = here ? c - c0 : -1;
    if (here) atomicAdd(mask_start + c - c0, 1);
    if (a.validate && split == 0 && (c < 0 || c >= C)) err |= 16;
  }
  __syncthreads();
  if (warp == 0) {
    // Starts of every class's slots, masks and pairs.
    int slots = 0, masks = 0, pairs = 0;
    for (int base = 0; base < nc; base += 32) {
      const int k = base + lane;
      const int s = k < nc ? slot_start[k] : 0, m = k < nc ? mask_start[k] : 0;
      int total_s, total_m, total_p;
      const int ss = warp_exclusive_sum(s, lane, &total_s), ms = warp_exclusive_sum(m, lane, &total_m);
      const int ps = warp_exclusive_sum(s * m, lane, &total_p);
      if (k < nc) {
        slot_start[k] = slots + ss;
        mask_start[k] = masks + ms;
        pair_start[k] = pairs + ps;
      }
      slots += total_s, masks += total_m, pairs += total_p;
    }
    if (lane == 0) slot_start[nc] = slots, mask_start[nc] = masks, pair_start[nc] = pairs;
  } else if (warp == 1) {
    int n = 0;
    for (int base = 0; base <= N; base += 32) {
      const int k = base + lane, q = k <= N ? steps[k] : -1;
      const u32 some = __ballot_sync(0xffffffffu, q >= 0);
      if (q >= 0) checks[n + __popc(some & ((1u << lane) - 1u))] = (u32)k << 16 | (u32)q;
      n += __popc(some);
    }
    if (lane == 0) s_checks = n;
  }
  // Areas of the masks matched here, and, when they are checked, of this CTA's share of all masks.
  for (int i = warp; i < N; i += warps) {
    const bool checked = a.validate && i % splits == split;
    if (mask_class[i] < 0 && !checked) continue;
    u64 area = 0;
    for (int g = lane; g < G; g += 32) area += raw[(int64_t)i * G + g];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) area += __shfl_xor_sync(0xffffffffu, area, off);
    if (lane == 0) {
      areas[i] = area;
      if (checked && area == 0) err |= 2;
    }
  }
  if (err) atomicOr(&s_err, err);
  __syncthreads();
  // Slots and masks grouped by class, in their own order within it; then the class's IoUs: inter / union, crowd
  // slots against the mask's area. A warp packs its class's pairs into full FP64 operations.
  const bool staged = pair_start[nc] <= room;
  auto iou_of = [&](int i, int g) -> long long {
    const u64 inter = raw[(int64_t)i * G + g];
    const u64 uni = crowd_s[g] ? areas[i] : areas[i] + ga[g] - inter;
    return inter ? __double_as_longlong((double)inter / (double)(uni > 1 ? uni : 1)) : 0;
  };
  for (int c = warp; c < nc; c += warps) {
    const int s0 = slot_start[c], ns = slot_start[c + 1] - s0, m0 = mask_start[c], nm = mask_start[c + 1] - m0;
    if (ns == 0 && nm == 0) continue;
    auto place = [&](const int* of, int n, int* out) {
      for (int base = 0; base < n; base += 32) {
        const int k = base + lane;
        const u32 mine = __ballot_sync(0xffffffffu, k < n && of[k] == c);
        if ((mine >> lane) & 1u) out[__popc(mine & ((1u << lane) - 1u))] = k;
        out += __popc(mine);
      }
    };
    place(slot_class, G, by_slot + s0);
    place(mask_class, N, by_mask + m0);
    __syncwarp();
    for (int k = lane; staged && k < ns * nm; k += 32)
      ious[pair_start[c] + k] = iou_of(by_mask[m0 + k / ns], by_slot[s0 + k % ns]);
  }
  __syncthreads();
  // Chains: item t * nc + c. A warp takes 32 of them, a lane each, then together those of many slots.
  const int checkpoints = s_checks;
  const int items = T * nc;  // the shared memory for it bounds T and C
  for (int base = warp * 32; base < items; base += warps * 32) {
    const int item = base + lane;
    const int t = item < items ? item / nc : 0, c = item < items ? item % nc : 0;
    const int slots = slot_start[c + 1] - slot_start[c], masks = mask_start[c + 1] - mask_start[c];
    const bool alone = item < items && (slots <= kSerialSlots || (slots <= 32 && slots * masks <= kSerialPairs));
    auto write = [&](int t_, int c_, u32 check, int tp, int fp) {
      const int64_t o = ((first_row + (check & 0xffffu)) * T + t_) * C + c0 + c_;
      const int n = positives[c_];
      a.itp[o] = tp;
      a.ifp[o] = fp;
      a.ifn[o] = n - tp;
      // tp / max(tp + fp, 1) and tp / max(positives, 1) (prefix.py:106-118)
      a.precision[o] = tp ? (double)tp / (double)(tp + fp) : 0.0;
      a.recall[o] = tp ? (double)tp / (double)(n > 1 ? n : 1) : 0.0;
    };
    if (alone) {
      const long long thr = __double_as_longlong(a.thresholds[t]);
      const int s0 = slot_start[c], m0 = mask_start[c];
      const long long* iou_c = ious + pair_start[c];
      int tp = 0, fp = 0, m = 0;
      u32 taken = 0;
      for (int e = 0; e < checkpoints; ++e) {
        const u32 check = checks[e];
        for (; m < masks && by_mask[m0 + m] < (int)(check >> 16); ++m) {
          long long best = -1;
          int best_k = -1;
          bool ignored = false;
          for (int k = 0; k < slots; ++k) {
            const int g = by_slot[s0 + k];
            const long long iou = staged ? iou_c[m * slots + k] : iou_of(by_mask[m0 + m], g);
            if (iou < thr) continue;
            if (crowd_s[g]) {
              ignored = true;
            } else if (!((taken >> k) & 1u) && iou > best) {
              best = iou;
              best_k = k;
            }
          }
          if (best_k >= 0) {
            taken |= 1u << best_k;
            ++tp;
          } else if (!ignored) {
            ++fp;
          }
        }
        write(t, c, check, tp, fp);
      }
    }
    for (u32 rest = __ballot_sync(0xffffffffu, item < items && !alone); rest; rest &= rest - 1) {
      const int together = base + __ffs(rest) - 1;
      const int tt = together / nc, cc = together % nc;
      const long long thr = __double_as_longlong(a.thresholds[tt]);
      const int s0 = slot_start[cc], ns = slot_start[cc + 1] - s0, m0 = mask_start[cc];
      const int nm = mask_start[cc + 1] - m0;
      const long long* iou_c = ious + pair_start[cc];
      u32* taken = used + tt * words;
      int tp = 0, fp = 0, m = 0;
      for (int e = 0; e < checkpoints; ++e) {
        const u32 check = checks[e];
        for (; m < nm && by_mask[m0 + m] < (int)(check >> 16); ++m) {
          long long best = -1;
          int best_k = INT_MAX;
          bool ignored = false;
          for (int k = lane; k < ns; k += 32) {
            const int g = by_slot[s0 + k];
            const long long iou = staged ? iou_c[m * ns + k] : iou_of(by_mask[m0 + m], g);
            if (iou < thr) continue;
            if (crowd_s[g]) {
              ignored = true;
            } else if (!((taken[(s0 + k) >> 5] >> ((s0 + k) & 31)) & 1u) && iou > best) {
              best = iou;  // a lane scans increasing k: strictly greater keeps the first slot
              best_k = k;
            }
          }
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) {
            const long long other = __shfl_xor_sync(0xffffffffu, best, off);
            const int other_k = __shfl_xor_sync(0xffffffffu, best_k, off);
            if (other > best || (other == best && other_k < best_k)) best = other, best_k = other_k;
          }
          if (best_k != INT_MAX) {
            // Classes of another warp share words at their ends.
            if (lane == 0) atomicOr(taken + ((s0 + best_k) >> 5), 1u << ((s0 + best_k) & 31));
            ++tp;
          } else if (!__any_sync(0xffffffffu, ignored)) {
            ++fp;
          }
          __syncwarp();
        }
        if (lane == 0) write(tt, cc, check, tp, fp);
      }
    }
  }
  if (tid == 0 && s_err) atomicOr(a.error, s_err);
}

// Both roles in one launch: matching first (`match_blocks` CTAs, the longer ones), then a CTA per checkpoint row.
// Neither reads what the other writes.
constexpr int kPrefixScoreThreads = 512;
__global__ void __launch_bounds__(kPrefixScoreThreads)
prefix_rows_kernel(PrefixMatch match, int splits, int match_blocks, int64_t B, const int* __restrict__ pairs,
                   int64_t* __restrict__ tp, int64_t* __restrict__ fp, int64_t* __restrict__ fn,
                   double* __restrict__ sums, int64_t* __restrict__ confusion, int smem) {
  wait_for_earlier_kernels();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int block = blockIdx.x, C = match.C;
  // Unchecked calls never read the word: where the pass gave up, their FP64 results are NaN.
  const int stopped = match.validate ? 0 : __ldcg(match.error) & kStoppedBits;
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  if (block < match_blocks) {
    match_classes(match, block / splits, block % splits, splits, smem_raw, smem);
    if (!stopped) return;
    __syncthreads();
    const int64_t* d = pdesc(match.descs, block / splits);
    const int per = (C + splits - 1) / splits, c0 = min(C, block % splits * per), nc = min(C, c0 + per) - c0;
    const int64_t first = d[kPrefixQBegin] * match.T, n = d[kPrefixQ] * match.T * nc;
    for (int64_t k = threadIdx.x; k < n; k += blockDim.x) {
      const int64_t o = (first + k / nc) * C + c0 + k % nc;
      match.precision[o] = match.recall[o] = nan;
    }
    return;
  }
  const int64_t row = block - match_blocks;
  score_row(match.descs, B, row, pairs, match.classes, match.gc, match.crowd, C, tp, fp, fn, sums, confusion, smem_raw,
            smem);
  if (!stopped) return;
  __syncthreads();
  for (int c = threadIdx.x; c < C; c += blockDim.x) sums[row * C + c] = nan;
}

}  // namespace
}  // namespace pe

using namespace pe;

PE_API int pe_prefix_desc_fields(void) { return kPrefixFields; }

// Batched segmentation_prefixes (prefix.py:12-122; replaces the `prefix` op,
// prefix_kernel.cu:142-199, for any number of images). Inputs: descriptor
// table (pe_prefix_desc_fields() int64 per image), step table (per image N+1
// ints: checkpoint index of prefix k or -1), classes (sum N int32), gc and
// crowd (sum G), isthing [C], thresholds [T] f64. Workspace (zeroed here):
// ga (sum G u32), raw (sum N*G u32), pairs (sum Q*G*(N+1) int32), counters
// (B*T*C*2 int32). Outputs per checkpoint row (R = sum Q), zeroed here where
// accumulated: tp/fp/fn int64 [R,C], sums f64 [R,C], confusion int64
// [R,C,C+1], itp/ifp/ifn int64 [R,T,C], precision/recall f64 [R,T,C]; then
// per_class [R,4,C], summaries [R,3,3], counts [R,3], miou [R] (pe_compute).
// Validation bits in *error: 1 unknown target slot, 2 empty prediction mask,
// 4 bad target class, 8 target areas vs metadata, 16 bad prediction class. Without validation, where the pass gave
// up (bits from 2^20), sums, precision and recall are NaN, and with them pq, sq and miou.
PE_API int pe_prefix(const int64_t* descs, int64_t B, int64_t total_chunks, int64_t total_rows, int64_t max_g,
                     int64_t max_p, int64_t max_cells, const int32_t* step_q, const int32_t* classes,
                     const int32_t* gc, const uint8_t* crowd, const uint8_t* isthing, const double* thresholds,
                     int64_t T, int64_t C, uint32_t* ga, int64_t ga_len, uint32_t* raw, int64_t raw_len,
                     int32_t* pairs, int64_t pairs_len, int32_t* counters, int64_t counters_len, int64_t* tp,
                     int64_t* fp, int64_t* fn, double* sums, int64_t* confusion, int64_t* itp, int64_t* ifp,
                     int64_t* ifn, double* precision, double* recall, double* per_class, double* summaries,
                     int64_t* counts, double* miou, int validate, int bulk, uint64_t* schedule, int32_t* error,
                     cudaStream_t stream) {
  PE_REQUIRE(B >= 0 && total_rows >= 0 && C > 0 && C < INT_MAX && T > 0 && T <= 1024 && max_g >= 0 &&
                 max_p >= 1 && max_p < 65536,
             "invalid prefix batch (T must be 1..1024, masks per image < 65535)");
  if (B == 0) return zero_spans({{error, 4}}, stream);
  const int64_t rows = 8 * total_rows * C;
  const int zeroed = zero_spans({{ga, 4 * ga_len}, {raw, 4 * raw_len}, {pairs, 4 * pairs_len},
                                 {counters, 4 * counters_len}, {error, 4}, {tp, rows}, {fp, rows}, {fn, rows},
                                 {sums, rows}, {confusion, rows * (C + 1)}, {schedule, schedule ? 8 : 0}},
                                stream);
  if (zeroed != kOk) return zeroed;
  if (total_chunks) {
    if (bulk) {
      const int64_t grid = std::min(total_chunks, (int64_t)sm_count() * 2);  // two CTAs per SM
      const size_t smem = sizeof(PrefixShared);
      // Owners fit in a byte per pixel when no image has more than 255 masks.
      auto kernel = max_p <= 256 ? prefix_pass_bulk_kernel<true> : prefix_pass_bulk_kernel<false>;
      PE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      launch_kernel(kernel, (unsigned)grid, kPbThreads, smem, stream, descs, B, total_chunks,
          reinterpret_cast<unsigned long long*>(schedule), step_q, ga, raw, pairs, error);
    } else {
      auto kernel = max_p <= 256 ? prefix_pass_kernel<true> : prefix_pass_kernel<false>;
      launch_kernel(kernel, (unsigned)total_chunks, kPxThreads, 0, stream, descs, B, step_q, ga, raw, pairs, error);
    }
    PE_LAUNCHED("prefix_pass");
    count_launch();
  }
  if (max_cells > 0) {
    launch_kernel(prefix_scan_kernel, dim3((unsigned)ceil_div(max_cells, 256), (unsigned)B), 256, 0, stream, descs, ga,
        pairs);
    PE_LAUNCHED("prefix_scan");
    count_launch();
  }
  {
    const size_t in_place = label_bytes(max_p) + sizeof(u64) * (max_g + max_p) + sizeof(int) * max_g +
                            score_staging_bytes(max_p) + 32;
    PE_REQUIRE(!total_rows || in_place <= 200 * 1024, "prefix histogram too large for scoring (G=%lld, N+1=%lld)",
               (long long)max_g, (long long)max_p);
    const size_t state = prefix_match_bytes(max_p - 1, max_g, T, C) + 8;
    PE_REQUIRE(state <= 201 * 1024, "prefix matching state too large (G=%lld, T=%lld, C=%lld)", (long long)max_g,
               (long long)T, (long long)C);
    // Two CTAs per SM, where the tables of a row and the IoUs of a CTA's classes have use for less.
    const size_t row = label_bytes(max_p) + score_bytes(max_g, max_p, C, max_g * max_p);
    const size_t ious = state + sizeof(long long) * (max_p - 1) * max_g;
    const size_t want = std::min<size_t>(std::max(row, ious), 110 * 1024);
    const size_t smem = std::max({want, state, total_rows ? in_place : 0});
    if (smem > 48 * 1024)
      PE_CUDA(cudaFuncSetAttribute(prefix_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // An image's classes on as many CTAs as there are SMs for the batch.
    const int64_t splits = std::max<int64_t>(1, std::min<int64_t>(ceil_div(C, kMatchClasses), sm_count() / B));
    const PrefixMatch match{descs, ga, raw, classes, gc, crowd, isthing, thresholds, (int)T, (int)C, step_q, itp, ifp,
                            ifn, precision, recall, validate, error};
    launch_kernel(prefix_rows_kernel, (unsigned)(B * splits + total_rows), kPrefixScoreThreads, smem, stream, match,
        (int)splits, (int)(B * splits), B, pairs, tp, fp, fn, sums, confusion, (int)smem);
    PE_LAUNCHED("prefix_rows");
    count_launch();
  }
  if (total_rows) {
    const int status = pe_compute(tp, fp, fn, sums, confusion, isthing, total_rows, C, per_class, summaries, counts,
                                  miou, nullptr, nullptr, nullptr, nullptr, nullptr, stream);
    if (status != kOk) return status;
  }
  if (validate) {
    int code = 0;
    PE_CUDA(cudaMemcpyAsync(&code, error, sizeof(int), cudaMemcpyDeviceToHost, stream));
    PE_CUDA(cudaStreamSynchronize(stream));
    return code;
  }
  return kOk;
}
