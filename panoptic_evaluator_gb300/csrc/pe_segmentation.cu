// Batched segmentation evaluation over a device table of image descriptors.
//
// Images may differ in size and in segment / detection counts. One update of
// SegmentationEvaluator (combined PQ + mIoU + mask AP with a shared target) is
//   1. seg_sort       per image, stable descending score order of detections;
//                     sorted scores/classes are written straight into the
//                     caller's record store.
//   2. seg_pass       ONE pass over the pixels: target+prediction slot maps
//                     (16-byte loads) feed the G x P pair histogram and the
//                     same target slots bin every detection mask (staged rows
//                     of 0/1 bytes, popcount per 16 pixels, warp-uniform skip
//                     of rows without a pixel). Persistent CTAs take halves of
//                     8192-pixel chunks from a counter; counts are summed over
//                     the warp and go to memory as reductions.
//   3. seg_score      per image: areas and validation, then (gated on the
//                     device error word) PQ/confusion accumulation and the
//                     detection areas / thing-class targets for matching.
//   4. match          batched COCO greedy matching (pe_instance.cu), gated too.
// InstanceEvaluator's mask-vs-mask IoU path uses the same table with
// inst_overlap (bit-packed AND + popcount over chunks, order indirection).
#include "pe_common.cuh"
#include "pe_score.cuh"
#include "pe_bins.cuh"
#include "pe_desc.cuh"
#include "pe_order.cuh"

#include <cfloat>
#include <map>
#include <mutex>

namespace pe {

template <typename Area>
int launch_match_gated(const u32* pairs, const int64_t* pair_off, const int64_t* d_off, const int64_t* g_off,
                       int64_t B, const int* pc, const Area* pa, const int* gc, const Area* ga, const uint8_t* crowd,
                       const double* areas, int C, int g_max, int8_t* flags, int64_t chain_stride, int64_t det_stride,
                       int* ranks, int64_t* counts, const int* gate, const uint32_t* class_bits, int unchecked,
                       cudaStream_t stream);

namespace {

constexpr int kPassThreads = 512;
constexpr int kPassPixels = 16;
constexpr int kChunk = kPassThreads * kPassPixels;  // 8192 pixels
constexpr int kScoreThreads = 1024;  // half of them when images outnumber the SMs
constexpr size_t kScoreSmemAlone = 200 * 1024, kScoreSmemShared = 110 * 1024;

__global__ void __launch_bounds__(kSortThreads) seg_sort_kernel(const int64_t* __restrict__ descs, ScoreOrder order) {
  wait_for_earlier_kernels();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  sort_image(desc_of(descs, blockIdx.x), order, smem_raw);
}

// Tunables of the fused pass (compile-time): masks per look-ahead group, and
// whether the first group is requested before the slot maps are consumed.
#ifndef PE_PASS_GROUP
#define PE_PASS_GROUP 4
#endif
#ifndef PE_PASS_PRELOAD
#define PE_PASS_PRELOAD 1
#endif
#ifndef PE_PASS_MIN_BLOCKS
#define PE_PASS_MIN_BLOCKS 1
#endif
constexpr int kGroup = PE_PASS_GROUP;

// 2. The fused pixel pass: one read of both slot maps and every detection mask.
__global__ void __launch_bounds__(kPassThreads, PE_PASS_MIN_BLOCKS)
seg_pass_kernel(const int64_t* __restrict__ descs, int64_t B, int64_t total_chunks, int64_t chunks_per_cta,
                const int64_t* __restrict__ bounds,
                const int64_t* __restrict__ order, u32* __restrict__ pairs, u32* __restrict__ dpairs,
                int* __restrict__ error) {
  wait_for_earlier_kernels();
  // Contiguous chunk range of this CTA: host-balanced bounds, or an even split.
  const int64_t c_begin = bounds ? bounds[blockIdx.x] : (int64_t)blockIdx.x * chunks_per_cta;
  const int64_t c_end = bounds ? min(bounds[blockIdx.x + 1], total_chunks) : min(c_begin + chunks_per_cta, total_chunks);
  if (c_begin >= c_end) return;
  int64_t b = image_of_chunk(descs, B, c_begin);
  bool bad = false;
  const int lane = threadIdx.x & 31;
  int64_t chunk = c_begin;
  while (chunk < c_end) {
    const int64_t* d = desc_of(descs, b);
    const int64_t first = d[kChunkBegin];
    const int64_t pixels = d[kPixels];
    const int64_t last = first + ceil_div(pixels, kChunk);  // exclusive
    if (chunk >= last) { ++b; continue; }
    const int G = (int)d[kG], P = (int)d[kP], D = (int)d[kD];
    const int* target = reinterpret_cast<const int*>(d[kTarget]);
    const int* pred = reinterpret_cast<const int*>(d[kPred]);
    const uint8_t* masks = reinterpret_cast<const uint8_t*>(d[kMasks]);
    const int64_t stride = d[kMaskStride];
    const int64_t* ord = order + d[kDetBegin];
    const bool vec_maps = d[kFlags] & 1, vec_masks = d[kFlags] & 2;
    u32* image_pairs = pairs + d[kPairBegin];
    u32* image_dpairs = dpairs + d[kDPairBegin];
    const int64_t stop = min(last, c_end);
    for (; chunk < stop; ++chunk) {
      const int64_t x = (chunk - first) * kChunk + (int64_t)threadIdx.x * kPassPixels;
      const int64_t xm = x < pixels ? x : pixels;
      uint4 cur[kGroup], nxt[kGroup];
      if (PE_PASS_PRELOAD) {  // first group of masks in flight before the slot maps are consumed
#pragma unroll
        for (int k = 0; k < kGroup; ++k)
          cur[k] = k < D ? load16_stream(masks + ord[k] * stride, xm, pixels, vec_masks) : make_uint4(0, 0, 0, 0);
      }
      int t[16];
      {
        int p[16];
        load16_maps(target, x, pixels, vec_maps, t);
        if (pred) {
          load16_maps(pred, x, pixels, vec_maps, p);
          add_pairs(t, p, x, pixels, G, P, image_pairs, bad);
        }
      }
      if (!PE_PASS_PRELOAD) {
#pragma unroll
        for (int k = 0; k < kGroup; ++k)
          cur[k] = k < D ? load16_stream(masks + ord[k] * stride, xm, pixels, vec_masks) : make_uint4(0, 0, 0, 0);
      }
      const LaneSlots ls = lane_slots(t, x, pixels, G, bad);
      // Detections: groups of kGroup masks with one group of look-ahead; one
      // warp-wide OR tells which masks of the group have any pixel here.
      for (int r0 = 0; r0 < D; r0 += kGroup) {
#pragma unroll
        for (int k = 0; k < kGroup; ++k) {
          const int r = r0 + kGroup + k;
          nxt[k] = r < D ? load16_stream(masks + ord[r] * stride, xm, pixels, vec_masks) : make_uint4(0, 0, 0, 0);
        }
        u32 bits = 0;
#pragma unroll
        for (int k = 0; k < kGroup; ++k) bits |= (u32)((cur[k].x | cur[k].y | cur[k].z | cur[k].w) != 0) << k;
        const u32 warp_bits = __reduce_or_sync(0xffffffffu, bits);
#pragma unroll
        for (int k = 0; k < kGroup; ++k)
          if ((warp_bits >> k) & 1u)   // uniform across the warp
            add_slots(t, ls, pack16(cur[k]), image_dpairs + (int64_t)(r0 + k) * G);
#pragma unroll
        for (int k = 0; k < kGroup; ++k) cur[k] = nxt[k];
      }
    }
    ++b;
  }
  if (bad && error) atomicOr(error, 1);
}

// 2b. The fused pass as a bulk-copy pipeline. ANY_ALIGN = false: every mask
// row starts on a 16-byte boundary (e.g. a ragged.SegmentationImages arena);
// true: rows at any byte offset, the producer copies the aligned 16-byte words
// covering each row segment and the consumers re-align them by the row's offset.
// Warp 8 is the producer: it takes 4096-pixel halves of 8192-pixel chunks,
// publishes each with its image's descriptor in a small queue of kHalfRing
// entries, prefetches its slot maps into L2 and streams its 4096-byte mask-row
// segments into a ring of kRing shared-memory slots with cp.async.bulk,
// completing on per-slot "full" mbarriers. What the producer waits for bounds the
// launch (by one lane, a stage took it 1800 cycles, 250 of them for a free slot: a
// load of each row's place in the score order, and a search for the image per
// half), so the whole warp produces: 32 places are loaded at once, one stage block
// ahead, a lane copies a row, the image is found in one round trip and the next
// half is claimed before this one's last rows: 8 images of 512 x 768 with 256
// detections 149 -> 124 us, 64 uneven images 322 -> 278 (6.3 TB/s). Halves come from a global counter (`schedule`,
// one atomicAdd per `grab` of them), so CTAs that run faster take more of them,
// or, without a counter, from a contiguous range of chunks per CTA. The counter's last halves
// are taken in parts, a range of the detections each: whole halves would leave most CTAs waiting
// for the few with one half more (see pe_seg_pass). Warps 0-7 consume: they
// take the next half from the queue, read the target/prediction slots of their
// 16 pixels with plain loads (kept in registers), then take each mask segment
// from the ring, bin it exactly as the register path does and release the slot
// on its "empty" mbarrier. All counts are integer atomics, so the result does
// not depend on which CTA took which chunk. Every wait is bounded by kWaitLimit
// clock cycles; a timeout sets bit 30 of *error, the producer waits for its
// copies in flight, and all roles return.
constexpr int kBulkConsumers = 256;
constexpr int kBulkThreads = kBulkConsumers + 32;
constexpr int kHalf = kBulkConsumers * kPassPixels;  // 4096 pixels per step
constexpr int kStageMasks = 4;  // mask-row segments per ring stage (one barrier each)
constexpr int kRing = 6;        // stages in flight per CTA (two CTAs hold 197 KB; 4 stages: 310 us where 6 take 293)
constexpr int kHalfRing = 4;    // published halves in flight per CTA
constexpr int kPartRows = 16;   // detections of a part, at least: its maps are read again, from L2
constexpr long long kWaitLimit = 4000000000ll;  // about two seconds of SM clock
constexpr int kTimeoutBit = 1 << 30;

struct BulkShared {
  unsigned char ring[kRing][kStageMasks][kHalf + 16];  // the aligned words covering each row segment
  unsigned char shift[kRing][kStageMasks];             // each row's start offset mod 16
  int64_t half_desc[kHalfRing][kDescFields];  // the image's descriptor
  int64_t half_x0[kHalfRing];     // first pixel of the half; -1 ends the CTA's work
  int half_rows[kHalfRing][2];    // detections [first, end); the first part counts the maps' pairs too
  uint64_t full[kRing];
  uint64_t empty[kRing];
  uint64_t half_full[kHalfRing];
  uint64_t half_empty[kHalfRing];
  int abort;
};

template <bool ANY_ALIGN>
__global__ void __launch_bounds__(kBulkThreads, 2)
seg_pass_bulk_kernel(const int64_t* __restrict__ descs, int64_t B, int64_t total_chunks, int64_t chunks_per_cta,
                     const int64_t* __restrict__ bounds, unsigned long long* __restrict__ schedule, int grab,
                     int64_t whole, int parts,
                     const int64_t* __restrict__ order, u32* __restrict__ pairs, u32* __restrict__ dpairs,
                     int* __restrict__ error) {
  wait_for_earlier_kernels();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BulkShared& sm = *reinterpret_cast<BulkShared*>(smem_raw);
  // Without a counter: a contiguous chunk range per CTA (host-balanced bounds, or an even split).
  const int64_t c_begin = bounds ? bounds[blockIdx.x] : (int64_t)blockIdx.x * chunks_per_cta;
  const int64_t c_end = bounds ? min(bounds[blockIdx.x + 1], total_chunks) : min(c_begin + chunks_per_cta, total_chunks);
  if (!schedule && c_begin >= c_end) return;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&sm.full[i], 1);
      mbar_init(&sm.empty[i], kBulkConsumers / 32);
    }
    for (int i = 0; i < kHalfRing; ++i) {
      mbar_init(&sm.half_full[i], 1);
      mbar_init(&sm.half_empty[i], kBulkConsumers / 32);
    }
    sm.abort = 0;
    mbar_fence_init();
  }
  __syncthreads();
  volatile int* abort = &sm.abort;

  if (threadIdx.x >= kBulkConsumers) {
    // ---- producer --------------------------------------------------------
    const int lane = threadIdx.x & 31;
    RingSlot<kRing> stage;
    RingSlot<kHalfRing> half;
    int64_t sent = 0, next = 2 * c_begin;  // stages; work is taken in halves, two per chunk
    // With a counter: the current claim of `grab` consecutive units, the first `whole` of them halves, then
    // the other halves' first parts, their second parts, and so on.
    int64_t claimed = 0, claim_end = 0;
    unsigned long long claim = 0;
    bool ok = true, asked = false;
    const int64_t split = 2 * total_chunks - whole, units = whole + split * parts;
    auto ask = [&] {
      if (lane == 0) claim = atomicAdd(schedule, (unsigned long long)grab);
      asked = true;
    };
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, kWaitLimit) && !*abort) != 0;
    };
    // Publish the next half (x0 -1: no more work); false when the wait for a free entry fails.
    auto publish = [&](int64_t word, int64_t x0, int first_row, int end_row) {
      if (!wait(&sm.half_empty[half.at], half.phase ^ 1u)) return false;
      if (lane < kDescFields) sm.half_desc[half.at][lane] = word;
      if (lane == 0) {
        sm.half_x0[half.at] = x0;
        sm.half_rows[half.at][0] = first_row;
        sm.half_rows[half.at][1] = end_row;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.half_full[half.at]);  // release: the entry is visible with the phase
      half.next();
      return true;
    };
    while (ok) {
      int64_t unit;
      int part = 0, of = 1;
      if (schedule) {
        if (claimed == claim_end) {
          if (!asked) ask();
          claimed = (int64_t)__shfl_sync(0xffffffffu, claim, 0);
          claim_end = min(claimed + grab, units);
          asked = false;
        }
        if (claimed >= claim_end) break;
        unit = claimed++;
        if (unit >= whole) {
          of = parts;
          part = (int)((unit - whole) / split);
          unit = whole + (unit - whole) % split;
        }
      } else {
        if (next >= 2 * c_end) break;
        unit = next++;
      }
      const int64_t chunk = unit >> 1;
      const int64_t b = find_row<kDescFields>(descs, B, kChunkBegin, chunk);
      const int64_t word = lane < kDescFields ? desc_of(descs, b)[lane] : 0;
      auto field = [&](int f) { return __shfl_sync(0xffffffffu, word, f); };
      const int64_t pixels = field(kPixels);
      const int64_t x0 = (chunk - field(kChunkBegin)) * kChunk + (unit & 1) * kHalf;
      if (x0 >= pixels) continue;  // the second half of an image's last chunk
      const int D = (int)field(kD);
      const int each = of == 1 ? D : max(kPartRows, (D + of - 1) / of);
      const int first_row = part * each, end_row = min(D, first_row + each);
      if (part > 0 && first_row >= D) continue;
      const int64_t stride = field(kMaskStride);
      const uint8_t* masks = reinterpret_cast<const uint8_t*>(field(kMasks)) + x0;
      const int64_t* ord = order + field(kDetBegin);
      int64_t place = first_row + lane < end_row ? ord[first_row + lane] : 0;
      if (!publish(word, x0, first_row, end_row)) {
        ok = false;
        break;
      }
      const int64_t len = min((int64_t)kHalf, pixels - x0);
      const uint32_t map_bytes = (uint32_t)((len * 4) & ~15ll);
      if ((field(kFlags) & 1) && map_bytes) {  // lane 0: the target map, lane 1: the prediction
        const int64_t map = field(lane == 1 ? kPred : kTarget);
        if (lane < (part == 0 ? 2 : 1) && map) bulk_prefetch_l2(reinterpret_cast<const int*>(map) + x0, map_bytes);
      }
      for (int r32 = first_row; ok && r32 < end_row; r32 += 32) {
        const uint8_t* row = masks + place * stride;  // lane l: row r32 + l
        if (r32 + 32 + lane < end_row) place = ord[r32 + 32 + lane];
        for (int r0 = r32; r0 < min(r32 + 32, end_row); r0 += kStageMasks) {
          if (!wait(&sm.empty[stage.at], stage.phase ^ 1u)) {
            ok = false;
            break;
          }
          const int n = min(kStageMasks, end_row - r0);
          // Rows may start at any byte: copy the aligned words from the one holding pixel x0 to the
          // one holding the segment's last byte; the consumers re-align by the row's offset.
          const uint64_t from = __shfl_sync(0xffffffffu, reinterpret_cast<uint64_t>(row), (r0 - r32 + lane) & 31);
          const int o = ANY_ALIGN ? (int)(from & 15) : 0;
          const uint32_t bytes = lane < n ? (uint32_t)round_up(len + o, 16) : 0u;
          if (ANY_ALIGN && lane < n) sm.shift[stage.at][lane] = (unsigned char)o;
          const uint32_t total = __reduce_add_sync(0xffffffffu, bytes);
          __syncwarp();
          if (lane == 0) mbar_arrive_expect_tx(&sm.full[stage.at], total);  // release: the offsets too
          __syncwarp();
          if (lane < n)
            bulk_copy_g2s(sm.ring[stage.at][lane], reinterpret_cast<const uint8_t*>(from) - o, bytes,
                          &sm.full[stage.at]);
          stage.next();
          ++sent;
          if (schedule && claimed == claim_end && !asked && r0 + 2 * kStageMasks >= end_row) ask();
        }
      }
    }
    if (ok) ok = publish(0, -1, 0, 0);
    if (!ok) {
      *abort = 1;
      if (lane == 0) atomicOr(error, kTimeoutBit);
    }
    // Wait for the copies still in flight into this CTA's shared memory.
    for (int64_t q = sent > kRing ? sent - kRing : 0; q < sent; ++q)
      mbar_wait(&sm.full[q % kRing], (uint32_t)((q / kRing) & 1), kWaitLimit);
    return;
  }

  // ---- consumers ---------------------------------------------------------
  const int ctid = threadIdx.x, lane = ctid & 31;
  RingSlot<kRing> stage;
  RingSlot<kHalfRing> half;
  bool ok = true, bad = false;
  while (ok) {
    const bool ready = mbar_wait(&sm.half_full[half.at], half.phase, kWaitLimit);
    if (!__all_sync(0xffffffffu, ready && !*abort)) {
      ok = false;
      break;
    }
    const int64_t x0 = sm.half_x0[half.at];
    const int first_row = sm.half_rows[half.at][0], end_row = sm.half_rows[half.at][1];
    const int64_t* d = sm.half_desc[half.at];
    if (x0 < 0) break;
    const int64_t pixels = d[kPixels];
    const int G = (int)d[kG], P = (int)d[kP];
    const int* target = reinterpret_cast<const int*>(d[kTarget]);
    const int* pred = first_row ? nullptr : reinterpret_cast<const int*>(d[kPred]);
    const bool vec_maps = d[kFlags] & 1;
    u32* image_pairs = pairs + d[kPairBegin];
    u32* image_dpairs = dpairs + d[kDPairBegin];
    __syncwarp();  // the entry is in registers
    if (lane == 0) mbar_arrive(&sm.half_empty[half.at]);
    half.next();
    const int64_t x = x0 + (int64_t)ctid * kPassPixels;
    const bool in_image = x - lane * kPassPixels < pixels;  // any of the warp's pixels
    int t[16];
    {
      int p[16];
      load16_maps(target, x, pixels, vec_maps, t);
      if (pred) {
        load16_maps(pred, x, pixels, vec_maps, p);
        add_pairs(t, p, x, pixels, G, P, image_pairs, bad);
      }
    }
    const LaneSlots ls = lane_slots(t, x, pixels, G, bad);
    for (int r0 = first_row; r0 < end_row; r0 += kStageMasks) {
      const bool got = mbar_wait(&sm.full[stage.at], stage.phase, kWaitLimit);
      if (!__all_sync(0xffffffffu, got && !*abort)) {  // warp-uniform decision
        ok = false;
        break;
      }
      // One warp-wide OR tells which masks of the stage have a pixel here (a superset: the staged words of all
      // lanes as they lie, since a lane's pixels end in the next lane's word, past the image with what the slot held
      // before); only those are re-aligned and counted, by one copy of the counting code, and `ls` holds no pixel
      // past the image.
      const unsigned char* staged = &sm.ring[stage.at][0][ctid * kPassPixels];
      constexpr int kRowBytes = kHalf + 16;
      u32 hit = 0;
#pragma unroll
      for (int k = 0; k < kStageMasks; ++k) {
        const uint4 a = *reinterpret_cast<const uint4*>(staged + k * kRowBytes);
        u32 any = a.x | a.y | a.z | a.w;
        if (ANY_ALIGN && lane == 31 && sm.shift[stage.at][k]) {  // the warp's pixels end in the next word
          const uint4 c = *reinterpret_cast<const uint4*>(staged + k * kRowBytes + 16);
          any |= c.x | c.y | c.z | c.w;
        }
        hit |= (u32)(any != 0) << k;
      }
      hit = __reduce_or_sync(0xffffffffu, in_image ? hit : 0u) & ((1u << min(kStageMasks, end_row - r0)) - 1u);
#pragma unroll 1
      for (; hit; hit &= hit - 1) {
        const int k = __ffs(hit) - 1;
        uint4 w = *reinterpret_cast<const uint4*>(staged + k * kRowBytes);
        if constexpr (ANY_ALIGN) {
          const int o = sm.shift[stage.at][k];  // the same for the whole warp
          if (o) w = realign16(w, *reinterpret_cast<const uint4*>(staged + k * kRowBytes + 16), o);
        }
        add_slots(t, ls, pack16(w), image_dpairs + (int64_t)(r0 + k) * G);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.empty[stage.at]);
      stage.next();
    }
  }
  if (!ok) {
    *abort = 1;
    if (lane == 0) atomicOr(error, kTimeoutBit);
  }
  if (bad && error) atomicOr(error, 1);
}

// 3. Per-image scoring. mode bit 1: areas + validation, bit 2: accumulate
// (gated by *error when bit 4 is set). smem: dynamic shared memory of the launch;
// an image whose tables do not fit it is scored in place.
__global__ void __launch_bounds__(kScoreThreads)
seg_score_kernel(const int64_t* __restrict__ descs, const u32* __restrict__ pairs, const u32* __restrict__ dpairs,
                 const int* __restrict__ gc, const int* __restrict__ pc, const uint8_t* __restrict__ crowd,
                 u64* __restrict__ areas, int* __restrict__ matched, ScoreOut out, int C,
                 const uint8_t* __restrict__ isthing, const int* __restrict__ det_classes,
                 const double* __restrict__ det_scores, double* __restrict__ det_pa, double* __restrict__ slot_ga,
                 int* __restrict__ slot_class, const double* __restrict__ ann_in, double* __restrict__ ann_out,
                 int mode, int validate, int reward, int smem, u32* __restrict__ class_bits,
                 int* __restrict__ error) {
  wait_for_earlier_kernels();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if ((mode & 4) && *reinterpret_cast<volatile int*>(error)) return;
  const int stopped = !validate && error ? __ldcg(error) & kStoppedBits : 0;
  const int64_t* d = desc_of(descs, blockIdx.x);
  const int G = (int)d[kG], P = (int)d[kP], D = (int)d[kD];
  const int64_t sb = d[kSlotBegin], pb = d[kPSlotBegin], db = d[kDetBegin];
  const u32* pan = pairs + d[kPairBegin];
  const bool blocks = P > 0 && ScoreTables::base_bytes(G, P, C) <= (size_t)smem;
  const ScoreTables t = ScoreTables::at(smem_raw, G, P, C, blocks ? smem : ScoreTables::base_bytes(G, P, C));
  const int shares = (int64_t)G * P > kSharedScore ? (int)gridDim.y : 1;  // CTAs that count the image's pairs
  const u32* det = dpairs + d[kDPairBegin];
  // Detection areas (full mask area: every slot, including void and stuff) and checks, by `parts` blocks: a warp
  // sums the rows of kAreaRows detections at once with coalesced loads, so their L2 round trips overlap.
  auto detection_areas = [&](int part, int parts) {
    constexpr int kAreaRows = 4;
    int err = 0;
    const int lane = threadIdx.x & 31, warps = parts * (blockDim.x >> 5);
    for (int r0 = part * (blockDim.x >> 5) + (threadIdx.x >> 5); r0 < D; r0 += kAreaRows * warps) {
      u64 sum[kAreaRows];
#pragma unroll
      for (int j = 0; j < kAreaRows; ++j) sum[j] = 0;
      for (int s = lane; s < G; s += 32) {
#pragma unroll
        for (int j = 0; j < kAreaRows; ++j) {
          const int r = r0 + j * warps;
          if (r < D) sum[j] += det[(int64_t)r * G + s];
        }
      }
#pragma unroll
      for (int j = 0; j < kAreaRows; ++j) {
        const int r = r0 + j * warps;
#pragma unroll
        for (int off = 16; off; off >>= 1) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], off);
        if (lane || r >= D) continue;
        det_pa[db + r] = (double)sum[j];
        if (validate) {
          const int c = det_classes[db + r];
          if (c < 0 || c >= C || !isthing[c]) err |= 8;
          if (sum[j] == 0) err |= 16;
          const double sc = det_scores[db + r];
          if (!(sc == sc) || sc == __longlong_as_double(0x7ff0000000000000ll) ||
              sc == -__longlong_as_double(0x7ff0000000000000ll))
            err |= 32;
        }
      }
    }
    return err;
  };
  if (blockIdx.y) {  // blocks beside the image's scoring: their share of the counts, then the detections
    if (blocks && shares > 1) score_totals(pan, t, gc + sb, crowd + sb, G, P, C, blockIdx.y, shares);
    if (!(mode & 1)) return;
    const int err = detection_areas(blockIdx.y - 1, gridDim.y - 1);
    if (err) atomicOr(error, err);
    return;
  }
  gc += sb; crowd += sb; matched += sb;
  pc += pb;
  u64* ar = areas + sb + pb;  // per image G + P entries at offset (slot_begin + pslot_begin)
  if (blocks) score_totals(pan, t, gc, crowd, G, P, C, 0, shares);
  if (mode & 1) {
    int err = 0;
    if (blocks) {
      for (int k = threadIdx.x; k < G; k += blockDim.x) ar[k] = t.row[k];
      for (int k = threadIdx.x; k < P; k += blockDim.x) ar[G + k] = t.col[k];
      if (validate)
        err = reward ? score_checks<true>(t, gc, pc, crowd, G, P, C) : score_checks<false>(t, gc, pc, crowd, G, P, C);
    } else if (P > 0) {
      err = reward ? score_areas<u32, true>(pan, gc, pc, crowd, ar, G, P, C, validate)
                   : score_areas<u32, false>(pan, gc, pc, crowd, ar, G, P, C, validate);
    }
    if (gridDim.y == 1) err |= detection_areas(0, 1);
    if (validate && ann_in) {
      for (int s = threadIdx.x; s < G; s += blockDim.x) {
        const double v = ann_in[sb + s];
        if (!(v >= 0.0) || v == __longlong_as_double(0x7ff0000000000000ll)) err |= 64;
      }
    }
    if (err) atomicOr(error, err);
    __syncthreads();
  }
  if (!(mode & 2)) return;
  if (stopped) {  // the counts are not all there, and nobody reads the word
    if (blockIdx.x || reward) return;
    for (int c = threadIdx.x; c < C; c += blockDim.x) out.iou_sum[c] = __longlong_as_double(0x7ff8000000000000ll);
    if (threadIdx.x == 0) atomicOr(error, kUncheckedBit);
    return;
  }
  if (reward) {  // per-image rows [B][C], no confusion (evaluator.py:497-538)
    const int64_t o = (int64_t)blockIdx.x * C;
    ScoreOut row{out.tp + o, out.fp + o, out.fn + o, out.iou_sum + o, nullptr};
    if (blocks) score_matches<u32, true>(pan, t, pc, G, P, C, row);
    else if (P > 0) score_accumulate<u32, true>(pan, gc, pc, crowd, ar, matched, G, P, C, row, smem_raw);
    return;
  }
  if (blocks) score_matches<u32, false>(pan, t, pc, G, P, C, out);
  else if (P > 0) score_accumulate<u32, false>(pan, gc, pc, crowd, ar, matched, G, P, C, out, smem_raw);
  // Classes present in the image for the matching (per-image bits): thing targets, and detections
  // (a class outside [0, C) marks class 0, whose matching warp handles such detections).
  u32* bits = class_bits ? class_bits + (int64_t)blockIdx.x * ((C + 31) / 32) : nullptr;
  if (bits) {
    for (int w = threadIdx.x; w < (C + 31) / 32; w += blockDim.x) bits[w] = 0;
    __syncthreads();
    for (int r = threadIdx.x; r < D; r += blockDim.x) {
      const int c = det_classes[db + r];
      const int k = c >= 0 && c < C ? c : 0;
      atomicOr(bits + (k >> 5), 1u << (k & 31));
    }
  }
  // Targets for matching: thing classes only, pixel areas, annotation areas.
  for (int s = threadIdx.x; s < G; s += blockDim.x) {
    const int c = gc[s];
    const int clamped = c < 0 ? 0 : (c >= C ? C - 1 : c);
    slot_class[sb + s] = (c >= 0 && isthing[clamped]) ? c : -1;
    if (bits && c >= 0 && c < C && isthing[c]) atomicOr(bits + (c >> 5), 1u << (c & 31));
    const double area = (double)ar[s];
    slot_ga[sb + s] = area;
    ann_out[sb + s] = ann_in ? ann_in[sb + s] : area;
  }
}

// Mask-vs-mask overlaps for InstanceEvaluator (pixel chunks of 4096).
constexpr int kOvThreads = 256;
constexpr int kOvWords = 128;

__device__ __forceinline__ uint32_t pack4(uint32_t w) { return (((w & 0x01010101u) * 0x08040201u) >> 24) & 0xfu; }

__global__ void __launch_bounds__(kOvThreads)
inst_overlap_kernel(const int64_t* __restrict__ descs, int64_t B, const int64_t* __restrict__ order,
                    const int* __restrict__ pc, const int* __restrict__ gc, u32* __restrict__ inter,
                    u64* __restrict__ pa, u64* __restrict__ ga) {
  wait_for_earlier_kernels();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int64_t b = image_of_chunk(descs, B, blockIdx.x);
  const int64_t* d = desc_of(descs, b);
  const int D = (int)d[kD], G = (int)d[kG];
  const int64_t pixels = d[kPixels], stride = d[kMaskStride];
  const uint8_t* pm = reinterpret_cast<const uint8_t*>(d[kMasks]);
  const uint8_t* gm = reinterpret_cast<const uint8_t*>(d[kTarget]);
  const bool vec = d[kFlags] & 2;
  const int64_t db = d[kDetBegin], gb = d[kSlotBegin];
  const int64_t x0 = (blockIdx.x - d[kChunkBegin]) * (int64_t)kOvWords * 32;
  const int rows = D + G;
  uint32_t* bits = reinterpret_cast<uint32_t*>(smem_raw);
  int2* range = reinterpret_cast<int2*>(bits + (int64_t)rows * kOvWords);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r = warp; r < rows; r += kOvThreads / 32) {
    const uint8_t* row = r < D ? pm + order[db + r] * stride : gm + (int64_t)(r - D) * stride;
    int first = kOvWords, last = -1, ones = 0;
    for (int k = lane; k < kOvWords; k += 32) {
      const int64_t x = x0 + (int64_t)k * 32;
      uint32_t word = 0;
      if (x < pixels) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint4 w = load16_mask(row, x + 16 * q, pixels, vec);
          word |= (pack4(w.x) | pack4(w.y) << 4 | pack4(w.z) << 8 | pack4(w.w) << 12) << (16 * q);
        }
      }
      bits[(int64_t)r * kOvWords + k] = word;
      ones += __popc(word);
      if (word) { first = min(first, k); last = max(last, k); }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
      last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
      ones += __shfl_xor_sync(0xffffffffu, ones, o);
    }
    if (lane == 0) {
      range[r] = make_int2(first, last);
      if (ones) atomicAdd(r < D ? pa + db + r : ga + gb + (r - D), (u64)ones);
    }
  }
  __syncthreads();
  u32* out = inter + d[kDPairBegin];
  for (int pair = threadIdx.x; pair < D * G; pair += blockDim.x) {
    const int i = pair / G, g = pair % G;
    if (pc[db + i] != gc[gb + g]) continue;
    const int2 rd = range[i], rg = range[D + g];
    const int lo = max(rd.x, rg.x), hi = min(rd.y, rg.y);
    if (lo > hi) continue;
    const uint32_t* a = bits + (int64_t)i * kOvWords;
    const uint32_t* c = bits + (int64_t)(D + g) * kOvWords;
    u32 count = 0;
    for (int k = lo; k <= hi; ++k) count += __popc(a[k] & c[k]);
    if (count) atomicAdd(out + pair, count);
  }
}

__global__ void __launch_bounds__(128) inst_gather_kernel(const int64_t* __restrict__ descs, FieldGather fields) {
  wait_for_earlier_kernels();
  gather_image(desc_of(descs, blockIdx.x), blockIdx.x, fields);
}

// Instance prep: pixel areas to double, validation of classes/scores/areas.
__global__ void inst_prepare_kernel(const int64_t* __restrict__ descs, const u64* __restrict__ pa_count,
                                    const u64* __restrict__ ga_count, double* __restrict__ pa, double* __restrict__ ga,
                                    const int* __restrict__ pc, const int* __restrict__ gc,
                                    const double* __restrict__ scores, const double* __restrict__ ann_in,
                                    double* __restrict__ ann_out, int C, int validate, u32* __restrict__ class_bits,
                                    int* __restrict__ error) {
  wait_for_earlier_kernels();
  const int64_t* d = desc_of(descs, blockIdx.x);
  const int D = (int)d[kD], G = (int)d[kG];
  const int64_t db = d[kDetBegin], gb = d[kSlotBegin];
  // Classes present in the image for the matching (a detection class outside [0, C) marks class 0).
  u32* bits = class_bits ? class_bits + (int64_t)blockIdx.x * ((C + 31) / 32) : nullptr;
  if (bits) {
    for (int w = threadIdx.x; w < (C + 31) / 32; w += blockDim.x) bits[w] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < D; i += blockDim.x) {
      const int c = pc[db + i];
      const int k = c >= 0 && c < C ? c : 0;
      atomicOr(bits + (k >> 5), 1u << (k & 31));
    }
    for (int g = threadIdx.x; g < G; g += blockDim.x) {
      const int c = gc[gb + g];
      if (c >= 0 && c < C) atomicOr(bits + (c >> 5), 1u << (c & 31));
    }
  }
  int err = 0;
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    pa[db + i] = (double)pa_count[db + i];
    if (validate) {
      if (pc[db + i] < 0 || pc[db + i] >= C) err |= 8;
      if (pa_count[db + i] == 0) err |= 16;
      const double s = scores[db + i];
      if (!(s == s) || s == inf || s == -inf) err |= 32;
    }
  }
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    const double area = (double)ga_count[gb + g];
    ga[gb + g] = area;
    ann_out[gb + g] = ann_in ? ann_in[gb + g] : area;
    if (validate) {
      if (gc[gb + g] < 0 || gc[gb + g] >= C) err |= 8;
      if (ga_count[gb + g] == 0) err |= 16;
      if (ann_in) {
        const double v = ann_in[gb + g];
        if (!(v >= 0.0) || v == inf) err |= 64;
      }
    }
  }
  if (err) atomicOr(error, err);
  if (!validate && error && blockIdx.x == 0 && threadIdx.x == 0 &&
      (*reinterpret_cast<volatile int*>(error) & kStoppedBits))
    atomicOr(error, kUncheckedBit);
}

}  // namespace
}  // namespace pe

using namespace pe;

PE_API int pe_desc_fields(void) { return kDescFields; }

// Workspace for pe_seg_sort: key/index scratch for images with more than 4096 detections.
PE_API int64_t pe_seg_sort_workspace(int64_t total_detections) {
  return (int64_t)2 * round_up(total_detections + 1, 64) * (int64_t)(sizeof(double) + sizeof(int)) + 256;
}

// Stable descending score order per image (instance.py:139-141). order[det_begin + r]
// is the image-local index of the r-th best detection; sorted scores/classes
// go to the given outputs at det_begin + r.
PE_API int pe_seg_sort(const int64_t* descs, int64_t B, const double* scores, const int32_t* classes,
                       int64_t total_detections, int64_t* order, double* sorted_scores, int32_t* sorted_classes,
                       void* workspace, int64_t workspace_bytes, cudaStream_t stream) {
  PE_REQUIRE(B >= 0 && total_detections >= 0, "invalid batch");
  PE_REQUIRE(workspace_bytes >= pe_seg_sort_workspace(total_detections), "sort workspace too small");
  if (B == 0 || total_detections == 0) return kOk;
  const ScoreOrder out = score_order(scores, classes, total_detections, order, sorted_scores, sorted_classes, workspace);
  PE_CUDA(cudaFuncSetAttribute(seg_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sort_bytes(out.cap)));
  launch_kernel(seg_sort_kernel, (unsigned)B, kSortThreads, sort_bytes(out.cap), stream, descs, out);
  PE_LAUNCHED("seg_sort");
  count_launch();
  return kOk;
}

// The fused pixel pass. pairs (u32, sum of G*P) and dpairs (u32, sum of D*G)
// are zeroed here. pan_cap / det_cap: the largest per-image G*P and D*G.
// schedule (bulk form only, optional): one device u64, zeroed here, from which
// CTAs take chunks dynamically (cta_bounds is then unused).
// Launch choices of the batched pass with a chunk counter, per bucket floor(log2(total chunks)): chunks a
// producer takes per counter grab (1, 2 or 4) and CTAs per SM (1 or 2). Without an entry: 1 and 2.
namespace {
struct PassChoice {
  int grab = 1;
  int per_sm = 2;
};
std::mutex g_pass_mutex;
std::map<int, PassChoice> g_pass_tuning;

int log2_floor(int64_t v) { return v > 0 ? 63 - __builtin_clzll((unsigned long long)v) : -1; }

PassChoice pass_choice(int64_t chunks) {
  std::lock_guard<std::mutex> lock(g_pass_mutex);
  const auto it = g_pass_tuning.find(log2_floor(chunks));
  return it == g_pass_tuning.end() ? PassChoice{} : it->second;
}
}  // namespace

PE_API int pe_tune_pass(int64_t chunks, int grab, int ctas_per_sm) {
  PE_REQUIRE(chunks > 0, "chunks must be positive");
  std::lock_guard<std::mutex> lock(g_pass_mutex);
  if (grab < 0) {
    g_pass_tuning.erase(log2_floor(chunks));
    return kOk;
  }
  PE_REQUIRE(grab == 1 || grab == 2 || grab == 4, "grab must be 1, 2 or 4 chunks");
  PE_REQUIRE(ctas_per_sm == 1 || ctas_per_sm == 2, "ctas_per_sm must be 1 or 2");
  g_pass_tuning[log2_floor(chunks)] = PassChoice{grab, ctas_per_sm};
  return kOk;
}

PE_API int pe_pass_choice(int64_t chunks, int32_t* grab, int32_t* ctas_per_sm) {
  PE_REQUIRE(chunks > 0 && grab && ctas_per_sm, "invalid query");
  const PassChoice c = pass_choice(chunks);
  *grab = c.grab;
  *ctas_per_sm = c.per_sm;
  return kOk;
}

PE_API int pe_seg_pass(const int64_t* descs, int64_t B, int64_t total_chunks, const int64_t* order, uint32_t* pairs,
                       int64_t pairs_len, uint32_t* dpairs, int64_t dpairs_len, int64_t pan_cap, int64_t det_cap,
                       int bulk, const int64_t* cta_bounds, int64_t ctas, uint64_t* schedule, int32_t* error,
                       cudaStream_t stream) {
  PE_REQUIRE(B >= 0 && total_chunks >= 0 && pairs_len >= 0 && dpairs_len >= 0, "invalid batch");
  // Keys of one image are G*P + D*G < 2^32 - 1 (pan_cap, det_cap: largest per-image G*P and D*G).
  PE_REQUIRE(pan_cap >= 0 && det_cap >= 0 && pan_cap + det_cap < (int64_t)UINT32_MAX, "histogram too large");
  const bool counted = bulk && schedule && B > 0 && total_chunks > 0;  // chunks from the counter
  const int zeroed = zero_spans({{pairs, 4 * pairs_len}, {dpairs, 4 * dpairs_len}, {schedule, counted ? 8 : 0}}, stream);
  if (zeroed != kOk) return zeroed;
  if (B == 0 || total_chunks == 0) return kOk;
  PE_REQUIRE(!cta_bounds || (ctas > 0 && ctas <= INT_MAX), "invalid CTA count");
  if (bulk) {
    const PassChoice choice = pass_choice(total_chunks);
    const int64_t max_ctas = (int64_t)sm_count() * 2;
    const int64_t per_cta = ceil_div(total_chunks, std::min(total_chunks, max_ctas));
    int64_t grid = cta_bounds ? ctas : ceil_div(total_chunks, per_cta);
    // Chunks taken from the counter, `grab` at a time, by the chosen CTAs per SM; half a chunk at a time
    // while the halves are fewer than kFewHalves per CTA, where a CTA left with one chunk more than the
    // others is a large part of the launch (384 chunks on 304 CTAs: 207 us by chunks, 161 by halves). There
    // the halves beyond the last full round go in kParts parts (149 us by the one-lane producer, 124 now);
    // with more rounds it measured the same either way.
    int grab = 2 * choice.grab, parts = 1;
    int64_t whole = 2 * total_chunks;
    if (schedule) {
      constexpr int64_t kFewHalves = 16;
      constexpr int kParts = 8;
      const int64_t all = (int64_t)sm_count() * choice.per_sm;
      if (whole < kFewHalves * all) {
        grab = 1;
        parts = kParts;
        whole = whole / all * all;
      }
      grid = std::min(ceil_div(whole + (2 * total_chunks - whole) * parts, grab), all);
      cta_bounds = nullptr;
    }
    const size_t smem = sizeof(BulkShared) + 128;
    auto kernel = bulk == 2 ? seg_pass_bulk_kernel<true> : seg_pass_bulk_kernel<false>;
    PE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    launch_kernel(kernel, (unsigned)grid, kBulkThreads, smem, stream, descs, B, total_chunks, per_cta, cta_bounds,
        reinterpret_cast<unsigned long long*>(schedule), grab, whole, parts, order, pairs, dpairs, error);
    PE_LAUNCHED("seg_pass_bulk");
    count_launch();
    return kOk;
  }
  const int64_t max_ctas = (int64_t)sm_count() * PE_PASS_MIN_BLOCKS;
  const int64_t per_cta = ceil_div(total_chunks, std::min(total_chunks, max_ctas));
  const int64_t grid = cta_bounds ? ctas : ceil_div(total_chunks, per_cta);
  launch_kernel(seg_pass_kernel, (unsigned)grid, kPassThreads, 0, stream, descs, B, total_chunks, per_cta, cta_bounds,
      order, pairs, dpairs, error);
  PE_LAUNCHED("seg_pass");
  count_launch();
  return kOk;
}

// Per-image scoring of the fused pass (see seg_score_kernel). areas: sum of
// (G+P) u64 at slot_begin + pslot_begin; matched: sum of G ints. state: dataset
// tp/fp/fn/iou_sum [C], confusion [C, C+1]. Validation bits: 1/2/4 panoptic,
// 8 detection class not a thing, 16 empty detection, 32 non-finite score,
// 64 invalid annotation area. Accumulation is skipped when any bit is set; without validation, where a kernel before
// this one gave up (bits from 2^20), the dataset IoU sums become NaN.
PE_API int pe_seg_score(const int64_t* descs, int64_t B, int64_t max_p, int64_t max_pairs, const uint32_t* pairs,
                        const uint32_t* dpairs,
                        const int32_t* gc, const int32_t* pc, const uint8_t* crowd, int64_t* areas, int32_t* matched,
                        int64_t* tp, int64_t* fp, int64_t* fn, double* iou_sum, int64_t* confusion, int64_t C,
                        const uint8_t* isthing, const int32_t* det_classes, const double* det_scores, double* det_pa,
                        double* slot_ga, int32_t* slot_class, const double* ann_in, double* ann_out, int validate,
                        int reward, uint32_t* class_bits, int32_t* error, cudaStream_t stream) {
  PE_REQUIRE(B >= 0 && C > 0 && C < INT_MAX, "invalid batch");
  u32* bits = reward ? nullptr : reinterpret_cast<u32*>(class_bits);
  if (B == 0) return kOk;
  const size_t in_place = score_staging_bytes(std::max<int64_t>(max_p, 1));
  PE_REQUIRE(in_place <= 200 * 1024, "too many prediction slots (P=%lld)", (long long)max_p);
  // Tables and entry list of the largest image, the target tables counted as for kScoreSlots slots (an
  // image with more takes the list's room, or the in-place form). One CTA per SM may take 200 KB; more
  // images than SMs share them, two CTAs each.
  constexpr int64_t kScoreSlots = 1024;
  const bool alone = B <= sm_count();
  const size_t want = score_bytes(kScoreSlots, max_p, C, max_pairs);
  const size_t smem = std::max(in_place, std::min(want, alone ? kScoreSmemAlone : kScoreSmemShared));
  const int threads = alone ? kScoreThreads : kScoreThreads / 2;
  // SMs without an image take a share of its counts and sum its detections' areas: 8 images of 257 x 277 slots and 256
  // detections took 41 us with both in the image's block and one list atomic per row, 21.9 now.
  const unsigned parts = score_parts(B, sm_count());
  const dim3 grid((unsigned)B, parts);
  if (smem > 48 * 1024)
    PE_CUDA(cudaFuncSetAttribute(seg_score_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  ScoreOut out{reinterpret_cast<u64*>(tp), reinterpret_cast<u64*>(fp), reinterpret_cast<u64*>(fn), iou_sum,
               reinterpret_cast<u64*>(confusion)};
  auto* ua = reinterpret_cast<u64*>(areas);
  if (validate) {
    launch_clusters(seg_score_kernel, grid, parts, threads, smem, stream, descs, pairs, dpairs, gc, pc, crowd, ua, matched,
        out, (int)C, isthing, det_classes, det_scores, det_pa, slot_ga, slot_class, ann_in, ann_out, 1, 1, reward,
        (int)smem, nullptr, error);
    PE_LAUNCHED("seg_score(areas)");
    launch_clusters(seg_score_kernel, grid, parts, threads, smem, stream, descs, pairs, dpairs, gc, pc, crowd, ua,
        matched, out, (int)C, isthing, det_classes, det_scores, det_pa, slot_ga, slot_class, ann_in, ann_out, 2 | 4, 1,
        reward, (int)smem, bits, error);
    PE_LAUNCHED("seg_score(accumulate)");
    count_launch(2);
    return kOk;
  }
  launch_clusters(seg_score_kernel, grid, parts, threads, smem, stream, descs, pairs, dpairs, gc, pc, crowd, ua, matched,
      out, (int)C, isthing, det_classes, det_scores, det_pa, slot_ga, slot_class, ann_in, ann_out, 1 | 2, 0, reward,
      (int)smem, bits, error);
  PE_LAUNCHED("seg_score");
  count_launch();
  return kOk;
}

// Batched greedy matching over the descriptor table, gated on *gate (when
// nonzero, every record is left out: rank 0, flags -1). pairs_u32: D x G intersections per image at dpair_begin.
// Offsets are read from device arrays d_off [B+1], g_off [B+1], pair_off [B].
PE_API int pe_seg_match(const uint32_t* pairs, const int64_t* pair_off, const int64_t* d_off, const int64_t* g_off,
                        int64_t B, const int32_t* pc, const double* pa, const int32_t* gc, const double* ga,
                        const uint8_t* crowd, const double* areas, int64_t C, int64_t g_max, int8_t* flags,
                        int64_t chain_stride, int64_t det_stride, int32_t* ranks, int64_t* counts,
                        const int32_t* gate, const uint32_t* class_bits, cudaStream_t stream) {
  PE_REQUIRE(B >= 0 && C > 0 && C <= INT_MAX / 120 && g_max >= 0 && g_max < INT_MAX, "invalid batch");
  return launch_match_gated(pairs, pair_off, d_off, g_off, B, pc, pa, gc, ga, crowd, areas, (int)C,
                            (int)std::max<int64_t>(g_max, 1), flags, chain_stride, det_stride, ranks, counts, gate,
                            class_bits, 0, stream);
}

// pe_seg_match from the pixel counts of pe_inst_counts, for a batch that pe_inst_prepare need not check: 5 us less of
// the stream. areas (optional): annotation areas, else the targets' pixels.
PE_API int pe_inst_match(const uint32_t* pairs, const int64_t* pair_off, const int64_t* d_off, const int64_t* g_off,
                         int64_t B, const int32_t* pc, const uint64_t* pa, const int32_t* gc, const uint64_t* ga,
                         const uint8_t* crowd, const double* areas, int64_t C, int64_t g_max, int8_t* flags,
                         int64_t chain_stride, int64_t det_stride, int32_t* ranks, int64_t* counts,
                         const int32_t* gate, const uint32_t* class_bits, cudaStream_t stream) {
  PE_REQUIRE(B >= 0 && C > 0 && C <= INT_MAX / 120 && g_max >= 0 && g_max < INT_MAX, "invalid batch");
  return launch_match_gated(pairs, pair_off, d_off, g_off, B, pc, reinterpret_cast<const u64*>(pa), gc,
                            reinterpret_cast<const u64*>(ga), crowd, areas, (int)C,
                            (int)std::max<int64_t>(g_max, 1), flags, chain_stride, det_stride, ranks, counts, gate,
                            class_bits, 1, stream);
}

// Mask-vs-mask overlaps and pixel areas for InstanceEvaluator over the
// descriptor table (kTarget = gt masks, kMasks = prediction masks, rows
// kMaskStride bytes apart, kChunkBegin in 4096-pixel chunks). inter (u32,
// sum of D*G) and the area counters pa (sum of D), ga (sum of G) are zeroed here.
PE_API int pe_inst_overlap(const int64_t* descs, int64_t B, int64_t total_chunks, int64_t max_rows,
                           const int64_t* order, const int32_t* pc, const int32_t* gc, uint32_t* inter,
                           int64_t inter_len, uint64_t* pa, int64_t pa_len, uint64_t* ga, int64_t ga_len,
                           cudaStream_t stream) {
  PE_REQUIRE(B >= 0 && total_chunks >= 0, "invalid batch");
  const int zeroed = zero_spans({{inter, 4 * inter_len}, {pa, 8 * pa_len}, {ga, 8 * ga_len}}, stream);
  if (zeroed != kOk) return zeroed;
  if (B == 0 || total_chunks == 0) return kOk;
  const size_t smem = (size_t)std::max<int64_t>(max_rows, 1) * (kOvWords * sizeof(uint32_t) + sizeof(int2));
  PE_REQUIRE(smem <= 220 * 1024, "too many masks per image for the overlap kernel (%lld)", (long long)max_rows);
  if (smem > 48 * 1024)
    PE_CUDA(cudaFuncSetAttribute(inst_overlap_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch_kernel(inst_overlap_kernel, (unsigned)total_chunks, kOvThreads, smem, stream, descs, B, order, pc, gc, inter,
      reinterpret_cast<u64*>(pa), reinterpret_cast<u64*>(ga));
  PE_LAUNCHED("inst_overlap");
  count_launch();
  return kOk;
}

// Pixel areas to FP64, annotation areas (given or pixel) and validation
// bits 8 (class), 16 (empty mask), 32 (score), 64 (annotation area).
// Flat instance metadata from per-image tensors (see inst_gather_kernel): pc [sum D] int32, scores
// [sum D] float64, gc / crowd / areas [sum G] (int32, uint8, float64; areas may be NULL).
PE_API int pe_inst_gather(const int64_t* descs, const int64_t* fields, int64_t B, int32_t* pc, double* scores,
                          int32_t* gc, uint8_t* crowd, double* areas, cudaStream_t stream) {
  PE_REQUIRE(B >= 0 && B <= INT_MAX, "invalid batch");
  if (B == 0) return kOk;
  launch_kernel(inst_gather_kernel, (unsigned)B, 128, 0, stream, descs,
      FieldGather{fields, pc, scores, gc, crowd, areas});
  PE_LAUNCHED("inst_gather");
  count_launch();
  return kOk;
}

PE_API int pe_inst_prepare(const int64_t* descs, int64_t B, const uint64_t* pa_count, const uint64_t* ga_count,
                           double* pa, double* ga, const int32_t* pc, const int32_t* gc, const double* scores,
                           const double* ann_in, double* ann_out, int64_t C, int validate, uint32_t* class_bits,
                           int32_t* error, cudaStream_t stream) {
  PE_REQUIRE(B >= 0 && C > 0 && C < INT_MAX, "invalid batch");
  if (B == 0) return kOk;
  launch_kernel(inst_prepare_kernel, (unsigned)B, 128, 0, stream, descs, reinterpret_cast<const u64*>(pa_count),
      reinterpret_cast<const u64*>(ga_count), pa, ga, pc, gc, scores, ann_in, ann_out, (int)C, validate,
      reinterpret_cast<u32*>(class_bits), error);
  PE_LAUNCHED("inst_prepare");
  count_launch();
  return kOk;
}
