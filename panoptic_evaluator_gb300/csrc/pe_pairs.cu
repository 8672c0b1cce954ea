// Detection x target mask intersections by streaming, and the choice between
// that and the tensor-core contraction: the mask IoU counts of InstanceEvaluator.
//
// Every mask byte is read once (once per 63 targets for the detections), so HBM
// is the floor, and what has to stay under it is the work per byte. Masks are
// sparse: an object covers a few percent of its image, so of the 512 pixels that
// a warp looks at, most masks hold none, and a pair of masks rarely meets. A
// producer warp streams 4096-pixel segments of the rows (targets first, then the
// detections in score order) through a ring of shared-memory stages with
// cp.async.bulk; a consumer warp tests the four rows of a stage with one
// warp-wide OR (a superset: rows start at any byte, and the staged words are
// tested as they lie), re-aligns and packs only rows with a pixel, keeps the
// targets' bits in shared memory and intersects a detection with the targets
// that are present, by AND and popcount.
//
// The contraction (pe_contract.cu) multiplies every pair whatever it holds: its
// time does not depend on the masks, rows reach it at 5.0 TB/s by TMA and staged,
// and more than 127 detections or 63 targets are read again for every tile.
// Streaming reads at 6.3 TB/s while masks are sparse (us, 16 images of 640 x 640
// with 100 x 50 masks of 0.8 %: 129 against 163). With rectangles of 1, 3, 5 and
// 20 % of 641 x 639, and one lane producing as it did (5.4 TB/s): 16 images of
// 100 x 50 masks 184, 209, 247, 516 against 223 by contraction; 32 of 100 x 8:
// 264, 269, 293, 520 against 350; 6 of 300 x 100: 290, 394, 491, 1284 against 590.
// Which of the two a batch gets is decided on the device, from a sample of its
// masks (sample_image): both are launched, the other one returns at once.
#include "pe_bins.cuh"
#include "pe_common.cuh"
#include "pe_contract.cuh"
#include "pe_order.cuh"

namespace pe {
namespace {

constexpr int kPairChunk = 4096;     // pixels, as kChunkBegin counts them
constexpr int kPairStage = 4;        // mask rows per ring stage
constexpr int kPairUnitRing = 4;     // published units in flight per CTA
constexpr int kPairTargets = 63;     // targets whose bits a warp keeps at a time
constexpr int kPairParts = 8;        // parts of a chunk's detections, at most, where CTAs are left without a chunk
constexpr int kPartDets = 16;        // detections of a part, at least: it reads the targets again
constexpr int kPairWarps = 8;        // consumer warps, 512 pixels each
constexpr int kPairConsumers = kPairWarps * 32, kPairThreads = kPairConsumers + 32;
constexpr int kPairRow = kPairChunk + 16;  // the aligned words covering a row segment
constexpr int kPairRing = 4;         // stages in flight per CTA
constexpr long long kPairWaitLimit = 4000000000ll;  // about two seconds of SM clock
constexpr int kPairTimeoutBit = 1 << 30;

struct PairShared {
  unsigned char ring[kPairRing][kPairStage][kPairRow];
  uint16_t bits[kPairWarps][kPairTargets][32];
  __align__(4) unsigned char shift[kPairRing][kPairStage];  // each row's start offset mod 16
  unsigned char target[kPairWarps][kPairTargets];  // kept targets, relative to the group
  int64_t desc[kPairUnitRing][kDescFields];  // the image's descriptor
  int64_t x0[kPairUnitRing];                 // first pixel; -1 ends the CTA's work
  int dets[kPairUnitRing][2];                // detections [first, end); the first part counts the targets' areas
  uint64_t full[kPairRing];
  uint64_t empty[kPairRing];
  uint64_t unit_full[kPairUnitRing];
  uint64_t unit_empty[kPairUnitRing];
  int abort;
};

// The sample: kSampleWindows windows of 512 pixels per image, four words of each row in every window;
// kSampleParts CTAs per image.
constexpr int kSampleThreads = 256;
constexpr int kSampleWindows = 16;
constexpr int kPartWindows = kSampleWindows / kSampleParts;
constexpr int kZeroBlocks = 32;
// Picoseconds of the whole device per row of a warp's 512 pixels, per row with a pixel there, and per pair of them.
constexpr u64 kRowCost = 42, kHitCost = 280, kPairCost = 15;

struct PairSample {
  u64* costs;  // null: no estimate wanted
  u32* inter;
  int64_t inter_len;
  u64* pa;
  int64_t pa_len;
  u64* ga;
  int64_t ga_len;
  unsigned long long* schedule;
};

// Estimates what streaming the image would take where the masks' content decides: costs[kSampleParts * image + part],
// from the rows with pixels in a part's windows. The blocks behind those of the images clear the outputs and the
// chunk counter.
__device__ __forceinline__ void sample_image(const int64_t* descs, int64_t samples, int64_t block, const PairSample& a) {
  if (block >= samples) {
    const int64_t first = (block - samples) * kSampleThreads + threadIdx.x;
    constexpr int64_t kStep = kZeroBlocks * kSampleThreads;
    for (int64_t i = first; i < a.inter_len; i += kStep) a.inter[i] = 0;
    for (int64_t i = first; i < a.pa_len; i += kStep) a.pa[i] = 0;
    for (int64_t i = first; i < a.ga_len; i += kStep) a.ga[i] = 0;
    if (first == 0 && a.schedule) *a.schedule = 0;
    return;
  }
  const int64_t image = block / kSampleParts;
  __shared__ int present[2][kPartWindows];  // targets, detections with a pixel in the window
  if (threadIdx.x < 2 * kPartWindows) present[threadIdx.x / kPartWindows][threadIdx.x % kPartWindows] = 0;
  __syncthreads();
  const int64_t* d = desc_of(descs, image);
  const int64_t pixels = d[kPixels], stride = d[kMaskStride], G = d[kG], D = d[kD];
  if (pixels > 0) {
    const int mine = threadIdx.x % kPartWindows;
    const int64_t window = block % kSampleParts * kPartWindows + mine;
    // One window in each sixteenth of the image, at changing columns.
    const int64_t x0 = pixels * (16 * window + 5 * window % 16) / (16 * kSampleWindows);
#pragma unroll 2
    for (int64_t r = threadIdx.x / kPartWindows; r < G + D; r += kSampleThreads / kPartWindows) {
      const uint8_t* row = r < G ? reinterpret_cast<const uint8_t*>(d[kTarget]) + r * stride
                                 : reinterpret_cast<const uint8_t*>(d[kMasks]) + (r - G) * stride;
      u32 any = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {  // the aligned word that holds the pixel
        const uintptr_t p = reinterpret_cast<uintptr_t>(row + min(x0 + 165 * k, pixels - 1)) & ~uintptr_t{15};
        const uint4 w = __ldg(reinterpret_cast<const uint4*>(p));
        any |= w.x | w.y | w.z | w.w;
      }
      if (any) atomicAdd(&present[r >= G][mine], 1);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const u64 passes = (u64)max(ceil_div(G, kPairTargets), (int64_t)1);
    u64 sum = 0;
    for (int w = 0; w < kPartWindows; ++w) {
      const u64 g = (u64)present[0][w], dets = (u64)present[1][w];
      sum += kRowCost * (u64)(G + D * passes) + kHitCost * (g + dets * passes) + kPairCost * g * dets;
    }
    a.costs[block] = sum * (u64)ceil_div(pixels, 512) / kSampleWindows;
  }
}

__global__ void __launch_bounds__(kSampleThreads)
inst_sample_kernel(const int64_t* __restrict__ descs, int64_t samples, PairSample sample) {
  wait_for_earlier_kernels();
  sample_image(descs, samples, blockIdx.x, sample);
}

// All that comes before the masks are counted, in one launch: the first B blocks gather and sort an image's
// metadata, the others sample and clear. As kernels of their own these took 4.7, 6.4 and 11.2 us one after another
// for 32 images of 100 detections; together 15.6 (16 images 10.3, one 7.9 for 10.6).
static_assert(kSampleThreads == kSortThreads, "one block size for both kinds of work");
__global__ void __launch_bounds__(kSampleThreads)
inst_begin_kernel(const int64_t* __restrict__ descs, int64_t B, FieldGather fields, ScoreOrder order, int64_t samples,
                  PairSample sample, int C, u32* class_bits) {
  wait_for_earlier_kernels();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (blockIdx.x >= B) {
    sample_image(descs, samples, blockIdx.x - B, sample);
    return;
  }
  const int64_t* d = desc_of(descs, blockIdx.x);
  gather_image(d, blockIdx.x, fields);
  __syncthreads();
  if (class_bits) mark_classes(d, blockIdx.x, fields, C, class_bits);
  sort_image(d, order, smem_raw);
}

__global__ void __launch_bounds__(kPairThreads, 2)
inst_pairs_kernel(const int64_t* __restrict__ descs, int64_t B, int64_t whole, int64_t split, int parts, Choice choice,
                  unsigned long long* __restrict__ schedule, const int64_t* __restrict__ order,
                  u32* __restrict__ inter, u64* __restrict__ pa, u64* __restrict__ ga, int* __restrict__ error) {
  wait_for_earlier_kernels();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PairShared& sm = *reinterpret_cast<PairShared*>(smem_raw);
  if (!streams(choice)) return;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kPairRing; ++i) {
      mbar_init(&sm.full[i], 1);
      mbar_init(&sm.empty[i], kPairWarps);
    }
    for (int i = 0; i < kPairUnitRing; ++i) {
      mbar_init(&sm.unit_full[i], 1);
      mbar_init(&sm.unit_empty[i], kPairWarps);
    }
    sm.abort = 0;
    mbar_fence_init();
  }
  __syncthreads();
  volatile int* abort = &sm.abort;

  if (threadIdx.x >= kPairConsumers) {
    // ---- producer ----------------------------------------------------------
    // By the whole warp, as in the fused pass (pe_segmentation.cu): 32 rows' addresses at once, a lane copies a row.
    // 32 COCO-like images: 242 -> 199 us, 6.3 TB/s.
    const int lane = threadIdx.x & 31;
    RingSlot<kPairRing> stage;
    RingSlot<kPairUnitRing> unit;
    int64_t sent = 0;
    unsigned long long claim = 0;
    bool ok = true, asked = false;
    auto ask = [&] {
      if (lane == 0) claim = atomicAdd(schedule, 1ull);
      asked = true;
    };
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, kPairWaitLimit) && !*abort) != 0;
    };
    auto publish = [&](int64_t word, int64_t x0, int first, int end) {
      if (!wait(&sm.unit_empty[unit.at], unit.phase ^ 1u)) return false;
      if (lane < kDescFields) sm.desc[unit.at][lane] = word;
      if (lane == 0) {
        sm.x0[unit.at] = x0;
        sm.dets[unit.at][0] = first;
        sm.dets[unit.at][1] = end;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.unit_full[unit.at]);  // release: the entry is visible with the phase
      unit.next();
      return true;
    };
    while (ok) {
      if (!asked) ask();
      int64_t chunk = (int64_t)__shfl_sync(0xffffffffu, claim, 0);  // whole ones, then each part of the others
      asked = false;
      if (chunk >= whole + split * parts) break;
      int part = 0, of = 1;
      if (chunk >= whole) {
        of = parts;
        part = (int)((chunk - whole) / split);
        chunk = whole + (chunk - whole) % split;
      }
      const int64_t b = find_row<kDescFields>(descs, B, kChunkBegin, chunk);
      const int64_t word = lane < kDescFields ? desc_of(descs, b)[lane] : 0;
      auto field = [&](int f) { return __shfl_sync(0xffffffffu, word, f); };
      const int64_t pixels = field(kPixels), stride = field(kMaskStride);
      const int64_t x0 = (chunk - field(kChunkBegin)) * (int64_t)kPairChunk;
      if (x0 >= pixels) continue;  // an image without pixels
      const int64_t len = min((int64_t)kPairChunk, pixels - x0);
      const int all = (int)field(kD), G = (int)field(kG);
      const int each = of == 1 ? all : max(kPartDets, (all + of - 1) / of);
      const int first = part * each, end = min(all, first + each), D = end - first;
      if (part > 0 && first >= all) continue;
      const uint8_t* pm = reinterpret_cast<const uint8_t*>(field(kMasks)) + x0;
      const uint8_t* gm = reinterpret_cast<const uint8_t*>(field(kTarget)) + x0;
      const int64_t* ord = order + field(kDetBegin) + first;
      if (!publish(word, x0, first, end)) {
        ok = false;
        break;
      }
      for (int g0 = 0; ok && (g0 == 0 || g0 < G); g0 += kPairTargets) {
        const int ng = min(kPairTargets, G - g0), rows = ng + D;
        // Row r of the group: target g0 + r, or the detection of rank r - ng.
        auto place_of = [&](int r) -> int64_t { return r < ng ? g0 + r : (r < rows ? ord[r - ng] : 0); };
        int64_t place = place_of(lane);
        for (int r32 = 0; ok && r32 < rows; r32 += 32) {
          const uint8_t* row = (r32 + lane < ng ? gm : pm) + place * stride;
          place = place_of(r32 + 32 + lane);
          for (int r0 = r32; r0 < min(r32 + 32, rows); r0 += kPairStage) {
            if (!wait(&sm.empty[stage.at], stage.phase ^ 1u)) {
              ok = false;
              break;
            }
            const uint64_t from = __shfl_sync(0xffffffffu, reinterpret_cast<uint64_t>(row), (r0 - r32 + lane) & 31);
            const bool mine = lane < min(kPairStage, rows - r0);
            const int o = (int)(from & 15);
            const uint32_t bytes = mine ? (uint32_t)round_up(len + o, 16) : 0u;
            if (mine) sm.shift[stage.at][lane] = (unsigned char)o;
            const uint32_t total = __reduce_add_sync(0xffffffffu, bytes);
            __syncwarp();
            if (lane == 0) mbar_arrive_expect_tx(&sm.full[stage.at], total);  // release: the offsets too
            __syncwarp();
            if (mine)
              bulk_copy_g2s(sm.ring[stage.at][lane], reinterpret_cast<const uint8_t*>(from) - o, bytes,
                            &sm.full[stage.at]);
            stage.next();
            ++sent;
            if (!asked && g0 + kPairTargets >= G && r0 + 2 * kPairStage >= rows) ask();
          }
        }
      }
    }
    if (ok) ok = publish(0, -1, 0, 0);
    if (!ok) {
      *abort = 1;
      if (lane == 0) atomicOr(error, kPairTimeoutBit);
    }
    for (int64_t q = sent > kPairRing ? sent - kPairRing : 0; q < sent; ++q)  // copies still in flight land first
      mbar_wait(&sm.full[q % kPairRing], (uint32_t)((q / kPairRing) & 1), kPairWaitLimit);
    return;
  }

  // ---- consumers -----------------------------------------------------------
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint16_t(*kept)[32] = sm.bits[warp];
  unsigned char* target = sm.target[warp];
  RingSlot<kPairRing> stage;
  RingSlot<kPairUnitRing> unit;
  bool ok = true;
  while (ok) {
    const bool ready = mbar_wait(&sm.unit_full[unit.at], unit.phase, kPairWaitLimit);
    if (!__all_sync(0xffffffffu, ready && !*abort)) {
      ok = false;
      break;
    }
    const int64_t* d = sm.desc[unit.at];
    const int64_t x0 = sm.x0[unit.at];
    if (x0 < 0) break;
    const int first = sm.dets[unit.at][0], D = sm.dets[unit.at][1] - first, G = (int)d[kG];
    const u32 inside = inside_bits(x0 + (int64_t)threadIdx.x * 16, d[kPixels]);
    u64* pa_img = pa + d[kDetBegin] + first;
    u64* ga_img = ga + d[kSlotBegin];
    u32* inter_img = inter + d[kDPairBegin] + (int64_t)first * G;
    __syncwarp();  // the entry is in registers
    if (lane == 0) mbar_arrive(&sm.unit_empty[unit.at]);
    unit.next();
    for (int g0 = 0; ok && (g0 == 0 || g0 < G); g0 += kPairTargets) {
      const int ng = min(kPairTargets, G - g0), rows = ng + D;
      int present = 0;  // targets of the group with pixels here (their bits in `kept`)
      u32 covered = 0;  // this lane's pixels under any of them
      for (int r0 = 0; r0 < rows; r0 += kPairStage) {
        const bool got = mbar_wait(&sm.full[stage.at], stage.phase, kPairWaitLimit);
        if (!__all_sync(0xffffffffu, got && !*abort)) {  // warp-uniform decision
          ok = false;
          break;
        }
        const unsigned char* staged = &sm.ring[stage.at][0][threadIdx.x * 16];
        const u32 shifts = *reinterpret_cast<const u32*>(sm.shift[stage.at]);
        u32 hit = 0, beyond = 0;
#pragma unroll
        for (int k = 0; k < kPairStage; ++k) {
          const uint4 w = *reinterpret_cast<const uint4*>(staged + k * kPairRow);
          hit |= (u32)((w.x | w.y | w.z | w.w) != 0) << k;
        }
        if (lane == 31 && shifts) {  // the warp's pixels end in the next word
#pragma unroll
          for (int k = 0; k < kPairStage; ++k) {
            const uint4 w = *reinterpret_cast<const uint4*>(staged + k * kPairRow + 16);
            beyond |= (u32)((w.x | w.y | w.z | w.w) != 0 && (shifts >> 8 * k & 15) != 0) << k;
          }
        }
        hit = __reduce_or_sync(0xffffffffu, hit | beyond) & ((1u << min(kPairStage, rows - r0)) - 1u);
#pragma unroll 1
        for (; hit; hit &= hit - 1) {
          const int k = __ffs(hit) - 1, r = r0 + k;
          // Packed as the words lie, then shifted: one shuffle and a bit shift instead of moving 16 bytes.
          const u32 bits = pack16(*reinterpret_cast<const uint4*>(staged + k * kPairRow));
          u32 next = __shfl_down_sync(0xffffffffu, bits, 1);
          if (lane == 31)
            next = beyond >> k & 1 ? pack16(*reinterpret_cast<const uint4*>(staged + k * kPairRow + 16)) : 0u;
          const u32 m = (bits | next << 16) >> (shifts >> 8 * k & 15) & inside;
          const u32 area = __reduce_add_sync(0xffffffffu, __popc(m));
          if (!area) continue;  // pixels of the neighbouring warp, or past the image
          if (r < ng) {
            if (lane == 0 && first == 0) atomicAdd(ga_img + g0 + r, (u64)area);
            kept[present][lane] = (uint16_t)m;
            target[present] = (unsigned char)r;
            covered |= m;
            ++present;
            continue;
          }
          if (g0 == 0 && lane == 0) atomicAdd(pa_img + (r - ng), (u64)area);
          if (!__any_sync(0xffffffffu, (m & covered) != 0)) continue;
          u32* out = inter_img + (int64_t)(r - ng) * G + g0;
          for (int s0 = 0; s0 < present; s0 += 32) {
            u32 mine = 0;  // of target s0 + lane
            for (int s = s0; s < min(s0 + 32, present); ++s) {
              const u32 count = __reduce_add_sync(0xffffffffu, __popc(m & kept[s][lane]));
              mine = lane == s - s0 ? count : mine;
            }
            if (mine) atomicAdd(out + target[s0 + lane], mine);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.empty[stage.at]);
        stage.next();
      }
    }
  }
  if (!ok) {
    *abort = 1;
    if (lane == 0) atomicOr(error, kPairTimeoutBit);
  }
}

}  // namespace
}  // namespace pe

using namespace pe;

// How long streaming a batch may take, in picoseconds by the sample's estimate (sample_image), to be faster than its
// contraction; 0: contract whatever the masks hold. Image b has dets[b] detection masks, gts[b] target masks and
// pixels[b] pixels; the fourth argument, the images that the contraction loads by TMA, is not read (they take as long
// as the others); sms: the device's SMs. Host side, no GPU work.
//
// Times, from 640 x 640 and 637 x 640 images with 100 x 8 and 100 x 50 masks of 0.8 % of the image: the contraction
// reads the rows of its tiles, with sixteen rows' worth of fixed work, at 5.6 TB/s, by TMA and staged; streaming reads
// the targets once and the detections once per 63 targets at 6.8 TB/s, or takes the estimate if that is longer, and
// its last chunks, the sample and the second launch take 14 us. Updates of 16 images 222 us contracted and 198
// streamed, of 8 135 and 130 (100 x 8) or 136 and 139 (100 x 50), of 4 92 and 98, with 7 us of them for the sample
// that no longer show (inst_begin_kernel).
PE_API int64_t pe_stream_limit(const int64_t* dets, const int64_t* gts, const int64_t* pixels,
                               const uint8_t* /*tma*/, int64_t B, int64_t sms) {
  PE_REQUIRE(B >= 0 && (B == 0 || (dets && gts && pixels)) && sms > 0, "invalid arguments");
  constexpr double kContracted = 5.6, kStreamed = 6.8, kFixed = 14e6;  // bytes per ps; ps
  constexpr int64_t kTileRows = 127, kTileCols = 63, kTileWork = 16;
  double contraction = 0.0, streamed = 0.0, chunks = 0.0;
  for (int64_t b = 0; b < B; ++b) {
    PE_REQUIRE(dets[b] >= 0 && gts[b] >= 0 && pixels[b] >= 0, "negative size for image %lld", (long long)b);
    const double m = (double)std::max<int64_t>(ceil_div(dets[b], kTileRows), 1);
    const double n = (double)std::max<int64_t>(ceil_div(gts[b], kTileCols), 1);
    const double D = (double)dets[b], G = (double)gts[b], P = (double)pixels[b];
    if (D + G == 0.0) continue;
    contraction += (D * n + G * m + kTileWork * m * n) * P / kContracted;
    streamed += (D * n + G) * P / kStreamed;
    chunks += std::ceil(P / kPairChunk);
  }
  // Fewer chunks than CTAs: measured while a chunk was the smallest share of the work, before the last ones went out
  // in parts (launch_counts), so batches of a few images stay with the contraction longer than they may have to.
  if (chunks > 0.0) streamed *= std::max(1.0, 2.0 * (double)sms / chunks);
  const double limit = contraction - kFixed;
  return streamed < limit ? (int64_t)std::min(limit, 9e18) : 0;
}

namespace {

bool valid_sample(int64_t B, int64_t inter_len, int64_t pa_len, int64_t ga_len) {
  return B >= 0 && B <= INT_MAX / (kSampleParts + 1) - kZeroBlocks && inter_len >= 0 && pa_len >= 0 && ga_len >= 0;
}

// `costs` and the chunk counter behind them: 8 B + 1 words.
PairSample pair_sample(uint64_t* work, int64_t B, uint32_t* inter, int64_t inter_len, uint64_t* pa, int64_t pa_len,
                       uint64_t* ga, int64_t ga_len) {
  return PairSample{reinterpret_cast<u64*>(work), inter, inter_len, reinterpret_cast<u64*>(pa), pa_len,
                    reinterpret_cast<u64*>(ga), ga_len,
                    work ? reinterpret_cast<unsigned long long*>(work + B * kSampleParts) : nullptr};
}

// Both ways, of which one works.
int launch_counts(const int64_t* descs, int64_t B, int64_t pair_chunks, const int64_t* blocks, int64_t n_blocks,
                  int64_t total_chunks, const int64_t* cta_bounds, int64_t ctas, const int64_t* order, uint32_t* inter,
                  uint64_t* pa, uint64_t* ga, const void* maps, int64_t limit, uint64_t* work, int32_t* error,
                  cudaStream_t stream) {
  const Choice choice{reinterpret_cast<const u64*>(work), B * kSampleParts, limit};
  const size_t smem = sizeof(PairShared);
  PE_CUDA(cudaFuncSetAttribute(inst_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // The chunks beyond the last full round in as many parts as that round has CTAs for: 32 COCO-like images (8 rounds)
  // 199 -> 194 us, 16 on a canvas (5.3) 128.5 -> 126.
  const int64_t slots = (int64_t)sm_count() * 2, whole = pair_chunks / slots * slots, split = pair_chunks - whole;
  const int64_t parts = split ? std::min<int64_t>(kPairParts, slots / split) : 1;
  const int64_t grid = std::min(whole + split * parts, slots);
  launch_kernel(inst_pairs_kernel, (unsigned)grid, kPairThreads, smem, stream, descs, B, whole, split, (int)parts, choice,
      reinterpret_cast<unsigned long long*>(work + B * kSampleParts), order, reinterpret_cast<u32*>(inter),
      reinterpret_cast<u64*>(pa), reinterpret_cast<u64*>(ga), error);
  PE_LAUNCHED("inst_pairs");
  count_launch();
  return launch_contract(descs, blocks, n_blocks, total_chunks, cta_bounds, ctas, order, inter, pa, ga, maps, choice,
                         error, stream);
}

}  // namespace

// pe_inst_gather and pe_seg_sort in one launch, which also clears the outputs of pe_inst_counts and, with a limit
// above 0, samples the masks for it (work: 8 B + 1 u64 of device scratch). class_bits (optional): the images' classes
// among C, for pe_inst_match.
PE_API int pe_inst_begin(const int64_t* descs, const int64_t* fields, int64_t B, int32_t* pc, double* scores,
                         int32_t* gc, uint8_t* crowd, double* areas, int64_t total_detections, int64_t* order,
                         double* sorted_scores, int32_t* sorted_classes, void* workspace, int64_t workspace_bytes,
                         uint32_t* inter, int64_t inter_len, uint64_t* pa, int64_t pa_len, uint64_t* ga,
                         int64_t ga_len, int64_t limit, uint64_t* work, int64_t C, uint32_t* class_bits,
                         cudaStream_t stream) {
  PE_REQUIRE(valid_sample(B, inter_len, pa_len, ga_len) && C >= 0 && C < INT_MAX && total_detections >= 0, "invalid batch");
  PE_REQUIRE(workspace_bytes >= pe_seg_sort_workspace(total_detections), "sort workspace too small");
  PE_REQUIRE(limit <= 0 || work, "a sample needs its scratch");
  const int64_t samples = limit > 0 ? B * kSampleParts : 0;
  const int64_t clearing = inter_len + pa_len + ga_len > 0 || samples ? kZeroBlocks : 0;
  if (B + clearing == 0) return kOk;
  const ScoreOrder out =
      score_order(scores, pc, total_detections, order, sorted_scores, sorted_classes, workspace);
  PE_CUDA(cudaFuncSetAttribute(inst_begin_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sort_bytes(kOrderCap)));
  launch_kernel(inst_begin_kernel, (unsigned)(B + samples + clearing), kSampleThreads, sort_bytes(out.cap), stream,
      descs, B, FieldGather{fields, pc, scores, gc, crowd, areas}, out, samples,
      pair_sample(samples ? work : nullptr, B, inter, inter_len, pa, pa_len, ga, ga_len), (int)C, class_bits);
  PE_LAUNCHED("inst_begin");
  count_launch();
  return kOk;
}

// The counts of pe_inst_contract into outputs that pe_inst_begin cleared, streamed where its sample stays within
// `limit` (0: contracted).
PE_API int pe_inst_counts(const int64_t* descs, int64_t B, int64_t pair_chunks, const int64_t* blocks,
                          int64_t n_blocks, int64_t total_chunks, const int64_t* cta_bounds, int64_t ctas,
                          const int64_t* order, uint32_t* inter, uint64_t* pa, uint64_t* ga, const void* maps,
                          int64_t limit, uint64_t* work, int32_t* error, cudaStream_t stream) {
  PE_REQUIRE(B >= 0 && pair_chunks >= 0 && n_blocks >= 0 && total_chunks >= 0 && (limit <= 0 || work), "invalid batch");
  PE_REQUIRE(n_blocks > 0 || total_chunks == 0, "chunks without blocks");
  PE_REQUIRE((reinterpret_cast<uintptr_t>(maps) & 63) == 0, "tensor maps must be 64-byte aligned");
  if (limit <= 0 || B == 0 || pair_chunks == 0)
    return launch_contract(descs, blocks, n_blocks, total_chunks, cta_bounds, ctas, order, inter, pa, ga, maps,
                           Choice{nullptr, 0, 0}, error, stream);
  return launch_counts(descs, B, pair_chunks, blocks, n_blocks, total_chunks, cta_bounds, ctas, order, inter, pa, ga,
                       maps, limit, work, error, stream);
}

// For callers that gather and sort by themselves (updates launch pe_inst_begin and pe_inst_counts):
// pe_inst_contract for a batch whose masks may be sparse: the same inputs, outputs and counts, streamed where
// pe_stream_limit's `limit` and a sample of the masks say that this is faster. pair_chunks: 4096-pixel chunks of
// the descriptor table (kChunkBegin); work: 8 B + 1 u64 of device scratch. Drop-in for the reference's
// pack_masks + overlap (instance_kernel.cu:10-39).
PE_API int pe_inst_intersect(const int64_t* descs, int64_t B, int64_t pair_chunks, const int64_t* blocks,
                             int64_t n_blocks, int64_t total_chunks, const int64_t* cta_bounds, int64_t ctas,
                             const int64_t* order, uint32_t* inter, int64_t inter_len, uint64_t* pa, int64_t pa_len,
                             uint64_t* ga, int64_t ga_len, const void* maps, int64_t limit, uint64_t* work,
                             int32_t* error, cudaStream_t stream) {
  PE_REQUIRE(valid_sample(B, inter_len, pa_len, ga_len) && pair_chunks >= 0 && work, "invalid batch");
  const int64_t samples = B * kSampleParts;
  launch_kernel(inst_sample_kernel, (unsigned)(samples + kZeroBlocks), kSampleThreads, 0, stream, descs, samples,
      pair_sample(work, B, inter, inter_len, pa, pa_len, ga, ga_len));
  PE_LAUNCHED("inst_sample");
  count_launch();
  if (B == 0 || pair_chunks == 0) return kOk;
  return launch_counts(descs, B, pair_chunks, blocks, n_blocks, total_chunks, cta_bounds, ctas, order, inter, pa, ga,
                       maps, limit, work, error, stream);
}
