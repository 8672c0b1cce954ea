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
// time does not depend on the masks. Rows on 16-byte boundaries reach it by TMA
// at 6.1 TB/s and stay there; rows at any byte offset move through shared memory
// four times (4.3 TB/s), and more than 127 detections or 63 targets are read again
// for every tile. There streaming is faster while masks are sparse (us, rectangles
// of 1, 3, 5 and 20 % of the image; 641 x 639): 16 images of 100 x 50 masks 184,
// 209, 247, 516 against 223 by contraction; 32 of 100 x 8: 264, 269, 293, 520
// against 350; 6 of 300 x 100: 290, 394, 491, 1284 against 590. 32 COCO-like images:
// 226 against 303, 5.4 TB/s. Which of the two a batch gets is decided on the device,
// from a sample of its masks (inst_sample_kernel): both are launched, the other one
// returns at once. The sample and the empty launch take 9 to 13 us.
#include "pe_bins.cuh"
#include "pe_common.cuh"
#include "pe_contract.cuh"
#include "pe_desc.cuh"

namespace pe {
namespace {

constexpr int kPairChunk = 4096;     // pixels, as kChunkBegin counts them
constexpr int kPairStage = 4;        // mask rows per ring stage
constexpr int kPairUnitRing = 4;     // published units in flight per CTA
constexpr int kPairTargets = 63;     // targets whose bits a warp keeps at a time
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

// Estimates what streaming the image would take where the masks' content decides: costs[kSampleParts * image + part],
// from the rows with pixels in a part's windows. The blocks behind clear the outputs and the chunk counter
// (a memset before).
__global__ void __launch_bounds__(kSampleThreads)
inst_sample_kernel(const int64_t* __restrict__ descs, int64_t B, u64* __restrict__ costs, u32* __restrict__ inter,
                   int64_t inter_len, u64* __restrict__ pa, int64_t pa_len, u64* __restrict__ ga, int64_t ga_len,
                   unsigned long long* __restrict__ schedule) {
  wait_for_earlier_kernels();
  const int64_t image = blockIdx.x / kSampleParts;
  if (image >= B) {
    const int64_t first = (blockIdx.x - B * kSampleParts) * kSampleThreads + threadIdx.x;
    constexpr int64_t kStep = kZeroBlocks * kSampleThreads;
    for (int64_t i = first; i < inter_len; i += kStep) inter[i] = 0;
    for (int64_t i = first; i < pa_len; i += kStep) pa[i] = 0;
    for (int64_t i = first; i < ga_len; i += kStep) ga[i] = 0;
    if (first == 0) *schedule = 0;
    return;
  }
  __shared__ int present[2][kPartWindows];  // targets, detections with a pixel in the window
  if (threadIdx.x < 2 * kPartWindows) present[threadIdx.x / kPartWindows][threadIdx.x % kPartWindows] = 0;
  __syncthreads();
  const int64_t* d = desc_of(descs, image);
  const int64_t pixels = d[kPixels], stride = d[kMaskStride], G = d[kG], D = d[kD];
  if (pixels > 0) {
    const int mine = threadIdx.x % kPartWindows;
    const int64_t window = blockIdx.x % kSampleParts * kPartWindows + mine;
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
    costs[blockIdx.x] = sum * (u64)ceil_div(pixels, 512) / kSampleWindows;
  }
}

__global__ void __launch_bounds__(kPairThreads, 2)
inst_pairs_kernel(const int64_t* __restrict__ descs, int64_t B, int64_t total_chunks, Choice choice,
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
    auto publish = [&](int64_t word, int64_t x0) {
      if (!wait(&sm.unit_empty[unit.at], unit.phase ^ 1u)) return false;
      if (lane < kDescFields) sm.desc[unit.at][lane] = word;
      if (lane == 0) sm.x0[unit.at] = x0;
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.unit_full[unit.at]);  // release: the entry is visible with the phase
      unit.next();
      return true;
    };
    while (ok) {
      if (!asked) ask();
      const int64_t chunk = (int64_t)__shfl_sync(0xffffffffu, claim, 0);
      asked = false;
      if (chunk >= total_chunks) break;
      const int64_t b = find_row<kDescFields>(descs, B, kChunkBegin, chunk);
      const int64_t word = lane < kDescFields ? desc_of(descs, b)[lane] : 0;
      auto field = [&](int f) { return __shfl_sync(0xffffffffu, word, f); };
      const int64_t pixels = field(kPixels), stride = field(kMaskStride);
      const int64_t x0 = (chunk - field(kChunkBegin)) * (int64_t)kPairChunk;
      if (x0 >= pixels) continue;  // an image without pixels
      const int64_t len = min((int64_t)kPairChunk, pixels - x0);
      const int D = (int)field(kD), G = (int)field(kG);
      const uint8_t* pm = reinterpret_cast<const uint8_t*>(field(kMasks)) + x0;
      const uint8_t* gm = reinterpret_cast<const uint8_t*>(field(kTarget)) + x0;
      const int64_t* ord = order + field(kDetBegin);
      if (!publish(word, x0)) {
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
    if (ok) ok = publish(0, -1);
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
    const int D = (int)d[kD], G = (int)d[kG];
    const u32 inside = inside_bits(x0 + (int64_t)threadIdx.x * 16, d[kPixels]);
    u64* pa_img = pa + d[kDetBegin];
    u64* ga_img = ga + d[kSlotBegin];
    u32* inter_img = inter + d[kDPairBegin];
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
            if (lane == 0) atomicAdd(ga_img + g0 + r, (u64)area);
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

// How long streaming a batch may take, in picoseconds by inst_sample_kernel's estimate, to be faster than its
// contraction; 0: contract whatever the masks hold. Image b has dets[b] detection masks, gts[b] target masks and
// pixels[b] pixels; tma (optional) marks the images that the contraction loads by TMA; sms: the device's SMs.
// Host side, no GPU work.
//
// Times, from 640 x 640 and 641 x 639 images with 100 x 8 to 300 x 100 masks: the contraction reads the rows of
// its tiles, with sixteen rows' worth of fixed work, at 4.75 TB/s staged and 6.6 TB/s by TMA; streaming reads the
// targets once and the detections once per 63 targets at 5.4 TB/s, or takes the estimate if that is longer. The
// sample and the second launch take 12 us.
PE_API int64_t pe_stream_limit(const int64_t* dets, const int64_t* gts, const int64_t* pixels, const uint8_t* tma,
                               int64_t B, int64_t sms) {
  PE_REQUIRE(B >= 0 && (B == 0 || (dets && gts && pixels)) && sms > 0, "invalid arguments");
  constexpr double kStaged = 4.75, kTma = 6.6, kStreamed = 5.4, kFixed = 12e6;  // bytes per ps; ps
  constexpr int64_t kTileRows = 127, kTileCols = 63, kTileWork = 16;
  double contraction = 0.0, streamed = 0.0, chunks = 0.0;
  for (int64_t b = 0; b < B; ++b) {
    PE_REQUIRE(dets[b] >= 0 && gts[b] >= 0 && pixels[b] >= 0, "negative size for image %lld", (long long)b);
    const double m = (double)std::max<int64_t>(ceil_div(dets[b], kTileRows), 1);
    const double n = (double)std::max<int64_t>(ceil_div(gts[b], kTileCols), 1);
    const double D = (double)dets[b], G = (double)gts[b], P = (double)pixels[b];
    if (D + G == 0.0) continue;
    contraction += (D * n + G * m + kTileWork * m * n) * P / (tma && tma[b] ? kTma : kStaged);
    streamed += (D * n + G) * P / kStreamed;
    chunks += std::ceil(P / kPairChunk);
  }
  const double slots = 2.0 * (double)sms;  // chunks in flight: a last wave that is nearly empty costs a whole one
  if (chunks > 0.0) streamed *= std::ceil(chunks / slots) * slots / chunks;
  const double limit = contraction - kFixed;
  return streamed < limit ? (int64_t)std::min(limit, 9e18) : 0;
}

// pe_inst_contract for a batch whose masks may be sparse: the same inputs, outputs and counts, streamed where
// pe_stream_limit's `limit` and a sample of the masks say that this is faster. pair_chunks: 4096-pixel chunks of
// the descriptor table (kChunkBegin); work: 8 B + 1 u64 of device scratch. Drop-in for the reference's
// pack_masks + overlap (instance_kernel.cu:10-39).
PE_API int pe_inst_intersect(const int64_t* descs, int64_t B, int64_t pair_chunks, const int64_t* blocks,
                             int64_t n_blocks, int64_t total_chunks, const int64_t* cta_bounds, int64_t ctas,
                             const int64_t* order, uint32_t* inter, int64_t inter_len, uint64_t* pa, int64_t pa_len,
                             uint64_t* ga, int64_t ga_len, const void* maps, int64_t limit, uint64_t* work,
                             int32_t* error, cudaStream_t stream) {
  PE_REQUIRE(B >= 0 && B <= INT_MAX / kSampleParts - kZeroBlocks && pair_chunks >= 0 && work, "invalid batch");
  PE_REQUIRE(inter_len >= 0 && pa_len >= 0 && ga_len >= 0, "invalid batch");
  u64* costs = reinterpret_cast<u64*>(work);
  unsigned long long* schedule = reinterpret_cast<unsigned long long*>(work + B * kSampleParts);
  launch_kernel(inst_sample_kernel, (unsigned)(B * kSampleParts + kZeroBlocks), kSampleThreads, 0, stream, descs, B,
      costs, reinterpret_cast<u32*>(inter), inter_len, reinterpret_cast<u64*>(pa), pa_len, reinterpret_cast<u64*>(ga),
      ga_len, schedule);
  PE_LAUNCHED("inst_sample");
  count_launch();
  if (B == 0 || pair_chunks == 0) return kOk;
  const Choice choice{costs, B * kSampleParts, limit};
  const size_t smem = sizeof(PairShared);
  PE_CUDA(cudaFuncSetAttribute(inst_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t grid = std::min(pair_chunks, (int64_t)sm_count() * 2);
  launch_kernel(inst_pairs_kernel, (unsigned)grid, kPairThreads, smem, stream, descs, B, pair_chunks, choice, schedule,
      order, reinterpret_cast<u32*>(inter), reinterpret_cast<u64*>(pa), reinterpret_cast<u64*>(ga), error);
  PE_LAUNCHED("inst_pairs");
  count_launch();
  return launch_contract(descs, blocks, n_blocks, total_chunks, cta_bounds, ctas, order, inter, pa, ga, maps, choice,
                         error, stream);
}
