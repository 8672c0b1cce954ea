// COCO mask AP/AR: detection x target-slot histograms, mask overlaps, greedy
// matching and 101-point precision/recall accumulation.
//
// Matching runs one CTA per (image, class): the class's detections (score
// order, top 100 ranked) and ground truths (metadata order) are compacted with
// ballots, every detection's candidate targets (IoU at least 0.5) are listed by
// falling IoU, one warp per detection, and then each of 40 threads owns one
// (area range x IoU threshold) chain and walks the detections through their
// candidate lists.
//
// Accumulation runs five or ten CTAs per class, each with two or one of the ten IoU
// thresholds: it gathers the class's records, sorts them by descending score,
// and one warp at a time builds a (threshold, area, maxDets) chain's precision
// envelope with integer comparisons only.
#include "pe_common.cuh"
#include "pe_sort.cuh"

#include <cfloat>

namespace pe {
namespace {

constexpr int kChains = 40;
constexpr int kMaxDets = 100;
constexpr int kMatchThreads = 256;  // threads of a matching CTA, half of them where CTAs are many

__device__ __forceinline__ void area_range(int a, double& lo, double& hi) {
  lo = a == 2 ? 1024.0 : (a == 3 ? 9216.0 : 0.0);
  hi = a == 1 ? 1024.0 : (a == 2 ? 9216.0 : 1e10);
}

__device__ __forceinline__ double iou_threshold(int t) {
  // instance.py:252 (0.8999999999999999 is the literal value, not 0.9).
  const double table[10] = {0.5, 0.55, 0.6, 0.65, 0.7, 0.75, 0.8, 0.85, 0.8999999999999999, 0.95};
  return table[t];
}

// Candidate entries of one class held at a time; a class with more lists one detection's at a time.
constexpr int kMatchList = 512;
__host__ __device__ inline int match_entries(int g_max) { return g_max > kMatchList ? g_max : kMatchList; }

// A detection of the class: its entries [first, first + length), its index in the image, bit a: its area is inside
// range a.
struct __align__(16) MatchRecord {
  int first, length, det;
  u32 ranges;
};

// Shared memory of one matching CTA for up to g_max targets per image: the class's detections, candidate IoUs and
// targets, 40 chains' taken bits, the class's targets.
__host__ __device__ inline size_t match_bytes(int g_max) {
  const int words = (g_max + 31) / 32;
  return sizeof(MatchRecord) * kMaxDets + (sizeof(long long) + sizeof(uint32_t)) * (size_t)match_entries(g_max) +
         sizeof(uint32_t) * kChains * (size_t)words + sizeof(uint16_t) * (size_t)g_max + (size_t)g_max + 16;
}

struct FlagLayout {
  int8_t* base;         // flags of image 0
  int64_t chain_stride;  // distance between chains
  int64_t det_stride;    // distance between detections
};

// ---- greedy matching ------------------------------------------------------

// The class of the n-th (0-based) set bit of row[0, words), or -1 when fewer
// bits are set; every lane of the warp gets the same answer.
__device__ __forceinline__ int nth_present_class(const u32* __restrict__ row, int words, int n, int lane) {
  for (int w0 = 0; w0 < words; w0 += 32) {
    const int w = w0 + lane;
    const u32 v = w < words ? row[w] : 0u;
    const int cnt = __popc(v);
    int incl = cnt;  // inclusive scan of the set bits over the lanes' words
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    if (n < total) {
      const int src = __ffs(__ballot_sync(0xffffffffu, incl > n)) - 1;  // the word holding bit n
      const int before = __shfl_sync(0xffffffffu, incl - cnt, src);
      u32 word = __shfl_sync(0xffffffffu, v, src);
      for (int k = n - before; k > 0; --k) word &= word - 1;  // drop the lower set bits
      return (w0 + src) * 32 + __ffs(word) - 1;
    }
    n -= total;
  }
  return -1;
}

// What bounds a class is the chain over its detections, so everything that does
// not depend on earlier matches is done before it and in parallel: IoUs (FP64
// division runs at 1/64 of the FP32 rate, and only pairs that can reach 0.5 are
// divided), candidates sorted by falling IoU, later targets first on ties, each
// with its crowd and area-ignored bits. A chain's step is then a walk to the
// first usable entry, usually one or two shared reads. 32 COCO-like images of
// 100 detections: 21.8 us against 50.7 with one warp per class that divided and
// balloted inside the chain; 8 images of 256 detections 27.4 against 153. The
// longest class sets the time, so a warp lists as many detections at a time as
// it has lanes for their targets, eight warps list, and a chain's records and
// first entries are read ahead of it: 16 images on a canvas 24.0 -> 14.1 us, 32
// COCO-like ones 21.9 -> 17.7, 8 of 256 detections 31.4 -> 22.2.
// Area: double, or the pixel counts themselves; areas == nullptr: the targets' own.
template <typename Count, typename Area>
__global__ void __launch_bounds__(kMatchThreads, 5)
match_kernel(const Count* __restrict__ pairs, const int64_t* __restrict__ pair_off,
             const int64_t* __restrict__ d_off, const int64_t* __restrict__ g_off, int single_d, int single_g,
             const int* __restrict__ pc, const Area* __restrict__ pa,
             const int* __restrict__ gc, const Area* __restrict__ ga, const uint8_t* __restrict__ crowd,
             const double* __restrict__ areas, int C, int g_max, FlagLayout flags, int* __restrict__ ranks,
             int64_t* __restrict__ counts, const int* __restrict__ gate,
             const u32* __restrict__ class_bits, int unchecked) {
  wait_for_earlier_kernels();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int stopped = gate ? *reinterpret_cast<const volatile int*>(gate) : 0;
  if (stopped) {  // validation failed upstream, or a kernel gave up: an unchecked caller counts these records all the same
    if (blockIdx.y || blockIdx.z) return;
    const int64_t d_begin = d_off ? d_off[blockIdx.x] : 0, d_end = d_off ? d_off[blockIdx.x + 1] : single_d;
    for (int64_t i = d_begin + threadIdx.x; i < d_end; i += blockDim.x) {
      ranks[i] = 0;
      for (int k = 0; k < kChains; ++k) flags.base[k * flags.chain_stride + i * flags.det_stride] = -1;
    }
    if (blockIdx.x == 0 && (stopped & kStoppedBits) && (unchecked || (stopped & kUncheckedBit)))
      for (int k = threadIdx.x; k < 4 * C; k += blockDim.x) counts[k] = kUnknownCount;
    return;
  }
  // Image b covers detections [d_off[b], d_off[b+1]) and targets [g_off[b], g_off[b+1]);
  // its D x G intersections start at pair_off[b]. Without offsets: one image. CTA (b, k) takes the k-th
  // class of image b: of all classes, or with per-image class bits of those present in it (about a third
  // in COCO-like batches), so that the CTAs left without a class come last.
  const int b = (int)blockIdx.x, entry = (int)(blockIdx.y + gridDim.y * blockIdx.z);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = (int)(blockDim.x >> 5);
  const int bit_words = (C + 31) / 32;
  const int c = class_bits ? nth_present_class(class_bits + (int64_t)b * bit_words, bit_words, entry, lane) : entry;
  if (c < 0 || c >= C) return;
  const int64_t d0 = d_off ? d_off[b] : 0, g0 = g_off ? g_off[b] : 0;
  const int D = d_off ? (int)(d_off[b + 1] - d0) : single_d;
  const int G = g_off ? (int)(g_off[b + 1] - g0) : single_g;
  const Count* P = pairs + (pair_off ? pair_off[b] : 0);
  pc += d0; pa += d0; ranks += d0;
  gc += g0; ga += g0; crowd += g0;
  if (areas) areas += g0;
  int8_t* fbase = flags.base + d0 * flags.det_stride;
  const int words = (g_max + 31) / 32, capacity = match_entries(g_max);
  // IoUs as IEEE bit patterns: for non-negative doubles the int64 order is the
  // numeric order, so lists and chains compare integers only.
  MatchRecord* recs = reinterpret_cast<MatchRecord*>(smem_raw);
  long long* iou_s = reinterpret_cast<long long*>(recs + kMaxDets);
  u32* cand = reinterpret_cast<u32*>(iou_s + capacity);  // target j | ignored-in-range bits << 16 | crowd << 20
  u32* used = cand + capacity;
  uint16_t* gts = reinterpret_cast<uint16_t*>(used + kChains * words);
  uint8_t* target_bits = reinterpret_cast<uint8_t*>(gts + g_max);  // bits 0-3: ignored in range a, bit 4: crowd
  __shared__ int s_nd, s_ng, s_total;
  const u32 below = (1u << lane) - 1;
  constexpr int kScanBlocks = 4;  // blocks of 32 whose loads a lane issues before the ballots use them
  if (warp == 0) {
    // Every detection's rank and flags are written by exactly one CTA: that of its class (beyond the
    // 100-detection cap: rank 0, all flags -1), or that of class 0 for classes outside [0, C).
    int nd = 0;
    for (int group = 0; group < D; group += 32 * kScanBlocks) {
      int dcs[kScanBlocks];
#pragma unroll
      for (int u = 0; u < kScanBlocks; ++u) {
        const int d = group + 32 * u + lane;
        dcs[u] = d < D ? pc[d] : -1;
      }
#pragma unroll
      for (int u = 0; u < kScanBlocks; ++u) {
        const int d = group + 32 * u + lane;
        const bool sel = d < D && dcs[u] == c;
        const u32 ballot = __ballot_sync(0xffffffffu, sel);
        bool unranked = c == 0 && d < D && (dcs[u] < 0 || dcs[u] >= C);
        if (sel) {
          const int rank = nd + __popc(ballot & below);
          if (rank < kMaxDets) {
            recs[rank].det = d;
            ranks[d] = rank + 1;
          } else {
            unranked = true;
          }
        }
        if (unranked) {
          ranks[d] = 0;
          for (int k = 0; k < kChains; ++k) fbase[k * flags.chain_stride + (int64_t)d * flags.det_stride] = -1;
        }
        nd += __popc(ballot);
      }
    }
    if (lane == 0) s_nd = min(nd, kMaxDets);
  } else if (warp == 1) {
    int ng = 0;
    for (int group = 0; group < G; group += 32 * kScanBlocks) {
      int gcs[kScanBlocks];
#pragma unroll
      for (int u = 0; u < kScanBlocks; ++u) {
        const int g = group + 32 * u + lane;
        gcs[u] = g < G ? gc[g] : -1;
      }
#pragma unroll
      for (int u = 0; u < kScanBlocks; ++u) {
        const u32 ballot = __ballot_sync(0xffffffffu, gcs[u] == c);
        if (gcs[u] == c) gts[ng + __popc(ballot & below)] = (uint16_t)(group + 32 * u + lane);
        ng += __popc(ballot);
      }
    }
    if (lane == 0) s_ng = ng;
  } else {
    for (int k = threadIdx.x - 64; k < kChains * words; k += blockDim.x - 64) used[k] = 0;
    if (threadIdx.x == 64) s_total = 0;
  }
  __syncthreads();
  const int nd = s_nd, ng = s_ng;
  // The targets' bits and the class's counts, all targets at once: inside the scan above, one block of 32 after
  // another, their loads and FP64 comparisons made 22.2 us 25.6 at 257 targets.
  for (int j0 = warp * 32; j0 < ng; j0 += (int)blockDim.x) {
    const int j = j0 + lane;
    int positive[4] = {0, 0, 0, 0};
    if (j < ng) {
      const int g = gts[j];
      const bool cr = crowd[g] != 0;
      const double area = areas ? areas[g] : (double)ga[g];
      u32 bits = (u32)cr << 4;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        double lo, hi;
        area_range(a, lo, hi);
        const bool out = area < lo || area > hi;
        bits |= (u32)(cr || out) << a;
        positive[a] = !cr && area >= lo && area <= hi;
      }
      target_bits[j] = (uint8_t)bits;
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int n = __popc(__ballot_sync(0xffffffffu, positive[a]));
      if (lane == 0 && n) atomicAdd(reinterpret_cast<u64*>(counts) + c * 4 + a, (u64)n);
    }
  }
  if (nd == 0) return;
  for (int i = threadIdx.x; i < nd; i += blockDim.x) {
    const double dpa = (double)pa[recs[i].det];
    u32 bits = 0;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      double lo, hi;
      area_range(a, lo, hi);
      bits |= (u32)(lo <= dpa && dpa <= hi) << a;
    }
    recs[i].ranges = bits;
  }
  __syncthreads();
  // Candidates of detection i into entries [at, at + n), sorted; `at` from the shared counter, or 0 for
  // one detection at a time. Entries past the capacity are counted, not stored. One warp.
  const long long lowest = __double_as_longlong(0.5);
  auto iou_between = [&](int d, int j) -> long long {
    const int g = gts[j];
    const double inter = (double)P[(int64_t)d * G + g], pa_d = (double)pa[d], ga_g = (double)ga[g];
    if (!(inter > 0.0)) return -1;
    const double uni = fmax((target_bits[j] & 16) ? pa_d : (pa_d + ga_g) - inter, 1.0);
    if (inter * 2.001 < uni) return -1;  // clearly under the lowest threshold: no division
    return __double_as_longlong(inter / uni);
  };
  auto list_candidates = [&](int i, bool alone) {
    const int d = recs[i].det;
    auto iou_of = [&](int j) -> long long { return j < ng ? iou_between(d, j) : -1; };
    const long long own = iou_of(lane);  // up to 32 targets: one evaluation serves both passes
    int n = __popc(__ballot_sync(0xffffffffu, own >= lowest)), at = 0;
    for (int j0 = 32; j0 < ng; j0 += 32) n += __popc(__ballot_sync(0xffffffffu, iou_of(j0 + lane) >= lowest));
    if (n && !alone) {
      if (lane == 0) at = atomicAdd(&s_total, n);
      at = __shfl_sync(0xffffffffu, at, 0);
    }
    for (int j0 = 0, k = at; k < at + n; j0 += 32) {
      const long long iou = j0 ? iou_of(j0 + lane) : own;
      const u32 ballot = __ballot_sync(0xffffffffu, iou >= lowest);
      const int e = k + __popc(ballot & below);
      if (iou >= lowest && e < capacity) {
        iou_s[e] = iou;
        cand[e] = (u32)(j0 + lane) | (u32)target_bits[j0 + lane] << 16;
      }
      k += __popc(ballot);
    }
    if (lane == 0) {
      recs[i].first = at;
      recs[i].length = n;
    }
    __syncwarp();
    if (n < 2 || at + n > capacity) return;
    // Falling IoU, later targets first on ties (entries were stored by rising target).
    if (n <= 32) {
      const long long v = lane < n ? iou_s[at + lane] : -1;
      const u32 w = lane < n ? cand[at + lane] : 0;
      int rank = 0;
      for (int k = 0; k < n; ++k) {
        const long long o = __shfl_sync(0xffffffffu, v, k);
        rank += o > v || (o == v && k > lane);
      }
      __syncwarp();
      if (lane < n) {
        iou_s[at + rank] = v;
        cand[at + rank] = w;
      }
    } else {  // odd-even transposition: many near-identical masks
      for (int phase = 0; phase < n; ++phase) {
        for (int k = (phase & 1) + 2 * lane; k + 1 < n; k += 64) {
          const long long x = iou_s[at + k], y = iou_s[at + k + 1];
          const u32 jx = cand[at + k], jy = cand[at + k + 1];
          if (x < y || (x == y && (jx & 0xffffu) < (jy & 0xffffu))) {
            iou_s[at + k] = y; iou_s[at + k + 1] = x;
            cand[at + k] = jy; cand[at + k + 1] = jx;
          }
        }
        __syncwarp();
      }
    }
    __syncwarp();
  };
  // The same for up to 32 targets: 32 / width detections i0, i0 + 1, ... at a time, `width` lanes each.
  const int width = ng <= 1 ? 1 : 1 << (32 - __clz(ng - 1));
  auto list_some = [&](int i0) {
    const int j = lane & (width - 1), group = lane - j, i = i0 + group / width;
    const bool valid = i < nd && j < ng;
    const long long iou = valid ? iou_between(recs[i].det, j) : -1;
    const u32 all = __ballot_sync(0xffffffffu, iou >= lowest);
    const u32 mine = (all >> group) & (width < 32 ? (1u << width) - 1u : 0xffffffffu);
    int at = 0;
    if (lane == 0 && all) at = atomicAdd(&s_total, __popc(all));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(all & ((1u << group) - 1u));
    const int n = __popc(mine), own = __popc(mine & ((1u << j) - 1u));
    const bool listed = iou >= lowest && at + n <= capacity;
    if (listed) iou_s[at + own] = iou;
    __syncwarp();
    int rank = 0;  // falling IoU, later targets first on ties
    for (int k = 0; listed && k < n; ++k) {
      const long long o = iou_s[at + k];
      rank += o > iou || (o == iou && k > own);
    }
    __syncwarp();
    if (listed) {
      iou_s[at + rank] = iou;
      cand[at + rank] = (u32)j | (u32)target_bits[j] << 16;
    }
    if (j == 0 && i < nd) {
      recs[i].first = at;
      recs[i].length = n;
    }
  };
  // One detection of one chain: eligible targets before ignored ones, the largest IoU, the later target
  // on ties (a taken target is skipped unless it is a crowd). `iou` and `w` are the detection's first entry,
  // `bits` the targets taken where they fit a word.
  const int chain = threadIdx.x, a = chain / 10;
  const long long thr = chain < kChains ? __double_as_longlong(iou_threshold(chain % 10)) : 0;
  u32* taken = used + chain * words;
  const bool in_word = ng <= 32;
  u32 bits = 0;
  auto step = [&](const MatchRecord& r, long long iou, u32 w) {
    int best = -1, ignored = -1;
    for (int e = r.first, end = r.first + r.length; e < end;) {
      if (iou < thr) break;
      const int j = (int)(w & 0xffffu);
      const u32 word = in_word ? bits : taken[j >> 5];
      if (((w >> 20) & 1u) || !((word >> (j & 31)) & 1u)) {
        if (!((w >> (16 + a)) & 1u)) {
          best = j;
          break;
        }
        if (ignored < 0) ignored = j;
      }
      if (++e < end) {
        iou = iou_s[e];
        w = cand[e];
      }
    }
    int8_t flag = best >= 0 ? 1 : -1;
    if (best < 0) best = ignored;
    if (best >= 0) {
      if (in_word) bits |= 1u << best;
      else taken[best >> 5] |= 1u << (best & 31);
    } else if ((r.ranges >> a) & 1) {
      flag = 0;
    }
    fbase[chain * flags.chain_stride + (int64_t)r.det * flags.det_stride] = flag;
  };
  if (ng <= 32)
    for (int i = warp * (32 / width); i < nd; i += warps * (32 / width)) list_some(i);
  else
    for (int i = warp; i < nd; i += warps) list_candidates(i, false);
  __syncthreads();
  if (s_total <= capacity) {
    if (chain >= kChains) return;
    // Two records and one first entry ahead of the chain. The last detections read the last one's again.
    MatchRecord now = recs[0], next = recs[min(1, nd - 1)];
    long long iou = iou_s[now.first];
    u32 w = cand[now.first];
    for (int i = 0; i < nd; ++i) {
      const MatchRecord after = recs[min(i + 2, nd - 1)];
      const long long iou_next = iou_s[next.first];
      const u32 w_next = cand[next.first];
      step(now, iou, w);
      now = next;
      next = after;
      iou = iou_next;
      w = w_next;
    }
    return;
  }
  for (int i = 0; i < nd; ++i) {  // more candidates than the list holds: one detection at a time
    if (warp == 0) list_candidates(i, true);
    __syncthreads();
    if (chain < kChains) step(recs[i], iou_s[recs[i].first], cand[recs[i].first]);
    __syncthreads();
  }
}

// ---- precision / recall accumulation -------------------------------------

constexpr int kAccThreads = 256;
constexpr int kSortCap = 1024;  // records of one class sorted and staged in shared memory, at most
constexpr int kSmallCap = 512;  // classes up to this many records: a smaller stage, more CTAs per SM
// IoU thresholds of one CTA: two, or one while that leaves SMs without a CTA. A CTA has twelve (threshold, area,
// maxDets) chains of each.
constexpr int kAccT = 2;
// Records up to which every CTA scans the class array itself; above, three kernels group the records by
// class first (at 3200 records and 80 classes they and their memset took 8 us of the stream).
constexpr int64_t kScanRecords = 8192;

__global__ void class_histogram_kernel(const int* __restrict__ classes, int64_t n, int C, int* __restrict__ hist) {
  wait_for_earlier_kernels();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = classes[i];
    if (c >= 0 && c < C) atomicAdd(hist + c, 1);
  }
}

// Exclusive scan of the class histogram into `cursor` (one CTA): cursor[c] is
// where class c's record indices start in the per-class list.
__global__ void __launch_bounds__(1024) class_offsets_kernel(const int* __restrict__ hist, int C, int* cursor) {
  wait_for_earlier_kernels();
  __shared__ int s_warp[32];
  const int per = (C + blockDim.x - 1) / blockDim.x;
  const int c0 = min(C, (int)threadIdx.x * per), c1 = min(C, c0 + per);
  int local = 0;
  for (int c = c0; c < c1; ++c) local += hist[c];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inclusive = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inclusive, o);
    if (lane >= o) inclusive += v;
  }
  if (lane == 31) s_warp[warp] = inclusive;
  __syncthreads();
  if (warp == 0) {
    int w = lane < (int)(blockDim.x >> 5) ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += v;
    }
    s_warp[lane] = w;  // inclusive over warps
  }
  __syncthreads();
  int running = inclusive - local + (warp ? s_warp[warp - 1] : 0);
  for (int c = c0; c < c1; ++c) {
    cursor[c] = running;
    running += hist[c];
  }
}

// Record indices grouped by class (order inside a class is arbitrary: the
// accumulation sorts each class by score, then record index).
__global__ void class_scatter_kernel(const int* __restrict__ classes, int64_t n, int C, int* cursor,
                                     int* __restrict__ list) {
  wait_for_earlier_kernels();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = classes[i];
    if (c >= 0 && c < C) list[atomicAdd(cursor + c, 1)] = (int)i;
  }
}

// Recall thresholds r at which the quotient r / 100 reaches the threshold fl(r * 0.01) (the product can
// round above it), as bits.
struct RecallBits {
  u64 lo, hi;
};
constexpr RecallBits recall_bits() {
  RecallBits b{0, 0};
  for (int r = 0; r <= 100; ++r)
    if ((double)r / 100.0 >= (double)r * 0.01) (r < 64 ? b.lo : b.hi) |= 1ull << (r & 63);
  return b;
}

// The smallest true-positive count t whose recall fl(t / np) reaches fl(r * 0.01). t / np and r / 100
// are equal or at least 1 / (100 np) apart, far more than the rounding of either side, so the exact
// integer comparison decides except where they are equal, and there the bit of r does.
__device__ __forceinline__ int64_t recall_reached_at(int64_t np, int r) {
  constexpr RecallBits bits = recall_bits();
  const int64_t scaled = np * r, t = (scaled + 99) / 100;
  const bool exact_ok = ((r < 64 ? bits.lo : bits.hi) >> (r & 63)) & 1ull;
  return t + (t * 100 == scaled && !exact_ok ? 1 : 0);
}

// 10 / kT CTAs per class. `scores` == nullptr means the records are already in
// global descending-score order. Records: classes[n], ranks[n] and flags at
// flags[chain * chain_stride + record * det_stride]; list / cursor / hist: the
// records grouped by class, or list == nullptr and every CTA scans `classes`.
// Classes with more than kSortCap records use per-class workspace regions (and
// one CTA, since the sort works in place there) instead of shared memory.
//
// A chain is handled by one warp at a time. Prefix counts of true and false
// positives over the score-ordered records come from ballots; the j-th true
// positive's cumulative false positives are kept per j. The precision envelope
// of the reference (the running maximum of precision from the end,
// instance.py:321) is a suffix maximum over j, taken with a warp scan; recall
// threshold r is first reached at the true positive j = tp_min[r], so
// precision[r] is the envelope at that j (instance.py:322-329). Runs of
// thresholds with the same envelope pair become segments. FP64 (1/64 of the FP32
// rate here) is spent only with full warps: every lane divides a different
// segment, then one warp sums all chains, a lane per chain. A CTA holds all
// twelve (area, maxDets) chains of its thresholds, so the precision array is
// written in 96-byte runs (one chain at a time wrote single 8-byte words, four
// times the sectors). chain_stats [c][chain] receives the sum of the chain's 101
// precision values and its recall (-1 when the class has no positives) for the
// summaries. 3200 records of 80 classes: 17.9 us (43.2, after 8 us of grouping
// kernels, with all 120 chains walked by four CTAs and FP64 recall thresholds);
// 100 records 10.5 (26.9).
template <int kCap, int kT>
struct AccShared {
  static constexpr int kChainsHere = 12 * kT;
  unsigned long long key[kCap];
  int idx[kCap];
  int rank[kCap];
  int8_t flags[kCap][4 * kT];  // the staged records' flags of this CTA's thresholds, [t][area]
  long long seg[kChainsHere][101];   // packed (tp, fp) of a segment, then its value
  unsigned char seg_lo[kChainsHere][101 + 3];
  unsigned short env[kAccThreads / 32][2][kCap + 1];
  int tp_min[4][101];
  int nseg[kChainsHere], hi[kChainsHere], tp[kChainsHere], off[kChainsHere + 1];
  int64_t npos[4];
  double none[4];  // precision where the curve has none: 0, or -1 without positives, NaN with kUnknownCount
  int count, before;
};

template <int kCap, int kT>
__global__ void __launch_bounds__(kAccThreads)
accumulate_kernel(const int* __restrict__ classes, int64_t n, const int* __restrict__ list,
                  const int* __restrict__ cursor, int* __restrict__ hist, const int* __restrict__ ranks,
                  const int8_t* __restrict__ flags, int64_t chain_stride, int64_t det_stride,
                  const double* __restrict__ scores, const int64_t* __restrict__ positives,
                  unsigned long long* __restrict__ ws_key, int* __restrict__ ws_idx,
                  int C, int* __restrict__ env_ws, double* __restrict__ precision,
                  double* __restrict__ recall, double* __restrict__ chain_stats, int above) {
  wait_for_earlier_kernels();
  constexpr int kParts = 10 / kT, kChainsHere = 12 * kT;
  // The bitonic sort pads a class's records to the next power of two inside the kCap-entry stage.
  static_assert(kCap > 0 && (kCap & (kCap - 1)) == 0, "a stage cap must be a power of two");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  AccShared<kCap, kT>& sm = *reinterpret_cast<AccShared<kCap, kT>*>(smem_raw);
  const int c = blockIdx.x / kParts, part = blockIdx.x % kParts;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = kAccThreads / 32;
  const unsigned below = (1u << lane) - 1u;
  // The second launch reads the count that the first one found: usually it has nothing to do (5.3 -> 3.0 us).
  if (above >= 0 && hist[c] <= above) return;
  if (threadIdx.x < 4) {
    const int64_t np = positives[c * 4 + threadIdx.x];
    sm.npos[threadIdx.x] = np;
    sm.none[threadIdx.x] = np > 0 ? 0.0 : (np < 0 ? __longlong_as_double(0x7ff8000000000000ll) : -1.0);
  }
  // Records of this class, and of the classes before it (where its workspace regions start).
  int count, before;
  if (list) {
    count = hist[c];
    before = cursor[c] - count;  // cursor[c] ends one past the class's segment after the scatter
  } else {
    if (threadIdx.x == 0) sm.count = sm.before = 0;
    __syncthreads();
    int lower = 0;
    constexpr int kLoads = 4;
    for (int64_t i0 = threadIdx.x; i0 < n; i0 += kLoads * kAccThreads) {
      int v[kLoads];
#pragma unroll
      for (int j = 0; j < kLoads; ++j) v[j] = i0 + j * kAccThreads < n ? classes[i0 + j * kAccThreads] : -1;
#pragma unroll
      for (int j = 0; j < kLoads; ++j) {
        lower += v[j] >= 0 && v[j] < c;
        if (v[j] != c) continue;
        const int at = atomicAdd(&sm.count, 1);
        if (at < kCap) sm.idx[at] = (int)(i0 + j * kAccThreads);
      }
    }
    if (lower) atomicAdd(&sm.before, lower);
    __syncthreads();
    count = sm.count;
    before = sm.before;
    if (above < 0 && part == 0 && threadIdx.x == 0) hist[c] = count;
  }
  // Classes of up to kCap records (more than `above`) are this launch's: the other launch takes the rest.
  if (count <= above || (kCap < kSortCap && count > kCap)) return;
  const bool staged = count <= kCap;
  const int parts = staged ? kParts : 1;
  if (part >= parts) return;
  int padded = 1;
  while (padded < max(count, 1)) padded <<= 1;
  unsigned long long* key = staged ? sm.key : ws_key + 2 * (int64_t)before;
  int* idx = staged ? sm.idx : ws_idx + 2 * (int64_t)before;
  if (!list && !staged) {  // more records than the stage: the scan again, into the workspace
    __syncthreads();
    if (threadIdx.x == 0) sm.count = 0;
    __syncthreads();
    for (int64_t i = threadIdx.x; i < n; i += kAccThreads)
      if (classes[i] == c) idx[atomicAdd(&sm.count, 1)] = (int)i;
    __syncthreads();
  }
  // Sorted by (score desc, index asc); without scores every key is equal and the sort restores record order.
  for (int k = threadIdx.x; k < count; k += kAccThreads) {
    const int i = list ? list[before + k] : idx[k];
    idx[k] = i;
    key[k] = score_key(scores ? scores[i] : 0.0);
  }
  for (int e = threadIdx.x; e < 4 * 101; e += kAccThreads) {
    const int a = e / 101, r = e % 101;
    sm.tp_min[a][r] = (int)recall_reached_at(positives[c * 4 + a], r);
  }
  __syncthreads();
  // By counting while the class is staged: 254 records took 8.5 us of a launch of 28 in the network's 36 stages.
  if (staged && count <= kAccThreads) rank_sort(key, idx, count);
  else if (staged) rank_sort<kCap / kAccThreads>(key, idx, count);
  else bitonic_sort<true>(key, idx, count, padded);
  __syncthreads();
  // Envelope arrays of this warp: 16-bit in shared memory when the class is staged, else 32-bit in the
  // workspace (each class owns 2 * warps * (count + 1) ints there).
  unsigned short* fp16 = sm.env[warp][0];
  unsigned short* t16 = sm.env[warp][1];
  int* fp32 = env_ws + 2 * (int64_t)warps * ((int64_t)before + c) + (int64_t)warp * 2 * (count + 1);
  int* t32 = fp32 + (count + 1);
  auto load_fp = [&](int j) -> unsigned { return staged ? fp16[j] : (unsigned)fp32[j]; };
  auto store_fp = [&](int j, unsigned v) { if (staged) fp16[j] = (unsigned short)v; else fp32[j] = (int)v; };
  auto load_t = [&](int j) -> unsigned { return staged ? t16[j] : (unsigned)t32[j]; };
  auto store_t = [&](int j, unsigned v) { if (staged) t16[j] = (unsigned short)v; else t32[j] = (int)v; };
  // Envelope order: (ct, cf) beats (bt, bf) when its precision ct / (ct + cf) is larger, or equal with
  // the incumbent at tp + fp = 1 (value 1 / (1 + eps) < 1.0) and the candidate not; (0, *) never wins.
  auto beats = [](unsigned ct, unsigned cf, unsigned bt, unsigned bf) {
    if (ct == 0) return false;
    if (bt == 0) return true;
    const int64_t lhs = (int64_t)ct * ((int64_t)bt + bf), rhs = (int64_t)bt * ((int64_t)ct + cf);
    return lhs > rhs || (lhs == rhs && bt + bf == 1 && ct + cf >= 2);
  };
  for (int group = part; group < kParts; group += parts) {
    const int t_base = group * kT;
    if (staged) {  // ranks and this group's flags of every record, in walk order
      for (int k = threadIdx.x; k < count; k += kAccThreads) sm.rank[k] = ranks[idx[k]];
      for (int e = threadIdx.x; e < count * 4 * kT; e += kAccThreads) {
        const int k = e / (4 * kT), f = e % (4 * kT), a = f % 4, t = f / 4;
        sm.flags[k][f] = flags[(a * 10 + t_base + t) * chain_stride + (int64_t)idx[k] * det_stride];
      }
      __syncthreads();
    }
    // Phase A (integers only): one warp per chain builds the chain's envelope segments.
    for (int ch = warp; ch < kChainsHere; ch += warps) {
      const int m = ch % 3, a = (ch / 3) % 4, t = ch / 12;
      int nseg = 0, hi = 0;
      unsigned tp = 0;
      if (sm.npos[a] > 0) {
        const int limit = m == 0 ? 1 : (m == 1 ? 10 : 100);
        const int64_t chain = (int64_t)(a * 10 + t_base + t) * chain_stride;
        // Prefix counts over the records within maxDets: the j-th true positive's cumulative false
        // positives (those before it) go to fp[j].
        unsigned fp = 0, selected = 0;
        for (int base = 0; base < count; base += 32) {
          const int k = base + lane;
          int f = -1;
          bool sel = false;
          if (k < count) {
            const int rank = staged ? sm.rank[k] : ranks[idx[k]];
            sel = rank >= 1 && rank <= limit;
            if (sel) f = staged ? sm.flags[k][t * 4 + a] : flags[chain + (int64_t)idx[k] * det_stride];
          }
          const unsigned bt = __ballot_sync(0xffffffffu, f == 1), bf = __ballot_sync(0xffffffffu, f == 0);
          selected |= __ballot_sync(0xffffffffu, sel);
          if (f == 1) store_fp(tp + __popc(bt & below) + 1, fp + __popc(bf & below));
          tp += __popc(bt);
          fp += __popc(bf);
        }
        if (selected) {  // without a detection within maxDets: a zero curve (instance.py:315-318)
          const int* tp_min = sm.tp_min[a];
          int reached = 0;  // thresholds reached at the final recall (tp_min is nondecreasing in r)
          for (int r = lane; r <= 100; r += 32) reached += tp_min[r] <= (int)tp;
          hi = __reduce_add_sync(0xffffffffu, reached);
          __syncwarp();
          // Suffix maximum of the envelope over j = tp, tp - 1, ..., 1 (lane 0 holds the largest j of a
          // chunk); the pair at j replaces fp[j] (its own entry, read first) and goes to t[j].
          unsigned ct = 0, cf = 0;  // the best pair of the chunks already scanned
          for (int top = (int)tp; top >= 1; top -= 32) {
            const int j = top - lane;
            unsigned vt = 0, vf = 0;
            if (j >= 1) { vt = (unsigned)j; vf = load_fp(j); }
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
              const unsigned ot = __shfl_up_sync(0xffffffffu, vt, off), of = __shfl_up_sync(0xffffffffu, vf, off);
              if (lane >= off && beats(ot, of, vt, vf)) { vt = ot; vf = of; }
            }
            if (beats(ct, cf, vt, vf)) { vt = ct; vf = cf; }
            if (j >= 1) { store_t(j, vt); store_fp(j, vf); }
            ct = __shfl_sync(0xffffffffu, vt, 31);
            cf = __shfl_sync(0xffffffffu, vf, 31);
          }
          __syncwarp();
          // Threshold r < hi takes the envelope at j = tp_min[r] (thresholds reached with no true positive
          // take the envelope over all of them); runs of equal pairs are the chain's segments.
          int prev_t = -1, prev_f = -1;
          for (int r0 = 0; r0 < hi; r0 += 32) {
            const int r = r0 + lane;
            unsigned pt = 0, pf = 0;
            if (r < hi && tp > 0) {
              const int j = max(tp_min[r], 1);
              pt = load_t(j);
              pf = load_fp(j);
            }
            int lt = __shfl_up_sync(0xffffffffu, (int)pt, 1), lf = __shfl_up_sync(0xffffffffu, (int)pf, 1);
            if (lane == 0) { lt = prev_t; lf = prev_f; }
            const bool start = r < hi && ((int)pt != lt || (int)pf != lf);
            const unsigned starts = __ballot_sync(0xffffffffu, start);
            if (start) {
              const int at = nseg + __popc(starts & below);
              sm.seg_lo[ch][at] = (unsigned char)r;
              sm.seg[ch][at] = (long long)(((unsigned long long)pt << 32) | pf);
            }
            nseg += __popc(starts);
            prev_t = __shfl_sync(0xffffffffu, (int)pt, 31);
            prev_f = __shfl_sync(0xffffffffu, (int)pf, 31);
          }
        }
      }
      if (lane == 0) {
        sm.nseg[ch] = nseg;
        sm.hi[ch] = hi;
        sm.tp[ch] = (int)tp;
      }
    }
    __syncthreads();
    if (warp == 0) {  // segment offsets (exclusive scan over the chains)
      static_assert(kChainsHere <= 32, "one lane per chain");
      const int v0 = lane < kChainsHere ? sm.nseg[lane] : 0;
      int v = v0;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= off) v += u;
      }
      if (lane < kChainsHere) sm.off[lane] = v - v0;
      if (lane == 31) sm.off[kChainsHere] = v;
    }
    __syncthreads();
    // Phase B: every segment's value, fl(tp / ((tp + fp) + eps)), the segments spread over all threads.
    for (int e = threadIdx.x; e < sm.off[kChainsHere]; e += kAccThreads) {
      int lo = 0, hi = kChainsHere - 1;  // chain holding flat segment e
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (sm.off[mid] <= e) lo = mid; else hi = mid - 1;
      }
      long long& slot = sm.seg[lo][e - sm.off[lo]];
      const unsigned long long pair = (unsigned long long)slot;
      const double bt = (double)(int)(pair >> 32), bf = (double)(int)(pair & 0xffffffffull);
      slot = __double_as_longlong(bt / ((bt + bf) + DBL_EPSILON));
    }
    __syncthreads();
    // Phase C: precision values (segment s covers [lo_s, lo_{s+1}), the last up to hi), twelve chains of a
    // (threshold, recall) next to one another; the last warp writes recalls and the chains' sums.
    if (warp == warps - 1) {
      if (lane < kChainsHere) {
        const int a = (lane / 3) % 4, t = t_base + lane / 12;
        const int64_t np = sm.npos[a];
        const double rc = np > 0 ? (double)sm.tp[lane] / (double)np : sm.none[a];
        recall[((int64_t)t * C + c) * 12 + lane % 12] = rc;
        if (chain_stats) {
          double sum = sm.none[a];
          const int nseg = sm.nseg[lane], hi = sm.hi[lane];
          for (int k = 0; k < nseg; ++k) {
            const int end = k + 1 < nseg ? sm.seg_lo[lane][k + 1] : hi;
            sum += __longlong_as_double(sm.seg[lane][k]) * (double)(end - sm.seg_lo[lane][k]);
          }
          double* stats = chain_stats + ((int64_t)c * 120 + t * 12 + lane % 12) * 2;
          stats[0] = sum;
          stats[1] = rc;
        }
      }
    } else {
      for (int e = threadIdx.x; e < kChainsHere * 101; e += kAccThreads - 32) {
        const int k = e % 12, r = (e / 12) % 101, t = e / (12 * 101), ch = t * 12 + k;
        double v = sm.none[k / 3];
        if (r < sm.hi[ch]) {
          int lo = 0, hi = sm.nseg[ch] - 1;  // the last segment starting at or before r
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (sm.seg_lo[ch][mid] <= r) lo = mid; else hi = mid - 1;
          }
          v = __longlong_as_double(sm.seg[ch][lo]);
        }
        precision[(((int64_t)(t_base + t) * 101 + r) * C + c) * 12 + k] = v;
      }
    }
    if (group + parts < kParts) __syncthreads();  // the next group rewrites the tables
  }
}

// The 12 summaries from per-chain statistics: CTA q reduces summary q over its
// (class, threshold) entries in a fixed order (thread-strided, each thread's
// loads issued together before any is used, then a butterfly per warp and the
// warps' partials in index order). One warp per summary walking the entries
// one dependent L2 load at a time took 26 us for 80 classes; the entries fit
// one load round per thread here.
constexpr int kSummarizeThreads = 256;
constexpr int kSummarizeLoads = 4;  // loads in flight per thread and round

__global__ void __launch_bounds__(kSummarizeThreads)
summarize_chains_kernel(const double* __restrict__ chain_stats, int C, double* __restrict__ out) {
  wait_for_earlier_kernels();
  const int q = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // summary -> (uses precision sums?, area, maxDets index, single threshold or -1)
  const bool is_ap = q < 4 || q == 5 || q == 7;
  const int area = (q < 3 || q >= 9) ? 0 : (q <= 4 ? 1 : (q <= 6 ? 2 : 3));
  const int mi = q >= 9 ? q - 9 : 2;
  const int only_t = q == 1 ? 0 : (q == 2 ? 5 : -1);
  const int nt = only_t >= 0 ? 1 : 10;
  const int64_t n = (int64_t)nt * C;  // entry e: class e / nt, threshold e % nt (or only_t)
  const int field = is_ap ? 0 : 1;
  const long long weight = is_ap ? 101 : 1;
  double sum = 0.0;
  long long cnt = 0;
  for (int64_t e0 = tid; e0 < n; e0 += (int64_t)kSummarizeLoads * kSummarizeThreads) {
    double v[kSummarizeLoads];
#pragma unroll
    for (int j = 0; j < kSummarizeLoads; ++j) {
      const int64_t e = e0 + (int64_t)j * kSummarizeThreads;
      v[j] = -1.0;
      if (e < n) {
        const int64_t c = e / nt;
        const int t = only_t >= 0 ? only_t : (int)(e - c * nt);
        v[j] = chain_stats[(c * 120 + t * 12 + area * 3 + mi) * 2 + field];
      }
    }
#pragma unroll
    for (int j = 0; j < kSummarizeLoads; ++j) {
      if (!(v[j] < 0.0)) {  // NaN: an unknown count
        sum += v[j];
        cnt += weight;
      }
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  }
  __shared__ double s_sum[kSummarizeThreads / 32];
  __shared__ long long s_cnt[kSummarizeThreads / 32];
  if (lane == 0) {
    s_sum[warp] = sum;
    s_cnt[warp] = cnt;
  }
  __syncthreads();
  if (tid == 0) {
    double total = 0.0;
    long long count = 0;
    for (int w = 0; w < kSummarizeThreads / 32; ++w) {
      total += s_sum[w];
      count += s_cnt[w];
    }
    out[q] = count ? total / (double)count : -1.0;
  }
}

// The 12 COCO summaries (instance.py:230-248): means of the entries >= 0.
__global__ void __launch_bounds__(256)
summarize_kernel(const double* __restrict__ precision, const double* __restrict__ recall, int C,
                 double* __restrict__ out) {
  wait_for_earlier_kernels();
  // out: ap, ap50, ap75, ap_small, ar_small, ap_medium, ar_medium, ap_large, ar_large, ar1, ar10, ar100
  __shared__ double s_sum[256];
  __shared__ int s_cnt[256];
  {
    const int q = blockIdx.x;  // one CTA per summary
    double sum = 0.0;
    int cnt = 0;
    const bool is_precision = q < 3 || q == 3 || q == 5 || q == 7;
    if (is_precision) {
      const int area = q < 3 ? 0 : (q == 3 ? 1 : (q == 5 ? 2 : 3));
      const int t0 = q == 1 ? 0 : (q == 2 ? 5 : 0);
      const int t1 = q == 1 ? 1 : (q == 2 ? 6 : 10);
      const int64_t per_t = (int64_t)101 * C;
      const int64_t total = (t1 - t0) * per_t;
      for (int64_t e = threadIdx.x; e < total; e += blockDim.x) {
        const int64_t t = t0 + e / per_t, rc = e % per_t;  // rc = r * C + c
        const double v = precision[((t * 101 * C + rc) * 4 + area) * 3 + 2];
        if (v >= 0) { sum += v; ++cnt; }
      }
    } else {
      int area = 0, mi = 2;
      if (q == 4) area = 1;
      else if (q == 6) area = 2;
      else if (q == 8) area = 3;
      else mi = q - 9;  // ar1, ar10, ar100
      const int64_t total = (int64_t)10 * C;
      for (int64_t e = threadIdx.x; e < total; e += blockDim.x) {
        const double v = recall[(e * 4 + area) * 3 + mi];
        if (v >= 0) { sum += v; ++cnt; }
      }
    }
    s_sum[threadIdx.x] = sum;
    s_cnt[threadIdx.x] = cnt;
    __syncthreads();
    for (int s = 128; s; s >>= 1) {
      if ((int)threadIdx.x < s) {
        s_sum[threadIdx.x] += s_sum[threadIdx.x + s];
        s_cnt[threadIdx.x] += s_cnt[threadIdx.x + s];
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) out[q] = s_cnt[0] ? s_sum[0] / (double)s_cnt[0] : -1.0;
    __syncthreads();
  }
}

// ---- detection x target-slot histogram -----------------------------------

constexpr int kDetThreads = 512;
constexpr int kDetPixels = 16;                      // pixels per thread
constexpr int kDetChunk = kDetThreads * kDetPixels;  // pixels per CTA

__device__ __forceinline__ void load16(const uint8_t* p, int64_t x, int64_t end, int align, uint32_t w[4]) {
  if (align == 16 && x + 16 <= end) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p + x));
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
  } else if (align == 4 && x + 16 <= end) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p + x);
    w[0] = __ldg(q); w[1] = __ldg(q + 1); w[2] = __ldg(q + 2); w[3] = __ldg(q + 3);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t v = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (x + 4 * k + j < end) v |= (uint32_t)(__ldg(p + x + 4 * k + j) != 0) << (8 * j);
      w[k] = v;
    }
  }
}

template <bool SMEM>
__global__ void __launch_bounds__(kDetThreads)
detection_histogram_kernel(const uint8_t* __restrict__ masks, int64_t pixels, int D, const int* __restrict__ target,
                           const int64_t* __restrict__ order, int S, int align, u64* __restrict__ pairs) {
  wait_for_earlier_kernels();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  u32* bins = reinterpret_cast<u32*>(smem_raw);
  const int bins_count = D * S;
  if (SMEM) {
    for (int k = threadIdx.x; k < bins_count; k += blockDim.x) bins[k] = 0;
    __syncthreads();
  }
  const int64_t x = (int64_t)blockIdx.x * kDetChunk + (int64_t)threadIdx.x * kDetPixels;
  int slot[kDetPixels];
  bool uniform = true;
#pragma unroll
  for (int j = 0; j < kDetPixels; ++j) {
    slot[j] = x + j < pixels ? target[x + j] : -1;
    if (slot[j] != slot[0]) uniform = false;
  }
  const bool valid0 = slot[0] >= 0 && slot[0] < S;
  for (int d = 0; d < D; ++d) {
    const uint8_t* mask = masks + order[d] * pixels;
    uint32_t w[4] = {0, 0, 0, 0};
    if (x < pixels) load16(mask, x, pixels, align, w);
    const bool any = (w[0] | w[1] | w[2] | w[3]) != 0;
    if (!__ballot_sync(0xffffffffu, any)) continue;
    // Lanes with one valid slot over their 16 pixels combine across the warp.
    const bool simple = any && uniform && valid0;
    const u32 count = simple ? (u32)(__popc(w[0]) + __popc(w[1]) + __popc(w[2]) + __popc(w[3])) : 0u;
    const u32 key = simple ? (u32)(d * S + slot[0]) : 0xffffffffu;
    const u32 peers = __match_any_sync(0xffffffffu, key);
    const u32 total = __reduce_add_sync(peers, count);
    if (simple && (threadIdx.x & 31) == (u32)(__ffs(peers) - 1)) {
      if (SMEM) atomicAdd(bins + key, total);
      else atomicAdd(pairs + key, (u64)total);
    }
    if (any && !simple) {
#pragma unroll
      for (int j = 0; j < kDetPixels; ++j) {
        const bool on = (w[j >> 2] >> (8 * (j & 3))) & 0xff;
        const int s = slot[j];
        if (on && s >= 0 && s < S) {
          if (SMEM) atomicAdd(bins + d * S + s, 1u);
          else atomicAdd(pairs + (int64_t)d * S + s, 1ull);
        }
      }
    }
  }
  if (SMEM) {
    __syncthreads();
    for (int k = threadIdx.x; k < bins_count; k += blockDim.x) {
      const u32 v = bins[k];
      if (v) atomicAdd(pairs + k, (u64)v);
    }
  }
}

// ---- mask x mask overlaps (bit-packed, sparse-aware) -----------------------

constexpr int kOvThreads = 256;
constexpr int kOvWords = 128;  // 32-bit words of packed pixels per CTA (4096 pixels)

// Pack 4 bytes holding 0/1 into 4 bits (any consistent bit order works for AND+popc).
__device__ __forceinline__ uint32_t pack4(uint32_t w) { return ((w & 0x01010101u) * 0x08040201u) >> 24 & 0xfu; }

__global__ void __launch_bounds__(kOvThreads)
mask_overlap_kernel(const uint8_t* __restrict__ pm, int D, const uint8_t* __restrict__ gm, int G, int64_t pixels,
                    int align, const int* __restrict__ pc, const int* __restrict__ gc, u64* __restrict__ inter) {
  wait_for_earlier_kernels();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int rows = D + G;
  uint32_t* bits = reinterpret_cast<uint32_t*>(smem_raw);            // rows x kOvWords
  int2* range = reinterpret_cast<int2*>(bits + (int64_t)rows * kOvWords);  // first/last nonzero word
  const int64_t x0 = (int64_t)blockIdx.x * kOvWords * 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // One warp packs one mask row of the chunk at a time: lane k packs word k + 32 i.
  for (int r = warp; r < rows; r += kOvThreads / 32) {
    const uint8_t* row = r < D ? pm + (int64_t)r * pixels : gm + (int64_t)(r - D) * pixels;
    int first = kOvWords, last = -1;
    for (int k = lane; k < kOvWords; k += 32) {
      const int64_t x = x0 + (int64_t)k * 32;
      uint32_t word = 0;
      if (x < pixels) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint32_t w[4];
          load16(row, x + 16 * q, pixels, align, w);
#pragma unroll
          for (int j = 0; j < 4; ++j) word |= pack4(w[j]) << (16 * q + 4 * j);
        }
      }
      bits[(int64_t)r * kOvWords + k] = word;
      if (word) { first = min(first, k); last = max(last, k); }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
      last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
    }
    if (lane == 0) range[r] = make_int2(first, last);
  }
  __syncthreads();
  for (int pair = threadIdx.x; pair < D * G; pair += blockDim.x) {
    const int d = pair / G, g = pair % G;
    if (pc[d] != gc[g]) continue;
    const int2 rd = range[d], rg = range[D + g];
    const int lo = max(rd.x, rg.x), hi = min(rd.y, rg.y);
    if (lo > hi) continue;
    const uint32_t* a = bits + (int64_t)d * kOvWords;
    const uint32_t* b = bits + (int64_t)(D + g) * kOvWords;
    u32 count = 0;
    for (int k = lo; k <= hi; ++k) count += __popc(a[k] & b[k]);
    if (count) atomicAdd(inter + pair, (u64)count);
  }
}

int alignment_of(const void* p, int64_t pixels) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  if ((a & 15) == 0 && pixels % 16 == 0) return 16;
  if ((a & 3) == 0 && pixels % 4 == 0) return 4;
  return 1;
}

}  // namespace

template <typename Count, typename Area>
int launch_match(const Count* pairs, const int64_t* pair_off, const int64_t* d_off,
                 const int64_t* g_off, int single_d, int single_g, int64_t B, const int* pc, const Area* pa,
                 const int* gc, const Area* ga, const uint8_t* crowd, const double* areas, int C, int g_max,
                 int8_t* flags, int64_t chain_stride, int64_t det_stride, int* ranks, int64_t* counts,
                 cudaStream_t stream, const int* gate = nullptr, const uint32_t* class_bits = nullptr,
                 int unchecked = 0) {
  if (B == 0) return kOk;
  const size_t smem = match_bytes(g_max);
  if (smem > 200 * 1024 || g_max > 65536) {
    set_error("too many ground-truth slots per image for matching (G=%d)", g_max);
    return kUnsupported;
  }
  PE_REQUIRE(B <= INT_MAX, "too many images for one matching launch (B=%lld)", (long long)B);
  const unsigned rows = (unsigned)std::min(C, 65535);
  const dim3 grid((unsigned)B, rows, (unsigned)ceil_div(C, rows));
  FlagLayout layout{flags, chain_stride, det_stride};
  // Many CTAs are bounded by how many an SM holds at a time (64 images of 133 classes: 30 us with 256 threads, 18.7
  // with 128), few by the longest class (32 images of 80: 17.7 us, 21.8 with 128 threads).
  const unsigned threads = B * C > 4096 ? kMatchThreads / 2 : kMatchThreads;
  auto kernel = match_kernel<Count, Area>;
  if (smem > 48 * 1024) PE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch_kernel(kernel, grid, threads, smem, stream, pairs, pair_off, d_off, g_off, single_d, single_g, pc, pa, gc, ga,
      crowd, areas, C, g_max, layout, ranks, counts, gate, class_bits, unchecked);
  PE_LAUNCHED("match");
  count_launch();
  return kOk;
}

template <typename Area>
int launch_match_gated(const u32* pairs, const int64_t* pair_off, const int64_t* d_off, const int64_t* g_off,
                       int64_t B, const int* pc, const Area* pa, const int* gc, const Area* ga, const uint8_t* crowd,
                       const double* areas, int C, int g_max, int8_t* flags, int64_t chain_stride, int64_t det_stride,
                       int* ranks, int64_t* counts, const int* gate, const uint32_t* class_bits, int unchecked,
                       cudaStream_t stream) {
  return launch_match(pairs, pair_off, d_off, g_off, 0, 0, B, pc, pa, gc, ga, crowd, areas, C, g_max, flags,
                      chain_stride, det_stride, ranks, counts, stream, gate, class_bits, unchecked);
}
template int launch_match_gated(const u32*, const int64_t*, const int64_t*, const int64_t*, int64_t, const int*,
                                const double*, const int*, const double*, const uint8_t*, const double*, int, int,
                                int8_t*, int64_t, int64_t, int*, int64_t*, const int*, const uint32_t*, int,
                                cudaStream_t);
template int launch_match_gated(const u32*, const int64_t*, const int64_t*, const int64_t*, int64_t, const int*,
                                const u64*, const int*, const u64*, const uint8_t*, const double*, int, int, int8_t*,
                                int64_t, int64_t, int*, int64_t*, const int*, const uint32_t*, int, cudaStream_t);

int64_t accumulate_workspace_bytes(int64_t n, int64_t C) {
  // Per-class overflow regions (each class's padded to a power of two, at most twice its records: 2n
  // entries), the per-class list (n), then the envelope arrays of classes sorted there.
  return (int64_t)round_up(2 * n + 1, 64) * (int64_t)(sizeof(double) + sizeof(int)) +
         (int64_t)round_up(n + 1, 64) * (int64_t)sizeof(int) +
         2 * (kAccThreads / 32) * (n + C) * (int64_t)sizeof(int);
}

template <int kCap, int kT>
int launch_accumulate_cap(const int* classes, int64_t n, const int* list, const int* cursor, int* hist,
                          const int* ranks, const int8_t* flags, int64_t chain_stride, int64_t det_stride,
                          const double* scores, const int64_t* positives, unsigned long long* ws_key, int* ws_idx,
                          int C, int* env_ws, double* precision, double* recall, double* chain_stats, int above,
                          cudaStream_t stream) {
  auto kernel = accumulate_kernel<kCap, kT>;
  const size_t smem = sizeof(AccShared<kCap, kT>);
  PE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch_kernel(kernel, (unsigned)(C * (10 / kT)), kAccThreads, smem, stream, classes, n, list, cursor, hist, ranks,
      flags, chain_stride, det_stride, scores, positives, ws_key, ws_idx, C, env_ws, precision, recall, chain_stats,
      above);
  PE_LAUNCHED("accumulate");
  count_launch();
  return kOk;
}

int launch_accumulate(const int* classes, const int* ranks, const int8_t* flags, int64_t chain_stride,
                      int64_t det_stride, const double* scores, int64_t n, const int64_t* positives, int C,
                      void* workspace, int64_t workspace_bytes, int* hist, int* cursor, double* precision,
                      double* recall, double* chain_stats, double* summary, cudaStream_t stream) {
  const int64_t need = accumulate_workspace_bytes(n, C);
  if (workspace_bytes < need) {
    set_error("accumulate workspace too small: %lld < %lld bytes", (long long)workspace_bytes, (long long)need);
    return kWorkspaceTooSmall;
  }
  const int64_t entries = round_up(2 * n + 1, 64);
  auto* ws_key = static_cast<unsigned long long*>(workspace);
  int* ws_idx = reinterpret_cast<int*>(ws_key + entries);
  int* list = ws_idx + entries;
  int* env_ws = list + round_up(n + 1, 64);
  if (n <= kScanRecords) {
    list = nullptr;
  } else {
    const int zeroed = zero_spans({{hist, 4 * C}}, stream);
    if (zeroed != kOk) return zeroed;
    const int64_t blocks = std::min<int64_t>(ceil_div(n, 256), (int64_t)sm_count() * 4);
    launch_kernel(class_histogram_kernel, (unsigned)blocks, 256, 0, stream, classes, n, C, hist);
    PE_LAUNCHED("class_histogram");
    launch_kernel(class_offsets_kernel, 1, 1024, 0, stream, hist, C, cursor);
    PE_LAUNCHED("class_offsets");
    launch_kernel(class_scatter_kernel, (unsigned)blocks, 256, 0, stream, classes, n, C, cursor, list);
    PE_LAUNCHED("class_scatter");
    count_launch(3);
  }
  // Classes of up to kSmallCap records in a smaller stage; when some class can be larger, a second launch
  // takes those (staged up to kSortCap, else in the workspace).
  const bool few = C * (10 / kAccT) <= sm_count();  // 15 classes of 230 records: 23.4 us, 20.1 with a threshold per CTA
  auto small = few ? launch_accumulate_cap<kSmallCap, 1> : launch_accumulate_cap<kSmallCap, kAccT>;
  auto large = few ? launch_accumulate_cap<kSortCap, 1> : launch_accumulate_cap<kSortCap, kAccT>;
  int status = small(classes, n, list, cursor, hist, ranks, flags, chain_stride, det_stride, scores, positives, ws_key,
                     ws_idx, C, env_ws, precision, recall, chain_stats, -1, stream);
  if (status == kOk && n > kSmallCap)
    status = large(classes, n, list, cursor, hist, ranks, flags, chain_stride, det_stride, scores, positives, ws_key,
                   ws_idx, C, env_ws, precision, recall, chain_stats, kSmallCap, stream);
  if (status != kOk) return status;
  if (summary) {
    launch_kernel(summarize_chains_kernel, 12, kSummarizeThreads, 0, stream, chain_stats, C, summary);
    PE_LAUNCHED("summarize_chains");
    count_launch();
  }
  return kOk;
}

int launch_summarize(const double* precision, const double* recall, int C, double* out, cudaStream_t stream) {
  launch_kernel(summarize_kernel, 12, 256, 0, stream, precision, recall, C, out);
  PE_LAUNCHED("summarize");
  count_launch();
  return kOk;
}

}  // namespace pe

using namespace pe;

// Drop-in for `instance_histogram` (instance_kernel.cu:335-363): pairs[rank, s]
// counts the pixels of mask order[rank] on target slot s (all slots, including
// void and stuff, so row sums are full detection areas). pairs is zeroed here.
PE_API int pe_instance_histogram(const uint8_t* masks, int64_t D, int64_t pixels, const int32_t* target,
                                 const int64_t* order, int64_t S, int64_t* pairs, cudaStream_t stream) {
  PE_REQUIRE(D >= 0 && D < INT_MAX && pixels > 0 && S > 0 && S < INT_MAX && D * S < INT_MAX,
             "invalid shared ground-truth inputs");
  if (D == 0) return kOk;
  const int zeroed = zero_spans({{pairs, 8 * D * S}}, stream);
  if (zeroed != kOk) return zeroed;
  const int64_t bins = D * S;
  const bool smem = bins <= 48 * 1024;
  const size_t smem_bytes = smem ? sizeof(u32) * bins : 0;
  const int64_t grid = ceil_div(pixels, kDetChunk);
  const int align = alignment_of(masks, pixels);
  auto* out = reinterpret_cast<u64*>(pairs);
  if (smem) {
    if (smem_bytes > 48 * 1024)
      PE_CUDA(cudaFuncSetAttribute(detection_histogram_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem_bytes));
    launch_kernel(detection_histogram_kernel<true>, (unsigned)grid, kDetThreads, smem_bytes, stream, masks, pixels,
        (int)D, target, order, (int)S, align, out);
  } else {
    launch_kernel(detection_histogram_kernel<false>, (unsigned)grid, kDetThreads, 0, stream, masks, pixels, (int)D,
        target, order, (int)S, align, out);
  }
  PE_LAUNCHED("detection_histogram");
  count_launch();
  return kOk;
}

// Drop-in for `instance_match_histogram` (instance_kernel.cu:365-381) and the
// matching half of `instance_update`: COCO greedy matching of D score-sorted
// detections against G targets from integer intersections pairs[D, G].
// Outputs flags [40, D] int8 (1 TP, 0 FP, -1 ignored / unmatched outside the
// area range), ranks [D] int32 (1..100 within class, 0 beyond), counts [C, 4]
// int64 positives (zeroed here).
PE_API int pe_instance_match(const int64_t* pairs, int64_t D, int64_t G, const int32_t* pc, const int32_t* gc,
                             const double* pa, const double* ga, const uint8_t* crowd, const double* areas,
                             int64_t C, int8_t* flags, int32_t* ranks, int64_t* counts, cudaStream_t stream) {
  PE_REQUIRE(D >= 0 && G >= 0 && D < INT_MAX && G < INT_MAX && D * G < INT_MAX, "too many instance pairs");
  PE_REQUIRE(C > 0 && C <= INT_MAX / 120, "invalid category count");
  const int zeroed = zero_spans({{counts, 32 * C}}, stream);
  if (zeroed != kOk) return zeroed;
  if (D == 0 && G == 0) return kOk;
  return launch_match(pairs, nullptr, nullptr, nullptr, (int)D, (int)G, 1, pc, pa, gc, ga, crowd, areas,
                      (int)C, (int)std::max<int64_t>(G, 1), flags, D, 1, ranks, counts, stream);
}

// Intersections of every same-class (prediction, target) mask pair:
// inter[d, g] = |pm[d] & gm[g]| for pc[d] == gc[g], 0 otherwise. Part of
// `instance_update` (instance_kernel.cu:282-309). inter is zeroed here.
PE_API int pe_mask_overlap(const uint8_t* pm, int64_t D, const uint8_t* gm, int64_t G, int64_t pixels,
                           const int32_t* pc, const int32_t* gc, int64_t* inter, cudaStream_t stream) {
  PE_REQUIRE(D >= 0 && G >= 0 && pixels > 0 && D * G < INT_MAX, "invalid instance masks");
  if (D == 0 || G == 0) return kOk;
  const int zeroed = zero_spans({{inter, 8 * D * G}}, stream);
  if (zeroed != kOk) return zeroed;
  const size_t smem = (size_t)(D + G) * (kOvWords * sizeof(uint32_t) + sizeof(int2));
  PE_REQUIRE(smem <= 220 * 1024, "too many masks per image for the overlap kernel (D+G=%lld)", (long long)(D + G));
  const int align = std::min(alignment_of(pm, pixels), alignment_of(gm, pixels));
  if (smem > 48 * 1024)
    PE_CUDA(cudaFuncSetAttribute(mask_overlap_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t grid = ceil_div(pixels, (int64_t)kOvWords * 32);
  launch_kernel(mask_overlap_kernel, (unsigned)grid, kOvThreads, smem, stream, pm, (int)D, gm, (int)G, pixels, align,
      pc, gc, reinterpret_cast<u64*>(inter));
  PE_LAUNCHED("mask_overlap");
  count_launch();
  return kOk;
}

// Workspace bytes pe_instance_accumulate needs for n records and C classes.
PE_API int64_t pe_instance_accumulate_workspace(int64_t n, int64_t C) {
  return accumulate_workspace_bytes(n, C) + 2 * round_up(sizeof(int) * C, 64) + round_up(sizeof(double) * 240 * C, 64) +
         64;
}

// Drop-in for `instance_compute` (instance_kernel.cu:311-333) when scores is
// NULL (records already in global descending-score order, flags [40, n]), and
// the record-store accumulation of InstanceEvaluator.compute when scores is
// given (records in update order; sorted here by score, stably). Flags are
// read at flags[chain * chain_stride + record * det_stride].
// Outputs precision [10, 101, C, 4, 3] and recall [10, C, 4, 3] (fully written).
PE_API int pe_instance_accumulate(const int32_t* classes, const int32_t* ranks, const int8_t* flags,
                                  int64_t chain_stride, int64_t det_stride, const double* scores, int64_t n,
                                  const int64_t* positives, int64_t C, void* workspace, int64_t workspace_bytes,
                                  double* precision, double* recall, double* summary, cudaStream_t stream) {
  PE_REQUIRE(n >= 0 && n < INT_MAX && C > 0 && C <= INT_MAX / 120, "invalid instance state shapes");
  const int64_t ints = round_up(sizeof(int) * C, 64);
  const int64_t head = 2 * ints + round_up(sizeof(double) * 240 * C, 64);
  PE_REQUIRE(workspace_bytes >= head, "workspace too small");
  int* hist = static_cast<int*>(workspace);
  int* cursor = reinterpret_cast<int*>(static_cast<char*>(workspace) + ints);
  double* chain_stats = reinterpret_cast<double*>(static_cast<char*>(workspace) + 2 * ints);
  void* rest = static_cast<char*>(workspace) + head;
  return launch_accumulate(classes, ranks, flags, chain_stride, det_stride, scores, n, positives, (int)C, rest,
                           workspace_bytes - head, hist, cursor, precision, recall, chain_stats, summary, stream);
}

// The 12 AP/AR summaries (instance.py:230-248) into out[12]: ap, ap50, ap75,
// ap_small, ar_small, ap_medium, ar_medium, ap_large, ar_large, ar1, ar10, ar100.
PE_API int pe_instance_summarize(const double* precision, const double* recall, int64_t C, double* out,
                                 cudaStream_t stream) {
  PE_REQUIRE(C > 0 && C < INT_MAX / 120, "invalid category count");
  return launch_summarize(precision, recall, (int)C, out, stream);
}
