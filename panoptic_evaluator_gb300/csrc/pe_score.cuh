// Per-image PQ scoring from a G x P pair histogram, shared by the per-call
// update (pe_panoptic.cu) and the batched segmentation pipeline.
//
// Semantics follow the reference (histogram_kernel.cu:100-206; CPU
// evaluator.py:381-417): union = ga + pa - inter - void_overlap, a match iff
// same class, non-crowd target and inter > union / 2 (integer), IoU in FP64,
// the last same-class crowd target sets the ignored area, FP iff ignored
// <= pa / 2, FN for unmatched non-crowd targets. Class sums of one image are
// reduced in prediction order, so per-image results do not depend on timing.
#pragma once

#include "pe_common.cuh"

#include <cooperative_groups.h>

namespace pe {

struct ScoreOut {
  u64* tp;          // [C] (+ image offset applied by the caller in reward mode)
  u64* fp;
  u64* fn;
  double* iou_sum;
  u64* confusion;   // C x (C+1), or nullptr
};

// Row and column sums into areas[0..G) / areas[G..G+P), plus validation bits.
template <typename Count, bool REWARD>
__device__ int score_areas(const Count* __restrict__ pairs, const int* __restrict__ gc, const int* __restrict__ pc,
                           const uint8_t* __restrict__ crowd, u64* __restrict__ areas, int G, int P, int C,
                           bool validate) {
  int err = 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  for (int g = warp; g < G; g += warps) {
    u64 sum = 0;
    for (int p = lane; p < P; p += 32) sum += (u64)pairs[(int64_t)g * P + p];
#pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) {
      areas[g] = sum;
      if (validate) {
        const int c = gc[g];
        if (c < -1 || c >= C || (g == 0 && (c != -1 || crowd[g]))) err |= 2;
        if (g > 0 && ((sum > 0) != (c >= 0))) err |= 4;
      }
    }
  }
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    u64 sum = 0;
    for (int g = 0; g < G; ++g) sum += (u64)pairs[(int64_t)g * P + p];
    areas[G + p] = sum;
    if (validate) {
      const int c = pc[p];
      if (c < -1 || c >= C || (p == 0 && c != -1)) err |= 2;
      if (p > 0 && (REWARD ? (sum > 0 && c < 0) : ((sum > 0) != (c >= 0)))) err |= 4;
    }
  }
  return err;
}

// Accumulate one image. Needs areas from score_areas (after a barrier), a
// G-entry `matched` scratch, and shared staging of P * 13 bytes.
template <typename Count, bool REWARD>
__device__ void score_accumulate(const Count* __restrict__ pairs, const int* __restrict__ gc,
                                 const int* __restrict__ pc, const uint8_t* __restrict__ crowd,
                                 const u64* __restrict__ areas, int* __restrict__ matched, int G, int P, int C,
                                 ScoreOut out, unsigned char* staging) {
  for (int g = threadIdx.x; g < G; g += blockDim.x) matched[g] = 0;
  __syncthreads();
  double* s_sum = reinterpret_cast<double*>(staging);
  int* s_cls = reinterpret_cast<int*>(s_sum + P);
  unsigned char* s_kind = reinterpret_cast<unsigned char*>(s_cls + P);
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    const int prediction = pc[p];
    const bool vp = prediction >= 0 && prediction < C;
    const u64 void_overlap = (u64)pairs[p];
    const u64 pa = areas[G + p];
    u64 ignored = void_overlap;
    bool pm = false;
    double sum = 0.0;
    for (int g = 0; g < G; ++g) {
      const int target = gc[g];
      const u64 inter = (u64)pairs[(int64_t)g * P + p];
      const bool vt = target >= 0 && target < C;
      if (!REWARD && out.confusion && vt && inter && !crowd[g])
        atomicAdd(out.confusion + (int64_t)target * (C + 1) + (vp ? prediction : C), inter);
      if (!vt || !vp || target != prediction) continue;
      if (crowd[g]) {
        ignored = void_overlap + inter;  // the last same-class crowd segment wins
      } else if (inter) {
        const u64 uni = areas[g] + pa - inter - void_overlap;
        if (inter > uni / 2) {
          pm = true;
          sum += (double)inter / (double)uni;
          matched[g] = 1;
        }
      }
    }
    const bool counted = vp && (!REWARD || pa > 0);
    s_cls[p] = counted ? prediction : -1;
    // ignored <= pa / 2 (the reference's FP64 test) is exactly 2 * ignored <= pa for integer counts.
    s_kind[p] = pm ? 1 : ((2 * ignored <= pa) ? 2 : 0);
    s_sum[p] = sum;
  }
  __syncthreads();
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    u64 ntp = 0, nfp = 0;
    double total = 0.0;
    for (int p = 0; p < P; ++p) {
      if (s_cls[p] != c) continue;
      if (s_kind[p] == 1) {
        ++ntp;
        total += s_sum[p];
      } else if (s_kind[p] == 2) {
        ++nfp;
      }
    }
    if (ntp) {
      atomicAdd(out.tp + c, ntp);
      atomicAdd(out.iou_sum + c, total);
    }
    if (nfp) atomicAdd(out.fp + c, nfp);
  }
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    const int c = gc[g];
    if (c >= 0 && c < C && !crowd[g] && !matched[g]) atomicAdd(out.fn + c, 1ull);
  }
}

// Scoring in one pass over the histogram: what bounds one image's scoring is
// latency (a CTA alone on its image reads G x P counts, and the chip holds few
// images), so the counts are read once, 32 neighbouring columns per warp with
// kScoreRows rows in flight, into row and column sums and a list of the nonzero
// entries (a few percent of them: segments overlap few segments). The matching
// then takes one list entry per thread. Targets are disjoint slots of one map,
// so at most one non-crowd target besides slot 0 has inter > union / 2 with a
// prediction (two would need inter_1 + inter_2 > pa - void_overlap >= inter_1 +
// inter_2): the reference's per-prediction sum has one term, and the last
// same-class crowd target is the largest such index. Same results as
// score_accumulate, the class sums added in the same order. Counts of one image
// are below 2^32, slots below 2^16 (the tables' shared memory holds fewer).
// 16 images of 101 x 121 slots: 44.7 -> 10.2 us; 8 of 257 x 277: 132 -> 29.3; 64
// of up to 150 x 170: 41 -> 17.6. Staging all counts and matching column by column
// instead of by list took 18, 71 and 33.
struct ScoreTables {
  double* acc;   // C per-class IoU sums
  double* iou;   // P: the matched target's IoU
  double* iou0;  // P: the same of target slot 0 (0.0 unless unvalidated metadata gives void a class)
  uint2* list;   // nonzero entries: (g << 16 | p, count)
  u32* col;      // P column sums
  u32* over;     // P: pixels on void (row 0)
  u32* row;      // G row sums
  int* pcls;     // P prediction classes, -1 outside [0, C)
  int* gcls;     // G target classes, -1 outside [0, C); crowd targets: -2 - class
  int* hit;      // P: 1 when matched
  int* matched;  // G: 1 when matched
  int* crowds;   // G: crowd slots with a class, unordered
  int* n;        // [0] nonzero entries found (beyond `cap`: not all listed), [1] crowd slots
  int cap;

  __host__ __device__ static size_t base_bytes(int64_t G, int64_t P, int64_t C) {
    return ((size_t)(C + 2 * P) * sizeof(double) + (size_t)(4 * P + 4 * G + 2) * sizeof(int) + 15) & ~size_t{15};
  }
  // Tables and the list in `bytes` of shared memory (at least base_bytes).
  __device__ static ScoreTables at(unsigned char* smem, int G, int P, int C, size_t bytes) {
    ScoreTables t;
    t.cap = (int)((bytes - base_bytes(G, P, C)) / sizeof(uint2));
    t.acc = reinterpret_cast<double*>(smem);
    t.iou = t.acc + C;
    t.iou0 = t.iou + P;
    t.list = reinterpret_cast<uint2*>(t.iou0 + P);
    t.col = reinterpret_cast<u32*>(t.list + t.cap);
    t.over = t.col + P;
    t.row = t.over + P;
    t.pcls = reinterpret_cast<int*>(t.row + G);
    t.gcls = t.pcls + P;
    t.hit = t.gcls + G;
    t.matched = t.hit + P;
    t.crowds = t.matched + G;
    t.n = t.crowds + G;
    return t;
  }
};

// Shared memory for up to `pairs` counts of one image: the tables and room for kScoreList entries.
constexpr size_t kScoreList = 4096;
inline size_t score_bytes(int64_t G, int64_t P, int64_t C, int64_t pairs) {
  return ScoreTables::base_bytes(G, P, C) + sizeof(uint2) * std::min<size_t>(kScoreList, (size_t)std::max<int64_t>(pairs, 1));
}

constexpr int kScoreRows = 8;  // rows whose loads a lane issues before using any

// CTAs of a cluster that share an image's counts: a CTA alone is bounded by what it issues, 3200 cycles per round of
// loads of its 32 warps (kScoreRound cells). A power of two up to 8 that leaves room, since a cluster takes its SMs
// from one of the chip's partitions. Two rounds are as fast alone (16 images of 101 x 121 slots 10.2 us, 10.9 in
// clusters of four).
constexpr int64_t kScoreRound = 8192, kSharedScore = 2 * kScoreRound;
inline unsigned score_parts(int64_t images, int sms) {
  for (int parts = 8; parts > 1; parts >>= 1)
    if (images * parts <= sms * (parts == 2 ? 9 : 7) / 10) return parts;
  return 1;
}

// Row and column sums, nonzero entries and the class tables. Synchronises the block before returning. With parts > 1
// the CTAs (0, 0 .. parts - 1) of a cluster take a share of the rows each and add what they found to the tables of
// part 0, which alone are complete on return: scoring 8 images of 257 x 277 slots 29.3 -> 21.9 us.
template <typename Count>
__device__ void score_totals(const Count* __restrict__ pairs, const ScoreTables& t, const int* __restrict__ gc,
                             const uint8_t* __restrict__ crowd, int G, int P, int C, int part = 0, int parts = 1) {
  const int row0 = (G * part + parts - 1) / parts, row1 = (G * (part + 1) + parts - 1) / parts;  // part 0 has row 0
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const u32 below = (1u << lane) - 1u;
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    t.row[g] = 0;
    t.matched[g] = 0;
  }
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    t.col[p] = 0;
    t.hit[p] = 0;
    t.iou[p] = t.iou0[p] = 0.0;
  }
  for (int c = threadIdx.x; c < C; c += blockDim.x) t.acc[c] = 0.0;
  if (threadIdx.x < 2) t.n[threadIdx.x] = 0;
  __syncthreads();
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    const int c = gc[g];
    const bool in = c >= 0 && c < C, cr = in && crowd[g];
    t.gcls[g] = in ? (cr ? -2 - c : c) : -1;
    if (cr) t.crowds[atomicAdd(t.n + 1, 1)] = g;
  }
  const int blocks = (P + 31) / 32, slices = max(1, warps / blocks);
  for (int unit = warp; unit < blocks * slices; unit += warps) {
    const int slice = unit / blocks, p = (unit - slice * blocks) * 32 + lane;
    const int g0 = row0 + (row1 - row0) * slice / slices, g1 = row0 + (row1 - row0) * (slice + 1) / slices;
    const Count* column = pairs + p;
    u32 sum = 0;
    u32 next[kScoreRows];
    auto load = [&](int g) {
      const Count* at = column + (int64_t)g * P;
#pragma unroll
      for (int j = 0; j < kScoreRows; ++j, at += P) next[j] = g + j < g1 && p < P ? (u32)*at : 0u;
    };
    if (g0 < g1) load(g0);
    for (int g = g0; g < g1; g += kScoreRows) {
      u32 v[kScoreRows], any = 0;
#pragma unroll
      for (int j = 0; j < kScoreRows; ++j) any |= v[j] = next[j];
      if (g + kScoreRows < g1) load(g + kScoreRows);
      if (g == 0 && p < P) t.over[p] = v[0];
      if (!__any_sync(0xffffffffu, any)) continue;  // most segments never meet
      // One place in the list for the entries of all these rows: every atomic on its length waits for the last.
      u32 some[kScoreRows];
      int count = 0;
#pragma unroll
      for (int j = 0; j < kScoreRows; ++j) {
        some[j] = __ballot_sync(0xffffffffu, v[j] != 0);
        count += __popc(some[j]);
      }
      int at = 0;
      if (lane == 0) at = atomicAdd(t.n, count);
      u32 total = 0;  // lane j: row g + j
#pragma unroll
      for (int j = 0; j < kScoreRows; ++j) {
        if (!some[j]) continue;  // the whole warp: most rows have no pixel in these columns
        sum += v[j];
        const u32 row = __reduce_add_sync(0xffffffffu, v[j]);
        total = lane == j ? row : total;
      }
      if (total) atomicAdd(t.row + g + lane, total);
      at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
      for (int j = 0; j < kScoreRows; ++j) {
        const int e = at + __popc(some[j] & below);
        if (v[j] && e < t.cap) t.list[e] = make_uint2((u32)(g + j) << 16 | (u32)p, v[j]);
        at += __popc(some[j]);
      }
    }
    if (sum) atomicAdd(t.col + p, sum);
  }
  __syncthreads();
  if (parts == 1) return;
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  cluster.sync();  // part 0 has its own sums; from here until the next barrier the others add theirs
  if (part) {
    __shared__ int s_at;
    const int n = t.n[0];
    if (threadIdx.x == 0) s_at = atomicAdd(cluster.map_shared_rank(t.n, 0), n);
    u32 *row = cluster.map_shared_rank(t.row, 0), *col = cluster.map_shared_rank(t.col, 0);
    uint2* list = cluster.map_shared_rank(t.list, 0);
    for (int g = row0 + threadIdx.x; g < row1; g += blockDim.x) row[g] = t.row[g];
    for (int p = threadIdx.x; p < P; p += blockDim.x)
      if (t.col[p]) atomicAdd(col + p, t.col[p]);
    __syncthreads();
    // A part whose own list overflowed has n > cap, so part 0 counts more than its list holds too.
    for (int e = threadIdx.x; e < min(n, t.cap); e += blockDim.x)
      if (s_at + e < t.cap) list[s_at + e] = t.list[e];
  }
  cluster.sync();
}

// The reference's value checks over the sums of score_totals (bits 2 and 4).
template <bool REWARD>
__device__ int score_checks(const ScoreTables& t, const int* __restrict__ gc, const int* __restrict__ pc,
                            const uint8_t* __restrict__ crowd, int G, int P, int C) {
  int err = 0;
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    const int c = gc[g];
    if (c < -1 || c >= C || (g == 0 && (c != -1 || crowd[g]))) err |= 2;
    if (g > 0 && ((t.row[g] > 0) != (c >= 0))) err |= 4;
  }
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    const int c = pc[p];
    if (c < -1 || c >= C || (p == 0 && c != -1)) err |= 2;
    if (p > 0 && (REWARD ? (t.col[p] > 0 && c < 0) : ((t.col[p] > 0) != (c >= 0)))) err |= 4;
  }
  return err;
}

// After score_totals: matches, confusion, tp / fp / fn and the class IoU sums.
template <typename Count, bool REWARD>
__device__ void score_matches(const Count* __restrict__ pairs, const ScoreTables& t, const int* __restrict__ pc, int G,
                              int P, int C, ScoreOut out) {
  const int lane = threadIdx.x & 31;
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    const int c = pc[p];
    t.pcls[p] = c >= 0 && c < C ? c : -1;
  }
  __syncthreads();
  auto entry = [&](int g, int p, u32 inter) {
    const int target = t.gcls[g];
    if (target < 0) return;
    const int prediction = t.pcls[p];
    if (!REWARD && out.confusion)
      atomicAdd(out.confusion + (int64_t)target * (C + 1) + (prediction >= 0 ? prediction : C), (u64)inter);
    if (target != prediction) return;
    const u64 uni = (u64)t.row[g] + t.col[p] - inter - t.over[p];
    if (inter > uni / 2) {  // one target at most besides slot 0: single writers
      (g ? t.iou : t.iou0)[p] = (double)inter / (double)uni;
      t.hit[p] = 1;
      t.matched[g] = 1;
    }
  };
  const int n = t.n[0];
  if (n <= t.cap) {
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
      const uint2 v = t.list[e];
      entry((int)(v.x >> 16), (int)(v.x & 0xffffu), v.y);
    }
  } else {  // more nonzero entries than the list holds: read the histogram again
    for (int64_t e = threadIdx.x; e < (int64_t)G * P; e += blockDim.x) {
      const u32 v = (u32)pairs[e];
      if (v) entry((int)(e / P), (int)(e % P), v);
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    // Class sums in prediction order: 32 predictions at a time, one lane per class of the group adding its
    // peers' IoUs one after another.
    for (int p0 = 0; p0 < P; p0 += 32) {
      const int p = p0 + lane;
      const int c = p < P && t.hit[p] ? t.pcls[p] : -1;
      u32 peers = __match_any_sync(0xffffffffu, c);
      if (c >= 0 && lane == __ffs(peers) - 1) {
        atomicAdd(out.tp + c, (u64)__popc(peers));
        double sum = t.acc[c];
        for (; peers; peers &= peers - 1) {
          const int q = p0 + __ffs(peers) - 1;
          sum += t.iou0[q] + t.iou[q];
        }
        t.acc[c] = sum;
      }
      __syncwarp();
    }
    for (int c = lane; c < C; c += 32)
      if (t.acc[c] > 0.0) atomicAdd(out.iou_sum + c, t.acc[c]);  // every matched IoU is above 0.5
  } else {
    const int tid = threadIdx.x - 32, step = blockDim.x - 32, crowds = t.n[1];
    for (int p = tid; p < P; p += step) {
      const int c = t.pcls[p];
      if (c < 0 || t.hit[p] || (REWARD && t.col[p] == 0)) continue;
      int last = -1;  // the last same-class crowd target
      for (int k = 0; k < crowds; ++k) {
        const int g = t.crowds[k];
        if (g > last && t.gcls[g] == -2 - c) last = g;
      }
      const u64 ignored = (u64)t.over[p] + (last >= 0 ? (u32)pairs[(int64_t)last * P + p] : 0u);
      if (2 * ignored <= t.col[p]) atomicAdd(out.fp + c, 1ull);
    }
    for (int g = tid; g < G; g += step)
      if (t.gcls[g] >= 0 && !t.matched[g]) atomicAdd(out.fn + t.gcls[g], 1ull);
  }
}

inline size_t score_staging_bytes(int64_t P) { return (size_t)P * (sizeof(double) + sizeof(int) + 1) + 16; }

}  // namespace pe
