// Shared helpers for the sm_103a kernels behind the pe_gb300 C ABI.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <cstdarg>
#include <climits>
#include <algorithm>
#include <initializer_list>

#include "pe_gb300.h"

#define PE_API extern "C" __attribute__((visibility("default")))

namespace pe {

using u64 = unsigned long long;
using u32 = unsigned int;

// Status codes shared by every entry point. Positive values are validation
// bitmasks with the reference's bit meanings (1: unknown ID / slot outside
// capacity, 2: bad class or slot 0 not void, 4: area/metadata mismatch).
enum Status : int {
  kOk = 0,
  kBadArgument = -1,
  kCudaError = -2,
  kWorkspaceTooSmall = -3,
  kUnsupported = -4,
};

// Bits of a batched update's error word from 2^20 up: a kernel gave up (a wait ran out, blocks came out of order),
// whatever the input was. A checked update reads the word and raises. One that checks nothing never reads it, so the
// kernels after it mark the evaluator's state instead: IoU sums NaN, positives kUnknownCount (any sum with counts is
// negative). PQ, SQ, mIoU, AP and AR of such a state are NaN until it is reset.
constexpr int kStoppedBits = ~((1 << 20) - 1);
constexpr int kUncheckedBit = 1 << 27;  // beside them: the update checks nothing
constexpr long long kUnknownCount = -(1ll << 40);

void set_error(const char* fmt, ...);

#define PE_REQUIRE(cond, ...)                  \
  do {                                         \
    if (!(cond)) {                             \
      ::pe::set_error(__VA_ARGS__);            \
      return ::pe::kBadArgument;               \
    }                                          \
  } while (0)

#define PE_CUDA(call)                                                     \
  do {                                                                    \
    cudaError_t _e = (call);                                              \
    if (_e != cudaSuccess) {                                              \
      ::pe::set_error("%s failed: %s", #call, cudaGetErrorString(_e));    \
      return ::pe::kCudaError;                                            \
    }                                                                     \
  } while (0)

#define PE_LAUNCHED(name)                                                        \
  do {                                                                           \
    cudaError_t _e = cudaGetLastError();                                         \
    if (_e != cudaSuccess) {                                                     \
      ::pe::set_error("launch of %s failed: %s", name, cudaGetErrorString(_e));  \
      return ::pe::kCudaError;                                                   \
    }                                                                            \
  } while (0)

int sm_count();            // SMs of the current device (cached per device)
int current_device();
// Zeroes buffers on the stream, all with one kernel: a memset per buffer costs about 2 us of host time and 1.4 us
// of the stream, and breaks the chain of kernels launched ahead (below). Per call: 16 reward
// images 27.7 -> 23.2 us, 16 panoptic images 43.1 -> 38.0, one instance image 112 -> 105. A Status.
struct ZeroSpan {
  void* ptr;
  int64_t bytes;
};
int zero_spans(std::initializer_list<ZeroSpan> spans, cudaStream_t stream);
void count_launch(int n = 1);  // launch counter exposed through pe_launch_count()

__host__ __device__ inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
__host__ __device__ inline int64_t round_up(int64_t a, int64_t b) { return ceil_div(a, b) * b; }

// ---- device helpers --------------------------------------------------------

// Warp-aggregated add: lanes holding the same key combine their values and
// one leader issues the atomic. Every lane of `active` must call it.
__device__ __forceinline__ void warp_add_shared(u32* bins, u32 active, u32 key, u32 value) {
  u32 peers = __match_any_sync(active, key);
  u32 total = __reduce_add_sync(peers, value);
  if ((threadIdx.x & 31) == (u32)(__ffs(peers) - 1)) atomicAdd(bins + key, total);
}

__device__ __forceinline__ void warp_add_global(u64* bins, u32 active, u64 key, u32 value) {
  u32 peers = __match_any_sync(active, key);
  u32 total = __reduce_add_sync(peers, value);
  if ((threadIdx.x & 31) == (u32)(__ffs(peers) - 1)) atomicAdd(bins + key, (u64)total);
}

// Slot of a map value. Without tables a value is its own slot when inside
// [0, S). With tables (sorted original IDs `ids[0..S)`, ids[0] = 0 for void)
// the slot comes from a binary search over ids[1..S), as the reference's
// lookup does (histogram_kernel.cu:25-38). Returns -1 when invalid.
__device__ __forceinline__ int resolve_slot(int64_t key, const int64_t* ids, const int* slots, int S) {
  if (ids == nullptr) return (key >= 0 && key < S) ? (int)key : -1;
  if (key == 0) return 0;
  if (key < 0 || key == INT64_MAX) return -1;
  int lo = 1, hi = S;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (ids[mid] < key) lo = mid + 1; else hi = mid;
  }
  if (lo == S || ids[lo] != key) return -1;
  int slot = slots[lo];
  return (slot > 0 && slot < S) ? slot : -1;
}

// ---- asynchronous copies and mbarriers (sm_90+ PTX) ------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// Make barrier initialisation visible to the async proxy before first use.
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// Wait for the phase of `bar` with the given parity; false after ~`limit`
// SM clock cycles (the caller then reports a timeout instead of hanging).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long limit) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long start = clock64();
  while (!mbar_try_wait(bar, parity))
    if (clock64() - start > limit) return false;
  return true;
}

// Bulk (non-tensor) copy global -> shared, completing `bytes` on `bar`.
// Both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Hint: bring [src, src + bytes) into L2 (16-byte aligned, multiple of 16).
__device__ __forceinline__ void bulk_prefetch_l2(const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

// A position in a ring of N slots with a full and an empty barrier each. A consumer waits for the full barrier's
// `phase`, a producer for the empty barrier's `phase ^ 1` (which a fresh barrier passes).
template <int N>
struct RingSlot {
  int at = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next() {
    if (++at == N) {
      at = 0;
      phase ^= 1u;
    }
  }
};

// The last of B table rows (kFields words each) whose `field` is at most `value`, the first row's being so; `field`
// does not fall. By a whole warp, 128 rows in one round trip: one thread's binary search takes a round trip a step.
template <int kFields>
__device__ __forceinline__ int64_t find_row(const int64_t* table, int64_t B, int field, int64_t value) {
  constexpr int kLoads = 4;
  const int lane = threadIdx.x & 31;
  int64_t lo = 0, hi = B;
  while (hi - lo > 1) {
    const int64_t step = (hi - lo + 32 * kLoads - 1) / (32 * kLoads);
    bool reached[kLoads];
#pragma unroll
    for (int j = 0; j < kLoads; ++j) {
      const int64_t row = lo + step * (lane + 32 * j);
      reached[j] = row < hi && __ldg(table + row * kFields + field) <= value;
    }
    int n = 0;
#pragma unroll
    for (int j = 0; j < kLoads; ++j) n += __popc(__ballot_sync(0xffffffffu, reached[j]));
    lo += step * (n - 1);
    hi = min(hi, lo + step);
  }
  return lo;
}

// Barrier among the first `threads` threads of the CTA (named barrier `id`).
__device__ __forceinline__ void named_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Bytes [o, o + 16) of the 32-byte string lo|hi (little-endian words), o in [0, 16): shifts by 8, 4
// and 0-3 bytes as selects and funnel shifts, with no branches (o may differ between lanes).
__device__ __forceinline__ uint4 realign16(uint4 lo, uint4 hi, int o) {
  uint32_t u0 = lo.x, u1 = lo.y, u2 = lo.z, u3 = lo.w, u4 = hi.x, u5 = hi.y, u6 = hi.z, u7 = hi.w;
  const bool b8 = o & 8, b4 = o & 4;
  u0 = b8 ? u2 : u0; u1 = b8 ? u3 : u1; u2 = b8 ? u4 : u2; u3 = b8 ? u5 : u3; u4 = b8 ? u6 : u4; u5 = b8 ? u7 : u5;
  u0 = b4 ? u1 : u0; u1 = b4 ? u2 : u1; u2 = b4 ? u3 : u2; u3 = b4 ? u4 : u3; u4 = b4 ? u5 : u4;
  const int sh = (o & 3) * 8;
  return make_uint4(__funnelshift_r(u0, u1, sh), __funnelshift_r(u1, u2, sh), __funnelshift_r(u2, u3, sh),
                    __funnelshift_r(u3, u4, sh));
}

// ---- kernels behind one another -------------------------------------------------
// An evaluator call is a chain of short kernels, and each launch that is prepared only when the kernel before it
// has ended and its writes are out costs 2 us of an idle chip. Every kernel of this library is launched with
// programmatic stream serialization and begins with wait_for_earlier_kernels(): its launch is under way while the
// kernel before ends, its blocks start when the last block before has left, and they go on once that kernel's
// writes are visible. No access comes before the wait, so a kernel that completed also stands for all before it.
// No kernel lets the next one start earlier (griddepcontrol.launch_dependents): the next one's read-only loads
// then never see memory that a running kernel writes, and it measured the same. Per call, us: 16 reward images
// 36.5 -> 28.8, 16 COCO-like panoptic images 48.6 -> 43.1, instance updates of 32 images 333 -> 312 and
// 259 -> 242, joint updates 300 -> 285 and 405 -> 389, prefixes of 8 images 260 -> 246.
__device__ __forceinline__ void wait_for_earlier_kernels() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

inline cudaLaunchAttribute early_launch() {
  cudaLaunchAttribute attribute = {};
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  return attribute;
}

// kernel<<<grid, block, smem, stream>>>(args...), launched ahead, in clusters of cluster_y CTAs along y. Errors are
// left to PE_LAUNCHED.
template <typename... Params, typename... Args>
void launch_clusters(void (*kernel)(Params...), dim3 grid, unsigned cluster_y, dim3 block, size_t smem,
                     cudaStream_t stream, Args... args) {
  static_assert(sizeof...(Params) == sizeof...(Args), "one argument per kernel parameter");
  cudaLaunchAttribute attributes[2] = {early_launch(), {}};
  attributes[1].id = cudaLaunchAttributeClusterDimension;
  attributes[1].val.clusterDim.x = attributes[1].val.clusterDim.z = 1;
  attributes[1].val.clusterDim.y = cluster_y;
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  config.attrs = attributes;
  config.numAttrs = cluster_y > 1 ? 2 : 1;
  cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

template <typename... Params, typename... Args>
void launch_kernel(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  launch_clusters(kernel, grid, 1, block, smem, stream, args...);
}

}  // namespace pe
