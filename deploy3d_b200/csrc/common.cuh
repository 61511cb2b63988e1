// Shared helpers for the sm_100a kernels: status handling, launch geometry, warp primitives and
// the 64-bit-slot open-addressing hash table used by the rulebook generator and the voxel encoders.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>
#include <stdint.h>
#include <stdlib.h>

#include "../../include/deploy3d_b200.h"

namespace d3d {

// NVTX range around every C-ABI enqueue, off unless the process was started with D3D_NVTX=1 (the reference has a
// per-layer profiler on the TensorRT side only, deploy3d/symfun/trt_utils/trt_module.py:20-44).
inline bool nvtx_enabled() {
  static const bool on = [] {
    const char* v = getenv("D3D_NVTX");
    return v && v[0] == '1';
  }();
  return on;
}
struct NvtxRange {
  bool on;
  explicit NvtxRange(const char* name) : on(nvtx_enabled()) {
    if (on) nvtxRangePushA(name);
  }
  ~NvtxRange() {
    if (on) nvtxRangePop();
  }
};
#define D3D_NVTX_RANGE(name) ::d3d::NvtxRange d3d_nvtx_range_(name)

constexpr int kNumSMs = 148;  // B200: 2 dies x 74 SMs; grids of streaming kernels are sized in multiples of it

#define D3D_CHECK_LAUNCH()                                  \
  do {                                                      \
    if (cudaGetLastError() != cudaSuccess) return D3D_ERR_CUDA; \
  } while (0)

#define D3D_REQUIRE(cond, code) \
  do {                          \
    if (!(cond)) return (code); \
  } while (0)

static inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
static inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }
static inline size_t next_pow2(size_t x) {
  size_t y = 1;
  while (y < x) y <<= 1;
  return y;
}
// Grid for a grid-stride kernel: enough CTAs to cover `work_items`, capped at `waves` full waves of the GPU.
static inline int stream_grid(int64_t work_items, int threads, int ctas_per_sm = 8) {
  int64_t need = ceil_div(work_items > 0 ? work_items : 1, threads);
  int64_t cap = (int64_t)kNumSMs * ctas_per_sm;
  return (int)(need < cap ? need : cap);
}

// Launch in `st`; `chained`: as a programmatic dependent of the kernel before it, for kernels that call pdl_wait() before
// they touch memory.  The launch gap inside a chain of 3-5 us kernels goes from about 1.2 to 0.4 us.
template <class... P, class... A>
int launch_chained(bool chained, void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid, cfg.blockDim = dim3(threads), cfg.dynamicSmemBytes = smem, cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...) == cudaSuccess ? D3D_OK : D3D_ERR_CUDA;
}
#define D3D_LAUNCH(chained, kern, grid, threads, smem, st, ...)                                              \
  do {                                                                                                       \
    const int rc_ = ::d3d::launch_chained(chained, kern, dim3(grid), threads, smem, st, __VA_ARGS__);        \
    if (rc_ != D3D_OK) return rc_;                                                                           \
  } while (0)

static inline size_t dtype_size(int dtype) {
  switch (dtype) {
    case D3D_FLOAT: return 4;
    case D3D_HALF: return 2;
    case D3D_BF16: return 2;
    case D3D_INT32: return 4;
    case D3D_INT8: return 1;
    case D3D_BOOL: return 1;
    default: return 0;
  }
}

// Bump allocator over the caller-provided workspace (256-byte granularity).
struct Carver {
  uint8_t* base;
  size_t off;
  explicit Carver(void* p) : base(reinterpret_cast<uint8_t*>(p)), off(0) {}
  template <class T> T* take(size_t count) {
    T* r = base ? reinterpret_cast<T*>(base + off) : nullptr;
    off += align_up(count * sizeof(T), 256);
    return r;
  }
};

// ---------------------------------------------------------------------------------------------
// Device side
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Inclusive scan of `v` over the CTA (blockDim.x multiple of 32, <= 1024). `warp_sums` : >= 32 ints of smem.
// Returns the exclusive prefix of this thread; *total receives the CTA sum.
__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums, int* total) {
  int lane = lane_id(), warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
  int inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += t;
  }
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int w = lane < nwarp ? warp_sums[lane] : 0;
    int winc = w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, winc, d);
      if (lane >= d) winc += t;
    }
    warp_sums[lane] = winc - w;  // exclusive warp offsets
    if (lane == 31) warp_sums[32] = winc;
  }
  __syncthreads();
  int excl = warp_sums[warp] + inc - v;
  *total = warp_sums[32];
  __syncthreads();
  return excl;
}

// ---------------------------------------------------------------------------------------------
// Open-addressing hash table on packed voxel keys.
//   slot word  = (key << 32) | value, EMPTY = all ones; one 64-bit CAS claims key and value together,
//                a 64-bit atomicMin on an owned slot keeps the smallest value (first touch).
//   key        = mixed-radix packing of (b, d0, d1, ..) into 31 bits (the linear offset the reference
//                uses as key, trt/include/common/refnd.h:48-54).
//   hash       = Murmur3 finaliser of (key >> 2) selects a 32-byte bucket of four slots, key & 3 selects the
//                slot inside it; probing advances by whole buckets.  Keys that differ only in the two low bits
//                (neighbours along the fastest axis) therefore share one 32-byte sector, so the three probes
//                a thread issues along x usually cost a single L2 sector instead of three.
//   capacity   = power of two chosen on the device from the live input count, >= 2 x the keys inserted.
// Probe loops are bounded by the capacity and report failure instead of spinning.
// ---------------------------------------------------------------------------------------------
constexpr unsigned long long kEmptySlot = ~0ull;

__device__ __forceinline__ uint32_t murmur_mix(uint32_t k) {
  k ^= k >> 16;
  k *= 0x85ebca6bu;
  k ^= k >> 13;
  k *= 0xc2b2ae35u;
  k ^= k >> 16;
  return k;
}

__device__ __forceinline__ uint32_t home_slot(uint32_t key, uint32_t cap_mask) {
  return ((murmur_mix(key >> 2) << 2) | (key & 3u)) & cap_mask;
}

// Insert (key -> min(value)). Returns the slot, or 0xFFFFFFFF when the table is full.
__device__ __forceinline__ uint32_t hash_insert_min(unsigned long long* table, uint32_t cap_mask, uint32_t key,
                                                    uint32_t value) {
  const unsigned long long mine = ((unsigned long long)key << 32) | value;
  uint32_t slot = home_slot(key, cap_mask);
  for (uint32_t probes = 0; probes <= (cap_mask >> 2); ++probes) {
    unsigned long long cur = table[slot];
    if (cur == kEmptySlot) {
      cur = atomicCAS(&table[slot], kEmptySlot, mine);
      if (cur == kEmptySlot) return slot;
    }
    if ((uint32_t)(cur >> 32) == key) {
      if ((uint32_t)cur > value) atomicMin(&table[slot], mine);
      return slot;
    }
    slot = (slot + 4u) & cap_mask;
  }
  return 0xFFFFFFFFu;
}

// The same insertion for key sets with few repeats (one voxel per key, or nearly): the slot is claimed without looking
// first, so the common case -- an empty home slot -- costs one round trip to the table instead of two.
__device__ __forceinline__ uint32_t hash_insert_min_claim_first(unsigned long long* table, uint32_t cap_mask,
                                                                uint32_t key, uint32_t value) {
  const unsigned long long mine = ((unsigned long long)key << 32) | value;
  uint32_t slot = home_slot(key, cap_mask);
  for (uint32_t probes = 0; probes <= (cap_mask >> 2); ++probes) {
    const unsigned long long cur = atomicCAS(&table[slot], kEmptySlot, mine);
    if (cur == kEmptySlot) return slot;
    if ((uint32_t)(cur >> 32) == key) {
      if ((uint32_t)cur > value) atomicMin(&table[slot], mine);
      return slot;
    }
    slot = (slot + 4u) & cap_mask;
  }
  return 0xFFFFFFFFu;
}

// Insertion for tables nobody probes by neighbourhood (the encoders): the whole key is hashed and probing is linear.  The
// bucketed home slots above keep the two low bits of the key, so keys that agree in them -- the ground of a scan, one
// height of a grid whose fastest axis is z -- would share a quarter of the table (cylinder grid, 120 k points: 48 us of
// probing at that quarter's load of nearly one).
__device__ __forceinline__ uint32_t hash_insert_min_scattered(unsigned long long* table, uint32_t cap_mask, uint32_t key,
                                                              uint32_t value) {
  const unsigned long long mine = ((unsigned long long)key << 32) | value;
  uint32_t slot = murmur_mix(key) & cap_mask;
  for (uint32_t probes = 0; probes <= cap_mask; ++probes) {
    const unsigned long long cur = atomicCAS(&table[slot], kEmptySlot, mine);
    if (cur == kEmptySlot) return slot;
    if ((uint32_t)(cur >> 32) == key) {
      if ((uint32_t)cur > value) atomicMin(&table[slot], mine);
      return slot;
    }
    slot = (slot + 1u) & cap_mask;
  }
  return 0xFFFFFFFFu;
}

// Lookup; returns the value or -1.
__device__ __forceinline__ int32_t hash_lookup(const unsigned long long* __restrict__ table, uint32_t cap_mask,
                                               uint32_t key) {
  uint32_t slot = home_slot(key, cap_mask);
  for (uint32_t probes = 0; probes <= (cap_mask >> 2); ++probes) {
    unsigned long long cur = __ldg(&table[slot]);
    if ((uint32_t)(cur >> 32) == key) return (int32_t)(uint32_t)cur;
    if (cur == kEmptySlot) return -1;
    slot = (slot + 4u) & cap_mask;
  }
  return -1;
}

// Lookup split in two so that a thread can have the first probes of several keys in flight at once: the caller
// loads `first = table[home_slot(key)]` for all its keys, then resolves each; only a collision walks on.
__device__ __forceinline__ int32_t hash_lookup_resolve(const unsigned long long* __restrict__ table, uint32_t cap_mask,
                                                       uint32_t key, unsigned long long first) {
  if ((uint32_t)(first >> 32) == key) return (int32_t)(uint32_t)first;
  if (first == kEmptySlot) return -1;
  uint32_t slot = (home_slot(key, cap_mask) + 4u) & cap_mask;
  for (uint32_t probes = 1; probes <= (cap_mask >> 2); ++probes) {
    unsigned long long cur = __ldg(&table[slot]);
    if ((uint32_t)(cur >> 32) == key) return (int32_t)(uint32_t)cur;
    if (cur == kEmptySlot) return -1;
    slot = (slot + 4u) & cap_mask;
  }
  return -1;
}

// Capacity (slots, power of two >= 16) for `keys` insertions at load factor <= 0.5, clamped to `cap_max`.
__device__ __forceinline__ uint32_t hash_capacity(long long keys, uint32_t cap_max) {
  unsigned long long want = (unsigned long long)(keys > 8 ? keys : 8) * 2ull;
  uint32_t cap = 16;
  while (cap < want && cap < cap_max) cap <<= 1;
  return cap;
}

// Checked build (-DDEPLOY3D_BOUNDS_CHECK, python -m deploy3d_b200.build --checked): every row id, table entry or
// coordinate a kernel is about to index with is range-checked first; the first violation is recorded (site, value,
// limit), every one counted, and the access skipped.  One record for the whole library, so the checked build is
// compiled as relocatable device code.  In the regular build the macro is the constant `true`: the kernels keep only
// the range checks they need for safety and drop out-of-range entries silently, as the reference does.
enum BoundsSite {
  kSiteMmTcId = 1,      // SPConvMM tensor-core kernel: neighbour id outside [-1, rows of the input tensor)
  kSiteMmSimtId = 2,    // SPConvMM SIMT kernel: the same
  kSiteTableEntry = 3,  // neighbour table build: rulebook entry with a negative gather or an out-of-range scatter index
  kSiteBevCoord = 4,    // BEVDensify: voxel coordinate outside the dense grid
  kSiteScatterTo = 5,   // ScatterTo: voxel id >= number of voxels
  kSiteGatherBack = 6,  // GatherBack: voxel id >= number of voxels
  kSiteMirror = 7,      // neighbour table build with the mirror hint: a centre-offset entry that does not map a row to
                        // itself (duplicate input coordinates: the rulebook is not mirror-symmetric)
};
#ifdef DEPLOY3D_BOUNDS_CHECK
extern __device__ int g_d3d_bounds[4];  // violations seen; site, value and limit of the first
__device__ __forceinline__ bool bounds_ok(long long v, long long lo, long long hi, int site) {
  if (v >= lo && v < hi) return true;
  if (atomicAdd(&g_d3d_bounds[0], 1) == 0) g_d3d_bounds[1] = site, g_d3d_bounds[2] = (int)v, g_d3d_bounds[3] = (int)hi;
  return false;
}
#define D3D_BOUNDS_OK(v, lo, hi, site) ::d3d::bounds_ok((long long)(v), (long long)(lo), (long long)(hi), site)
#else
#define D3D_BOUNDS_OK(v, lo, hi, site) true
#endif

// Soft failures a kernel reports in the caller's optional status word (atomicOr; the word is the caller's to
// clear): they drop work instead of faulting, exactly where the reference is silent
// (trt/include/common/hash32.h:70, trt/spconv/index.cu:163-168).
__device__ __forceinline__ void report_status(int32_t* status, int bit) {
  if (status) atomicOr(status, bit);
}

template <class T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <class T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Programmatic dependent launch: let the next kernel of the stream start, wait for the one before.  Both do nothing in a
// kernel launched without the attribute.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Sum of the counts of the blocks in front of this one, by the whole block: a few hundred to a few thousand words that
// every block reads for itself.  (A scan kernel between the count and its use costs a launch and runs on one CTA; blocks
// that wait for each other's prefixes in one pass poll the same lines a thousand at a time: 28 us where the count kernel
// and this take 11, 300 k points.)  What all blocks read together grows with the square of their number, so beyond
// kMaxSummedBlocks scan_counts() is launched in between after all and `scanned` counts are prefixes already: mean encoder
// by summing / scanning 32 / 35 us at 1172 blocks, 53.7 / 51.7 at 4096, 156 / 144 at 16 k, 736 / 525 at 65 k; strided tables
// 66 / 71 us at 2594 blocks of words, 84 / 80 at 8458, 1482 / 635 at 122 k.  `scratch`: a word per warp.
constexpr int kMaxSummedBlocks = 4096;
template <int kThreads>
__device__ __forceinline__ int preceding_sum(const int32_t* __restrict__ counts, int blk, bool scanned, int* scratch) {
  if (scanned) return __ldg(counts + blk);
  int s = 0;
  for (int j = threadIdx.x; j < blk; j += kThreads) s += __ldg(counts + j);
  s = __reduce_add_sync(0xffffffffu, s);
  if (lane_id() == 0) scratch[threadIdx.x >> 5] = s;
  __syncthreads();
  s = 0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) s += scratch[w];
  return s;
}

// Single CTA, in place: counts[i] becomes the sum of the counts in front of it.  Eight counts a thread and turn, the next
// turn's loads ahead of this one's barriers.  counts: on 16 bytes.
static __global__ void __launch_bounds__(1024) scan_counts_kernel(int32_t* __restrict__ counts, int n) {
  __shared__ int scratch[40];
  pdl_release();
  pdl_wait();
  constexpr int kItems = 8, kTurn = 1024 * kItems;
  int carry = 0;
  int4 next[2];
  auto load = [&](int at) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = at + 4 * h;
      int4 v = make_int4(0, 0, 0, 0);
      if (i + 3 < n) v = *reinterpret_cast<const int4*>(counts + i);
      else if (i < n) v.x = counts[i], v.y = i + 1 < n ? counts[i + 1] : 0, v.z = i + 2 < n ? counts[i + 2] : 0;
      next[h] = v;
    }
  };
  load(threadIdx.x * kItems);
  for (int at0 = 0; at0 < n; at0 += kTurn) {
    const int at = at0 + threadIdx.x * kItems;
    int v[kItems] = {next[0].x, next[0].y, next[0].z, next[0].w, next[1].x, next[1].y, next[1].z, next[1].w};
    if (at < n - kTurn) load(at + kTurn);  // n - kTurn: no overflow near the largest n
    else next[0] = next[1] = make_int4(0, 0, 0, 0);
    int mine = 0;
#pragma unroll
    for (int e = 0; e < kItems; ++e) mine += v[e];
    int total, sum = carry + block_exclusive_scan(mine, scratch, &total);
#pragma unroll
    for (int e = 0; e < kItems; ++e) {
      const int c = v[e];
      v[e] = sum, sum += c;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = at + 4 * h;
      if (i + 3 < n) *reinterpret_cast<int4*>(counts + i) = make_int4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
      else
        for (int q = 0; q < 4; ++q)
          if (i + q < n) counts[i + q] = v[4 * h + q];
    }
    carry += total;
  }
}

// Between the kernel that counts per block and the one that numbers: whether the counts are prefixes now (`*scanned`).
static inline int scan_counts(int32_t* counts, int blocks, bool chained, cudaStream_t st, bool* scanned) {
  *scanned = blocks > kMaxSummedBlocks;
  if (*scanned) D3D_LAUNCH(chained, scan_counts_kernel, 1, 1024, 0, st, counts, blocks);
  return D3D_OK;
}

// Single CTA: in-place exclusive scan of `totals[0..n)`; *clamped_total = min(sum, limit).  A sum above the limit
// (more voxels than the output buffers hold: the surplus is dropped) sets D3D_STATUS_OUTPUT_OVERFLOW.
static __global__ void scan_totals_kernel(int32_t* totals, int n, int32_t limit, int32_t* clamped_total,
                                          int32_t* status = nullptr) {
  __shared__ int scratch[40];
  int carry = 0;
  for (int base = 0; base < n; base += blockDim.x) {
    int j = base + threadIdx.x;
    int v = j < n ? totals[j] : 0;
    int total;
    int ex = block_exclusive_scan(v, scratch, &total);
    if (j < n) totals[j] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) {
    *clamped_total = carry < limit ? carry : limit;
    if (carry > limit) report_status(status, D3D_STATUS_OUTPUT_OVERFLOW);
  }
}

}  // namespace d3d
