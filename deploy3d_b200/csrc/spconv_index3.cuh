// Rulebooks of 3-D kernels with at most three taps per axis (27 offsets): the kernels every LiDAR network uses.
// Included by spconv_index.cu, whose Geometry and live_count it shares.
//
// How a voxel id is found.  Keys are linear offsets into the grid, so the plainest table is the grid itself:
//   direct  int32 [cells], -1 = empty.  Insertion is a result-less atomicMin, a lookup one load, x-neighbours share a
//           32-byte sector; nothing is hashed and nothing collides.  The price is clearing the grid (5 TB/s).
//   bits    one bit per cell says whether a voxel is there, a hash table where.  For submanifold probes of fine, nearly
//           empty grids (85 M cells, 0.3 M voxels: 24 of 27 probes miss): the three probes along x are answered by
//           one word, and only the hits -- three per voxel -- go to the hash table.
// Which one is taken depends on cells per voxel (see pick_lookup in spconv_index.cu).
//
// What a pass hands on.  The pairs of a block of 256 inputs are kept as one list, sorted by offset and input (value and
// 8-bit position in the block), instead of a dense [offset][input] table: 1.5 to 16 of 27 entries exist, and the later
// pass reads and writes only those.
#pragma once

namespace d3d {
namespace {

constexpr int kTaps3 = 27;  // offsets of the enclosing 3 x 3 x 3 kernel: g = (a * 3 + b) * 3 + c
constexpr int kBlockWarps = kIdxThreads / 32;

// A neighbour table (SPConvMM's layout) a pass fills for tiles of the voxels it walks: slot s of the table is offset
// g_of_slot[s] of the pass.
struct TableTarget {
  int32_t* ids;
  uint32_t* mask;
  uint32_t* rows;
  int32_t* perm;
  int kvol;
  signed char g_of_slot[kTaps3], slot_of_g[kTaps3];  // -1: the table does not have that offset
};
constexpr int kMaxTargets = 8;
struct Targets {
  int count;
  int64_t tiles;  // of every target
  TableTarget t[kMaxTargets];
};

struct PairLists {
  int32_t* value;      // [block][256 * kvol]
  uint8_t* local;      // the same: position of the input in its block
  int32_t* counts;     // [kvol][nblk]
  int nblk;
};

struct Lookup3 {
  int32_t* direct;             // null: bits + slots
  unsigned long long* slots;
  uint32_t cap_max;
  uint32_t* bits;
};

// Clears what a rulebook starts from: the lookup (live part of the hash table, all of the grid or of the bit map), the
// ticket of segment_scan_kernel, and the row masks / output map of a neighbour table that is filled by scattering.
struct ClearArgs {
  Lookup3 look;
  int64_t direct_words, bit_words;
  int fan;
  int32_t* state;
  uint32_t* rows;
  int64_t row_words;
  int32_t* perm;
  int64_t perm_words, m_max;
};
__global__ void __launch_bounds__(256) clear3_kernel(const ClearArgs a, const int32_t* num_act_in, int64_t n_max) {
  pdl_release();
  pdl_wait();
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (int64_t)gridDim.x * blockDim.x;
  if (tid == 0 && a.state) a.state[2] = 0;
  const uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u), zero = make_uint4(0u, 0u, 0u, 0u);
  auto fill = [&](void* p, int64_t bytes16, const uint4& v) {
    uint4* d = reinterpret_cast<uint4*>(p);
    int64_t i = tid;
    for (; i + 3 * nth < bytes16; i += 4 * nth) d[i] = v, d[i + nth] = v, d[i + 2 * nth] = v, d[i + 3 * nth] = v;
    for (; i < bytes16; i += nth) d[i] = v;
  };
  if (a.look.direct) fill(a.look.direct, a.direct_words / 4, ones);  // sizes are padded to 256 bytes
  if (a.look.bits) fill(a.look.bits, a.bit_words / 4, zero);
  if (a.look.slots) {  // without a count (cleared ahead of the frame's voxels): all of them
    const uint32_t cap = !num_act_in ? a.look.cap_max : hash_capacity((long long)live_count(num_act_in, n_max) * a.fan, a.look.cap_max);
    fill(a.look.slots, cap / 2, ones);
  }
  if (a.rows) fill(a.rows, a.row_words / 4, zero);
  for (int64_t i = tid; i < a.perm_words; i += nth) a.perm[i] = i < a.m_max ? (int32_t)i : -1;
}

__global__ void __launch_bounds__(kIdxThreads)
subm_mark3_kernel(const Lookup3 look, const int32_t* __restrict__ coors, const int32_t* num_act_in, int64_t n_max,
                  const Geometry g, int32_t* status) {
  pdl_release();
  pdl_wait();
  const int n = live_count(num_act_in, n_max);
  const int i = blockIdx.x * kIdxThreads + threadIdx.x;
  if (i >= n) return;
  const int4 c = __ldg(reinterpret_cast<const int4*>(coors) + i);
  if ((uint32_t)c.x >= (uint32_t)g.shape[0] || (uint32_t)c.y >= (uint32_t)g.shape[1] ||
      (uint32_t)c.z >= (uint32_t)g.shape[2] || (uint32_t)c.w >= (uint32_t)g.shape[3])
    return;
  const uint32_t key = (((uint32_t)c.x * g.shape[1] + c.y) * g.shape[2] + c.z) * g.shape[3] + c.w;
  if (look.direct) {
    atomicMin(reinterpret_cast<unsigned*>(look.direct) + key, (unsigned)i);
    return;
  }
  atomicOr(look.bits + (key >> 5), 1u << (key & 31));
  const uint32_t mask = hash_capacity((long long)n * kSubmFan, look.cap_max) - 1;
  if (hash_insert_min_claim_first(look.slots, mask, key, (uint32_t)i) == 0xFFFFFFFFu)
    report_status(status, D3D_STATUS_HASH_FULL);
}

// What a block of 256 inputs has found: values[g][thread] where bit g of the thread's mask is set.
struct Found {
  int values[kTaps3][kIdxThreads];
  uint32_t hits[kTaps3][kBlockWarps];  // ballots
  int base[kTaps3][kBlockWarps];       // where the pairs of an (offset, warp) start in the block's list
};

// Ballots of all offsets; afterwards every thread may read f.hits.
__device__ __forceinline__ void publish_hits(Found& f, uint32_t mask) {
  const int lane = lane_id(), warp = threadIdx.x >> 5;
#pragma unroll
  for (int g = 0; g < kTaps3; ++g) {
    const unsigned b = __ballot_sync(0xffffffffu, (mask >> g) & 1u);
    if (lane == 0) f.hits[g][warp] = b;
  }
  __syncthreads();
}

// Appends the block's pairs to its list, sorted by kernel offset and input, and publishes their numbers per offset.
// `g.ksize` tells which of the 27 offsets exist; kernel offset k = (a * ks1 + b) * ks2 + c ascends with g.
__device__ __forceinline__ void write_lists(Found& f, const Geometry& g, uint32_t mask, const PairLists& lists) {
  const int lane = lane_id(), warp = threadIdx.x >> 5, blk = blockIdx.x;
  if (warp == 0) {
    int total = 0, k = 0;
    bool exists = false;
    if (lane < kTaps3) {
      const int a = lane / 9, b = lane / 3 % 3, c = lane % 3;
      exists = a < g.ksize[0] && b < g.ksize[1] && c < g.ksize[2];
      k = (a * g.ksize[1] + b) * g.ksize[2] + c;
#pragma unroll
      for (int w = 0; w < kBlockWarps; ++w) total += __popc(f.hits[lane][w]);
    }
    int inc = total;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += t;
    }
    if (lane < kTaps3) {
      int at = inc - total;
#pragma unroll
      for (int w = 0; w < kBlockWarps; ++w) {
        f.base[lane][w] = at;
        at += __popc(f.hits[lane][w]);
      }
    }
    if (exists) lists.counts[(int64_t)k * lists.nblk + blk] = total;
  }
  __syncthreads();
  int32_t* value = lists.value + (int64_t)blk * kIdxThreads * g.kvol;
  uint8_t* local = lists.local + (int64_t)blk * kIdxThreads * g.kvol;
  for (uint32_t rest = mask; rest; rest &= rest - 1u) {
    const int q = __ffs(rest) - 1;
    const int pos = f.base[q][warp] + __popc(f.hits[q][warp] & lanemask_lt());
    value[pos] = f.values[q][threadIdx.x];
    local[pos] = (uint8_t)threadIdx.x;
  }
}

// The block's part of the neighbour tables but for the ids: the ballots as row masks, offset masks per tile, and the
// identity output map.  A block covers two tiles of 128.
__device__ __forceinline__ void write_target_masks(const uint32_t (&hits)[kTaps3][kBlockWarps], const Targets& targets,
                                                   int64_t n_max) {
  const int64_t tile0 = (int64_t)blockIdx.x * (kIdxThreads / 128), pos = tile0 * 128 + threadIdx.x;
  const int tiles_here = (int)min((int64_t)(kIdxThreads / 128), targets.tiles - tile0);
  for (int q = 0; q < targets.count; ++q) {
    const TableTarget& t = targets.t[q];
    if ((int)threadIdx.x < tiles_here * 128) t.perm[pos] = pos < n_max ? (int32_t)pos : -1;
    // rows[tile][slot][4]: consecutive words across the block's tiles
    uint32_t* rows = t.rows + tile0 * t.kvol * 4;
    for (int w = threadIdx.x; w < tiles_here * t.kvol * 4; w += kIdxThreads) {
      const int tl = w / (t.kvol * 4), s = w / 4 % t.kvol, quarter = w & 3;
      rows[w] = hits[t.g_of_slot[s]][tl * 4 + quarter];
    }
    if ((int)threadIdx.x < tiles_here) {
      uint32_t any = 0u;
      for (int s = 0; s < t.kvol; ++s) {
        const uint32_t* h = &hits[t.g_of_slot[s]][threadIdx.x * 4];
        if (h[0] | h[1] | h[2] | h[3]) any |= 1u << s;
      }
      t.mask[tile0 + threadIdx.x] = any;
    }
  }
}

// The ids of a submanifold pass's block in its columns, where a neighbour exists (nothing needs initialising).
__device__ __forceinline__ void write_targets(const Found& f, uint32_t mask, const Targets& targets, int64_t n_max) {
  write_target_masks(f.hits, targets, n_max);
  const int64_t pos = (int64_t)blockIdx.x * kIdxThreads + threadIdx.x, tile = pos >> 7;
  if (tile >= targets.tiles) return;
  for (int q = 0; q < targets.count; ++q) {
    const TableTarget& t = targets.t[q];
    int32_t* col = t.ids + tile * t.kvol * 128 + (pos & 127);
#pragma unroll
    for (int g = 0; g < kTaps3; ++g)
      if (((mask >> g) & 1u) && t.slot_of_g[g] >= 0) col[t.slot_of_g[g] * 128] = f.values[g][threadIdx.x];
  }
}

// A block without a live voxel: its tiles take part in no offset.
__device__ __forceinline__ void write_empty_targets(const Targets& targets, int64_t n_max) {
  const int64_t tile0 = (int64_t)blockIdx.x * (kIdxThreads / 128);
  const int tiles_here = (int)min((int64_t)(kIdxThreads / 128), targets.tiles - tile0);
  if (tiles_here <= 0) return;
  const int64_t pos = tile0 * 128 + threadIdx.x;
  for (int q = 0; q < targets.count; ++q) {
    const TableTarget& t = targets.t[q];
    if ((int)threadIdx.x < tiles_here * 128) t.perm[pos] = pos < n_max ? (int32_t)pos : -1;
    for (int w = threadIdx.x; w < tiles_here * t.kvol * 4; w += kIdxThreads) t.rows[tile0 * t.kvol * 4 + w] = 0u;
    if ((int)threadIdx.x < tiles_here) t.mask[tile0 + threadIdx.x] = 0u;
  }
}

// Submanifold neighbours: the voxel at coor + pad - tap * dilation for every tap (trt/spconv/index.cu:48-84), one thread
// per voxel.  kDirect: 27 independent loads from the grid.  Otherwise nine words of the bit map (one per (z, y) row; a
// second one where the taps straddle a word), then the hash slots of the hits, four in flight.
// lists.value == null: no rulebook is wanted, only the tables.
template <bool kDirect>
__global__ void __launch_bounds__(kIdxThreads)
subm_find3_kernel(const Lookup3 look, const int32_t* __restrict__ coors, const int32_t* num_act_in, int64_t n_max,
                  const Geometry g, const PairLists lists, const Targets targets) {
  __shared__ Found f;
  pdl_release();
  pdl_wait();
  const int n = live_count(num_act_in, n_max);
  if ((int64_t)blockIdx.x * kIdxThreads >= n) {
    write_empty_targets(targets, n_max);
    return;
  }
  const int i = blockIdx.x * kIdxThreads + threadIdx.x;
  int4 c = make_int4(-1, 0, 0, 0);
  if (i < n) c = __ldg(reinterpret_cast<const int4*>(coors) + i);
  const bool batch_ok = (uint32_t)c.x < (uint32_t)g.shape[0];
  const int b0 = c.y + g.pad[0], b1 = c.z + g.pad[1], b2 = c.w + g.pad[2];
  const uint32_t s1 = (uint32_t)g.shape[1], s2 = (uint32_t)g.shape[2], s3 = (uint32_t)g.shape[3];
  const uint32_t key0 = (((uint32_t)c.x * s1 + (uint32_t)b0) * s2 + (uint32_t)b1) * s3 + (uint32_t)b2;
  const uint32_t step0 = (uint32_t)g.dil[0] * s2 * s3, step1 = (uint32_t)g.dil[1] * s3, step2 = (uint32_t)g.dil[2];
  uint32_t mask = 0u;
  if (kDirect) {
    int v[kTaps3];
#pragma unroll
    for (int q = 0; q < kTaps3; ++q) {
      const int a = q / 9, b = q / 3 % 3, t = q % 3;
      const bool ok = batch_ok && a < g.ksize[0] && b < g.ksize[1] && t < g.ksize[2] &&
                      (uint32_t)(b0 - a * g.dil[0]) < s1 && (uint32_t)(b1 - b * g.dil[1]) < s2 &&
                      (uint32_t)(b2 - t * g.dil[2]) < s3;
      v[q] = __ldg(look.direct + (ok ? key0 - a * step0 - b * step1 - t * step2 : 0u));  // always a load: all in flight
      if (!ok) v[q] = -1;
    }
#pragma unroll
    for (int q = 0; q < kTaps3; ++q) {
      if (v[q] >= 0) mask |= 1u << q;
      f.values[q][threadIdx.x] = v[q];
    }
  } else {
    // the x taps of a row span [lo, hi] inside the grid; bit j of a row's window is x = lo + j (2 * dilation < 32)
    const int lo = max(b2 - (g.ksize[2] - 1) * g.dil[2], 0), hi = min(b2, (int)s3 - 1);
    uint32_t window[9];
#pragma unroll
    for (int r = 0; r < 9; ++r) {
      const int a = r / 3, b = r % 3;
      window[r] = 0u;
      if (batch_ok && lo <= hi && a < g.ksize[0] && b < g.ksize[1] && (uint32_t)(b0 - a * g.dil[0]) < s1 &&
          (uint32_t)(b1 - b * g.dil[1]) < s2) {
        const uint32_t p = key0 - a * step0 - b * step1 - (uint32_t)(b2 - lo);
        const uint32_t w0 = __ldg(look.bits + (p >> 5));
        const uint32_t last = (p + (uint32_t)(hi - lo)) >> 5;
        const uint32_t w1 = last != (p >> 5) ? __ldg(look.bits + last) : 0u;
        window[r] = __funnelshift_r(w0, w1, p & 31);
      }
    }
#pragma unroll
    for (int q = 0; q < kTaps3; ++q) {
      const int t = q % 3, x = b2 - t * g.dil[2];
      if (t < g.ksize[2] && x >= lo && x <= hi && ((window[q / 3] >> (x - lo)) & 1u)) mask |= 1u << q;
    }
    const uint32_t cap = hash_capacity((long long)n * kSubmFan, look.cap_max) - 1;
    for (uint32_t rest = mask; rest;) {
      constexpr int kFlight = 4;
      int q[kFlight];
      uint32_t key[kFlight];
      unsigned long long first[kFlight];
#pragma unroll
      for (int e = 0; e < kFlight; ++e) {
        q[e] = rest ? __ffs(rest) - 1 : -1;
        rest &= rest - 1u;
        key[e] = key0 - (uint32_t)(q[e] / 9) * step0 - (uint32_t)(q[e] / 3 % 3) * step1 - (uint32_t)(q[e] % 3) * step2;
        if (q[e] >= 0) first[e] = __ldg(look.slots + home_slot(key[e], cap));
      }
#pragma unroll
      for (int e = 0; e < kFlight; ++e) {
        if (q[e] < 0) continue;
        const int v = hash_lookup_resolve(look.slots, cap, key[e], first[e]);
        if (v < 0) mask &= ~(1u << q[e]);  // a voxel the full hash table had no slot for
        f.values[q[e]][threadIdx.x] = v;
      }
    }
  }
  publish_hits(f, mask);
  write_targets(f, mask, targets, n_max);
  if (lists.value) write_lists(f, g, mask, lists);
}

// The rulebook from the lists: a block copies its runs to their places in the segments, and the blocks behind the last
// one fill the padding.  grid: nblk + fill blocks.
__global__ void __launch_bounds__(kIdxThreads)
emit_index3_kernel(const PairLists lists, const int32_t* __restrict__ seg, const int32_t* num_act_in, int64_t n_max,
                   int kvol, int32_t* __restrict__ index, int64_t row_len, const int32_t* __restrict__ state) {
  __shared__ int first[32], place[32];  // of every offset: start in the list, start in the index
  pdl_release();
  pdl_wait();
  const int nblk = lists.nblk, blk = blockIdx.x;
  if (blk >= nblk) {
    fill_padding(seg, kvol, index, row_len, state, (int64_t)(blk - nblk) * kIdxThreads + threadIdx.x,
                 (int64_t)(gridDim.x - nblk) * kIdxThreads);
    return;
  }
  const int n = live_count(num_act_in, n_max);
  if ((int64_t)blk * kIdxThreads >= n) return;
  const int live_blk = (n + kIdxThreads - 1) / kIdxThreads;
  if (threadIdx.x < 32) {
    const int k = threadIdx.x;
    int start = 0, count = 0;
    if (k < kvol) {
      const int32_t* row = lists.counts + (int64_t)k * nblk;  // exclusive prefix by now
      start = row[blk];
      count = (blk + 1 < live_blk ? row[blk + 1] : seg[kvol + 1 + k]) - start;
      place[k] = seg[k] + start;
    }
    int inc = count;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, d);
      if (k >= d) inc += t;
    }
    first[k] = inc - count;
    if (k == 31) place[31] = inc;  // kvol <= 27: the last word holds the total
  }
  __syncthreads();
  const int total = place[31];
  const int32_t* value = lists.value + (int64_t)blk * kIdxThreads * kvol;
  const uint8_t* local = lists.local + (int64_t)blk * kIdxThreads * kvol;
  for (int e = threadIdx.x; e < total; e += kIdxThreads) {
    int k = 0;  // the last offset whose run starts at or before e (empty runs share their start with the next one)
#pragma unroll
    for (int step = 16; step; step >>= 1)
      if (k + step < kvol && first[k + step] <= e) k += step;
    const int64_t pos = (int64_t)place[k] + (e - first[k]);
    if (pos < row_len) {
      index[pos] = blk * kIdxThreads + local[e];
      index[row_len + pos] = value[e];
      index[2 * row_len + pos] = k;
    }
  }
}

// ---- strided and transposed rulebooks over the grid itself --------------------------------------------------------------
// The taps of an input that reach an output, per axis and ascending: at most kTaps of three (two when the stride is at
// least two), so that kTaps^3 combinations are all there are.
template <int kTaps> struct Taps {
  int count[3], out[3][kTaps], tap[3][kTaps];
};
template <int kTaps> __device__ __forceinline__ Taps<kTaps> taps_of(const Geometry& g, const int4& c, bool live) {
  Taps<kTaps> t;
  const int in[3] = {c.y, c.z, c.w};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    t.count[d] = 0;
#pragma unroll
    for (int e = 0; e < kTaps; ++e) t.out[d][e] = t.tap[d][e] = 0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      int o;
      if (!(live && j < g.ksize[d] && out_coord(g, d, in[d], j, &o))) continue;
#pragma unroll
      for (int e = 0; e < kTaps; ++e)
        if (e == t.count[d]) t.out[d][e] = o, t.tap[d][e] = j;
      ++t.count[d];
    }
  }
  return t;
}
// Combination e (in ascending order of the kernel offset): whether it exists, its cell, its offset.
template <int kTaps> struct Combo {
  bool ok;
  int x[3];     // output coordinates
  int tap[3];
};
template <int kTaps> __device__ __forceinline__ Combo<kTaps> combo(const Taps<kTaps>& t, int e) {
  const int pick[3] = {e / (kTaps * kTaps), e / kTaps % kTaps, e % kTaps};
  Combo<kTaps> r;
  r.ok = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    r.ok = r.ok && pick[d] < t.count[d];
    r.x[d] = t.out[d][pick[d]], r.tap[d] = t.tap[d][pick[d]];
  }
  return r;
}
template <int kTaps> __device__ __forceinline__ uint32_t cell_of(const Geometry& g, const Combo<kTaps>& r, int batch) {
  return (((uint32_t)batch * (uint32_t)g.shape[1] + (uint32_t)r.x[0]) * (uint32_t)g.shape[2] + (uint32_t)r.x[1]) *
             (uint32_t)g.shape[3] + (uint32_t)r.x[2];
}
template <int kTaps> __device__ __forceinline__ int offset_of(const Geometry& g, const Combo<kTaps>& r) {
  return (r.tap[0] * g.ksize[1] + r.tap[1]) * g.ksize[2] + r.tap[2];
}

// Row `id` of the output coordinates: one store where the rows start on 16 bytes (`rows16`), else four -- the buffer is the
// caller's, maybe a piece of an arena of words.
__device__ __forceinline__ bool rows_on_16_bytes(const int32_t* out_coors) {
  return (reinterpret_cast<uintptr_t>(out_coors) & 15) == 0;
}
__device__ __forceinline__ void store_coor(int32_t* __restrict__ out_coors, bool rows16, int64_t id, const int4& c) {
  if (rows16) {
    reinterpret_cast<int4*>(out_coors)[id] = c;
  } else {
    int32_t* row = out_coors + id * 4;
    row[0] = c.x, row[1] = c.y, row[2] = c.z, row[3] = c.w;
  }
}

// Every candidate pair (input i, offset k) leaves i * kvol + k in its output's cell if it is the smallest so far.
template <int kTaps>
__global__ void __launch_bounds__(kIdxThreads)
conv_mark3_kernel(int32_t* __restrict__ grid, const int32_t* __restrict__ coors, const int32_t* num_act_in,
                  int64_t n_max, const Geometry g) {
  pdl_release();
  pdl_wait();
  const int n = live_count(num_act_in, n_max);
  const int i = blockIdx.x * kIdxThreads + threadIdx.x;
  if (i >= n) return;
  const int4 c = __ldg(reinterpret_cast<const int4*>(coors) + i);
  if ((uint32_t)c.x >= (uint32_t)g.shape[0]) return;
  const Taps<kTaps> t = taps_of<kTaps>(g, c, true);
#pragma unroll
  for (int e = 0; e < kTaps * kTaps * kTaps; ++e) {
    const Combo<kTaps> r = combo(t, e);
    if (r.ok)
      atomicMin(reinterpret_cast<unsigned*>(grid) + cell_of(g, r, c.x), (unsigned)(i * g.kvol + offset_of(g, r)));
  }
}

// Cells after numbering: an output's id with the sign bit set, or kDropped beyond maxNumActOut.
constexpr int kDropped = -2;
constexpr int kIdBit = -2147483647 - 1;

// The pair whose id is left in a cell numbers that output: in pair order, i.e. by first touch (index.cu:104-121).  First
// the winning combinations of every input and their number per block, then the numbers themselves.
template <int kTaps>
__global__ void __launch_bounds__(kIdxThreads)
conv_count3_kernel(const int32_t* __restrict__ grid, const int32_t* __restrict__ coors, const int32_t* num_act_in,
                   int64_t n_max, const Geometry g, uint32_t* __restrict__ wins, int32_t* __restrict__ counts) {
  __shared__ int sums[kBlockWarps];
  pdl_release();
  pdl_wait();
  const int n = live_count(num_act_in, n_max);
  if ((int64_t)blockIdx.x * kIdxThreads >= n) return;
  const int i = blockIdx.x * kIdxThreads + threadIdx.x;
  int4 c = make_int4(-1, 0, 0, 0);
  if (i < n) c = __ldg(reinterpret_cast<const int4*>(coors) + i);
  constexpr int kCombos = kTaps * kTaps * kTaps;
  const Taps<kTaps> t = taps_of<kTaps>(g, c, (uint32_t)c.x < (uint32_t)g.shape[0]);
  int32_t left[kCombos];
#pragma unroll
  for (int e = 0; e < kCombos; ++e) {
    const Combo<kTaps> r = combo(t, e);
    left[e] = r.ok ? __ldg(grid + cell_of(g, r, c.x)) : -1;
  }
  uint32_t bits = 0u;
#pragma unroll
  for (int e = 0; e < kCombos; ++e)
    if (left[e] >= 0 && left[e] == i * g.kvol + offset_of(g, combo(t, e))) bits |= 1u << e;
  if (i < n) wins[i] = bits;
  const int sum = __reduce_add_sync(0xffffffffu, __popc(bits));
  if (lane_id() == 0) sums[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    int total = 0;
    for (int w = 0; w < kBlockWarps; ++w) total += sums[w];
    counts[blockIdx.x] = total;
  }
}

template <int kTaps>
__global__ void __launch_bounds__(kIdxThreads)
conv_number3_kernel(int32_t* __restrict__ grid, const int32_t* __restrict__ coors, const int32_t* num_act_in,
                    int64_t n_max, const Geometry g, int32_t max_out, const uint32_t* __restrict__ wins,
                    const int32_t* __restrict__ counts, bool scanned, int32_t* __restrict__ out_coors,
                    int32_t* __restrict__ num_act_out, int32_t* status) {
  __shared__ int scratch[40], sums[kBlockWarps];
  pdl_release();
  pdl_wait();
  const int n = live_count(num_act_in, n_max);
  if (n == 0 && blockIdx.x == 0 && threadIdx.x == 0) *num_act_out = 0;
  if ((int64_t)blockIdx.x * kIdxThreads >= n) return;
  const int i = blockIdx.x * kIdxThreads + threadIdx.x;
  const uint32_t bits = i < n ? __ldg(wins + i) : 0u;
  int4 c = make_int4(-1, 0, 0, 0);
  if (bits) c = __ldg(reinterpret_cast<const int4*>(coors) + i);
  const int base = preceding_sum<kIdxThreads>(counts, blockIdx.x, scanned, sums);
  int total;
  int id = base + block_exclusive_scan(__popc(bits), scratch, &total);
  if (threadIdx.x == 0 && ((int64_t)blockIdx.x + 1) * kIdxThreads >= n) {
    const long long all = (long long)base + total;  // the last live block knows the number of outputs
    *num_act_out = (int32_t)(all < max_out ? all : max_out);
    if (all > max_out) report_status(status, D3D_STATUS_OUTPUT_OVERFLOW);
  }
  if (!bits) return;
  const bool rows16 = rows_on_16_bytes(out_coors);
  constexpr int kCombos = kTaps * kTaps * kTaps;
  const Taps<kTaps> t = taps_of<kTaps>(g, c, true);
#pragma unroll
  for (int e = 0; e < kCombos; ++e) {
    if (!((bits >> e) & 1u)) continue;
    const Combo<kTaps> r = combo(t, e);
    if (id < max_out) {
      grid[cell_of(g, r, c.x)] = kIdBit | id;
      store_coor(out_coors, rows16, id, make_int4(c.x, r.x[0], r.x[1], r.x[2]));
    } else {
      grid[cell_of(g, r, c.x)] = kDropped;  // the pairs of this output are dropped (index.cu:158-172)
    }
    ++id;
  }
}

// The pairs of the numbered outputs as lists for the rulebook.  kFindSpare: shared memory asked for on top, which keeps an SM
// from taking more than four blocks -- launched ahead of their turn they settle wherever the kernel in front has left
// room, and a few hundred blocks then crowd on some SMs (120 k inputs: 31 us with eight to an SM, 20 with four).  Launched
// plainly the limit costs nothing (rulebook with persistent buffers, with / without it: 35.8 / 35.8 us at 30 k inputs,
// 45.8 / 45.8 at 120 k, 61.8 / 63.3 at 280 k), so it is the same there.
constexpr int kFindSpare = 18 * 1024;
template <int kTaps>
__global__ void __launch_bounds__(kIdxThreads)
conv_find3_kernel(const int32_t* __restrict__ grid, const int32_t* __restrict__ coors, const int32_t* num_act_in,
                  int64_t n_max, const Geometry g, const PairLists lists) {
  __shared__ Found f;
  pdl_release();
  pdl_wait();
  const int n = live_count(num_act_in, n_max);
  if ((int64_t)blockIdx.x * kIdxThreads >= n) return;
  const int i = blockIdx.x * kIdxThreads + threadIdx.x;
  int4 c = make_int4(-1, 0, 0, 0);
  if (i < n) c = __ldg(reinterpret_cast<const int4*>(coors) + i);
  constexpr int kCombos = kTaps * kTaps * kTaps;
  const Taps<kTaps> t = taps_of<kTaps>(g, c, (uint32_t)c.x < (uint32_t)g.shape[0]);
  int32_t id[kCombos];
#pragma unroll
  for (int e = 0; e < kCombos; ++e) {
    const Combo<kTaps> r = combo(t, e);
    id[e] = __ldg(grid + (r.ok ? cell_of(g, r, c.x) : 0u));  // always a load: all are in flight together
    if (!r.ok) id[e] = kDropped;
  }
  uint32_t mask = 0u;
#pragma unroll
  for (int e = 0; e < kCombos; ++e) {
    if (id[e] == kDropped) continue;
    const Combo<kTaps> r = combo(t, e);
    const int q = (r.tap[0] * 3 + r.tap[1]) * 3 + r.tap[2];
    mask |= 1u << q;
    f.values[q][threadIdx.x] = id[e] & ~kIdBit;
  }
  publish_hits(f, mask);
  write_lists(f, g, mask, lists);
}

}  // namespace
}  // namespace d3d
