// Neighbour tables of strided kernels and of everything behind them, without the rulebook: a bit per cell and ranks.
// Included by spconv_index.cu after spconv_index3.cuh.
//
// A rulebook has to number its outputs by first touch, which takes a grid of 4 bytes per cell.  The tables alone do not:
// with the outputs numbered in the order of their cells, an output's id is its rank among the set bits, and
//     words[cell / 32] = {bits, voxels in front of the word}
// answers "is there a voxel, and which" with one 8-byte load, for all the taps of a kernel row at once.  The structure is
// 16 times smaller than the grid of ids (11 M cells: 2.7 MB, all of it in L2), so nothing large is cleared, and since
// neighbouring threads now work on neighbouring voxels their loads share sectors.  What bounds the passes is the latency
// of scattered loads.  B200, detector frame, second level of 463 k voxels: submanifold look-up 65 us from the grid of ids,
// 31 from ranks (beside convolutions); forward table of the third level 30 us by scattering, 21 from its outputs; frames
// 1687 -> 1582 us (300 k points) and 852 -> 756 us (120 k).
#pragma once

namespace d3d {
namespace {

struct RankGrid {
  const uint2* words;
  int shape[4];  // batch and extents of the voxel set
};
__device__ __forceinline__ int rank_of(const uint2& w, uint32_t bit) {  // -1: no voxel
  return (w.x >> bit) & 1u ? (int)w.y + __popc(w.x & ((1u << bit) - 1u)) : -1;
}

// Sets the bit of every output some input reaches; taps along x that fall into one word share an atomic.
template <int kTaps>
__global__ void __launch_bounds__(kIdxThreads)
rank_mark3_kernel(uint2* __restrict__ words, const int32_t* __restrict__ coors, const int32_t* num_act_in, int64_t n_max,
                  const Geometry g) {
  const int n = live_count(num_act_in, n_max);
  const int i = blockIdx.x * kIdxThreads + threadIdx.x;
  if (i >= n) return;
  const int4 c = __ldg(reinterpret_cast<const int4*>(coors) + i);
  if ((uint32_t)c.x >= (uint32_t)g.shape[0]) return;
  const Taps<kTaps> t = taps_of<kTaps>(g, c, true);
#pragma unroll
  for (int e = 0; e < kTaps * kTaps; ++e) {
    uint32_t word = 0u, bits = 0u;
#pragma unroll
    for (int x = 0; x < kTaps; ++x) {
      const Combo<kTaps> r = combo(t, e * kTaps + x);
      if (!r.ok) continue;
      const uint32_t cell = cell_of(g, r, c.x);
      if (bits && cell >> 5 != word) {
        atomicOr(&words[word].x, bits);
        bits = 0u;
      }
      word = cell >> 5, bits |= 1u << (cell & 31);
    }
    if (bits) atomicOr(&words[word].x, bits);
  }
}

// A word a thread: first the voxels of a block, then their ranks and coordinates.
constexpr int kRankWords = 256;
__global__ void __launch_bounds__(kRankWords)
rank_count3_kernel(const uint2* __restrict__ words, int64_t count, int32_t* __restrict__ block_counts) {
  __shared__ int sums[kRankWords / 32];
  const int64_t at = (int64_t)blockIdx.x * kRankWords + threadIdx.x;
  const int sum = __reduce_add_sync(0xffffffffu, at < count ? __popc(words[at].x) : 0);
  if (lane_id() == 0) sums[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    int total = 0;
#pragma unroll
    for (int w = 0; w < kRankWords / 32; ++w) total += sums[w];
    block_counts[blockIdx.x] = total;
  }
}

// Ids beyond max_out have no coordinates; look-ups compare with the count and drop them.  A thread writes the voxels of
// its word one after the other, so what counts on dense levels is a short step: coordinates advance by carries instead of
// divisions, one word a thread instead of four (the deepest level, 2 blocks then: 43 us beside a convolution).
__global__ void __launch_bounds__(kRankWords)
rank_number3_kernel(uint2* __restrict__ words, int64_t count, const int32_t* __restrict__ block_counts, bool scanned, const Geometry g,
                    int32_t max_out, int32_t* __restrict__ out_coors, int32_t* __restrict__ num_act_out,
                    int32_t* status) {
  __shared__ int scratch[40], sums[kRankWords / 32];
  const int64_t at = (int64_t)blockIdx.x * kRankWords + threadIdx.x;
  uint32_t rest = at < count ? words[at].x : 0u;
  const int base = preceding_sum<kRankWords>(block_counts, blockIdx.x, scanned, sums);
  int total;
  int id = base + block_exclusive_scan(__popc(rest), scratch, &total);
  if (threadIdx.x == 0 && blockIdx.x == gridDim.x - 1) {
    const long long all = (long long)base + total;
    *num_act_out = (int32_t)(all < max_out ? all : max_out);
    if (all > max_out) report_status(status, D3D_STATUS_OUTPUT_OVERFLOW);
  }
  if (!rest) return;
  words[at].y = (uint32_t)id;
  const uint32_t s1 = (uint32_t)g.shape[1], s2 = (uint32_t)g.shape[2], s3 = (uint32_t)g.shape[3];
  const uint32_t cell = (uint32_t)(at << 5), row = cell / s3, plane = row / s2;
  uint32_t b = plane / s1, z = plane - b * s1, y = row - plane * s2, x = cell - row * s3;
  const bool rows16 = rows_on_16_bytes(out_coors);
  for (int seen = 0; rest && id < max_out; rest &= rest - 1u, ++id) {
    const int bit = __ffs(rest) - 1;
    x += (uint32_t)(bit - seen), seen = bit;
    while (x >= s3) {
      x -= s3;
      if (++y == s2) {
        y = 0;
        if (++z == s1) z = 0, ++b;
      }
    }
    store_coor(out_coors, rows16, id, make_int4((int)b, (int)z, (int)y, (int)x));
  }
}

// The neighbour a voxel of the walked set has through tap t of axis d lies at coordinate * mul[d] + add[d] + t * step[d]
// of `grid`: the voxels themselves for submanifold kernels, the inputs of a strided one seen from its outputs.  All taps
// of a kernel row lie within two words (|step[2]| < 16).
struct RankWalk {
  RankGrid grid;
  const int32_t* grid_count;  // live voxels of `grid`
  int32_t grid_max;
  int mul[3], add[3], step[3], ksize[3];
};
__global__ void __launch_bounds__(kIdxThreads)
rank_find3_kernel(const RankWalk walk, const int32_t* __restrict__ coors, const int32_t* num_act, int64_t n_max,
                  const Targets targets) {
  __shared__ uint32_t hits[kTaps3][kBlockWarps];
  const int n = live_count(num_act, n_max);
  if ((int64_t)blockIdx.x * kIdxThreads >= n) {
    write_empty_targets(targets, n_max);
    return;
  }
  const int limit = live_count(walk.grid_count, walk.grid_max);
  const int i = blockIdx.x * kIdxThreads + threadIdx.x;
  int4 c = make_int4(-1, 0, 0, 0);
  if (i < n) c = __ldg(reinterpret_cast<const int4*>(coors) + i);
  const bool batch_ok = (uint32_t)c.x < (uint32_t)walk.grid.shape[0];
  const int s1 = walk.grid.shape[1], s2 = walk.grid.shape[2], s3 = walk.grid.shape[3];
  const int z0 = c.y * walk.mul[0] + walk.add[0], y0 = c.z * walk.mul[1] + walk.add[1],
            x0 = c.w * walk.mul[2] + walk.add[2];
  // the cells of a row the taps span
  const int x1 = x0 + (walk.ksize[2] - 1) * walk.step[2];
  const int lo = max(min(x0, x1), 0), hi = min(max(x0, x1), s3 - 1);
  uint2 w0[9], w1[9];
#pragma unroll
  for (int r = 0; r < 9; ++r) {
    const int a = r / 3, b = r % 3, z = z0 + a * walk.step[0], y = y0 + b * walk.step[1];
    w0[r] = w1[r] = make_uint2(0u, 0u);
    if (batch_ok && lo <= hi && a < walk.ksize[0] && b < walk.ksize[1] && (uint32_t)z < (uint32_t)s1 &&
        (uint32_t)y < (uint32_t)s2) {
      const uint32_t row = (((uint32_t)c.x * s1 + z) * s2 + y) * (uint32_t)s3;
      const uint32_t first = (row + lo) >> 5, last = (row + hi) >> 5;
      w0[r] = __ldg(walk.grid.words + first);
      if (last != first) w1[r] = __ldg(walk.grid.words + last);
    }
  }
  int v[kTaps3];
#pragma unroll
  for (int q = 0; q < kTaps3; ++q) {
    const int r = q / 3, x = x0 + q % 3 * walk.step[2];
    const uint32_t row = (((uint32_t)c.x * s1 + (z0 + r / 3 * walk.step[0])) * s2 + (y0 + r % 3 * walk.step[1])) *
                         (uint32_t)s3;
    const uint32_t cell = row + x;
    const uint2 w = cell >> 5 == (row + lo) >> 5 ? w0[r] : w1[r];
    const int id = q % 3 < walk.ksize[2] && x >= lo && x <= hi ? rank_of(w, cell & 31) : -1;
    v[q] = id < limit ? id : -1;
  }
  const int lane = lane_id(), warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < kTaps3; ++q) {
    const unsigned b = __ballot_sync(0xffffffffu, v[q] >= 0);
    if (lane == 0) hits[q][warp] = b;
  }
  __syncthreads();
  write_target_masks(hits, targets, n_max);
  const int64_t pos = (int64_t)blockIdx.x * kIdxThreads + threadIdx.x, tile = pos >> 7;
  if (tile >= targets.tiles) return;
  for (int j = 0; j < targets.count; ++j) {
    const TableTarget& t = targets.t[j];
    int32_t* col = t.ids + tile * t.kvol * 128 + (pos & 127);
#pragma unroll
    for (int q = 0; q < kTaps3; ++q)
      if (v[q] >= 0 && t.slot_of_g[q] >= 0) col[t.slot_of_g[q] * 128] = v[q];
  }
}

// Strided pairs seen from the inputs, for inputs that have no ranks of their own (a forward table by scattering ids and
// row-mask bits) and for the inverse table (inputs gather from outputs; columns like a submanifold table).
template <int kTaps>
__global__ void __launch_bounds__(kIdxThreads)
rank_scatter3_kernel(const uint2* __restrict__ words, const int32_t* __restrict__ num_act_out, int32_t max_out,
                     const int32_t* __restrict__ coors, const int32_t* num_act_in, int64_t n_max, const Geometry g,
                     int32_t* __restrict__ fwd_ids, uint32_t* __restrict__ fwd_rows, const Targets inverse) {
  __shared__ uint32_t hits[kTaps3][kBlockWarps];
  const int n = live_count(num_act_in, n_max);
  if ((int64_t)blockIdx.x * kIdxThreads >= n) {
    write_empty_targets(inverse, n_max);
    return;
  }
  const int limit = live_count(num_act_out, max_out);
  const int i = blockIdx.x * kIdxThreads + threadIdx.x;
  int4 c = make_int4(-1, 0, 0, 0);
  if (i < n) c = __ldg(reinterpret_cast<const int4*>(coors) + i);
  constexpr int kCombos = kTaps * kTaps * kTaps;
  const Taps<kTaps> t = taps_of<kTaps>(g, c, (uint32_t)c.x < (uint32_t)g.shape[0]);
  uint2 w[kCombos];
#pragma unroll
  for (int e = 0; e < kCombos; ++e) {
    const Combo<kTaps> r = combo(t, e);
    w[e] = __ldg(words + (r.ok ? cell_of(g, r, c.x) >> 5 : 0u));  // always a load: all are in flight together
    if (!r.ok) w[e].x = 0u;
  }
  int id[kCombos];
  uint32_t mask = 0u;
#pragma unroll
  for (int e = 0; e < kCombos; ++e) {
    const Combo<kTaps> r = combo(t, e);
    const int o = r.ok ? rank_of(w[e], cell_of(g, r, c.x) & 31) : -1;
    id[e] = o < limit ? o : -1;
    if (id[e] < 0) continue;
    mask |= 1u << ((r.tap[0] * 3 + r.tap[1]) * 3 + r.tap[2]);
    if (fwd_ids) {
      const int64_t blk = (int64_t)(id[e] >> 7) * g.kvol + offset_of(g, r);
      fwd_ids[blk * 128 + (id[e] & 127)] = i;
      atomicOr(fwd_rows + blk * 4 + ((id[e] & 127) >> 5), 1u << (id[e] & 31));
    }
  }
  if (inverse.count == 0) return;
  const int lane = lane_id(), warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < kTaps3; ++q) {
    const unsigned b = __ballot_sync(0xffffffffu, (mask >> q) & 1u);
    if (lane == 0) hits[q][warp] = b;
  }
  __syncthreads();
  write_target_masks(hits, inverse, n_max);
  const int64_t pos = (int64_t)blockIdx.x * kIdxThreads + threadIdx.x, tile = pos >> 7;
  if (tile >= inverse.tiles) return;
  for (int j = 0; j < inverse.count; ++j) {
    const TableTarget& target = inverse.t[j];
    int32_t* col = target.ids + tile * target.kvol * 128 + (pos & 127);
#pragma unroll
    for (int e = 0; e < kCombos; ++e) {
      const Combo<kTaps> r = combo(t, e);
      if (id[e] >= 0) col[target.slot_of_g[(r.tap[0] * 3 + r.tap[1]) * 3 + r.tap[2]] * 128] = id[e];
    }
  }
}

}  // namespace
}  // namespace d3d
