// SimpleMeanEncoder and CylinderEncoder: point cloud -> voxels.
//
// Replace voxel_encoder::func::simpleMeanEncoder (trt/voxel_encoder/simple_mean_trt.cu:121-168, kernels :28-102)
// and voxel_encoder::func::CylinderEncoder (trt/voxel_encoder/cylinder_trt.cu:130-174, kernels :28-111).
// Both share one scheme: each point leaves its own index in its voxel's slot (the smallest index survives); the points
// that "own" their voxel are counted per block and numbered in point order, which numbers the voxels by first touch; a
// last pass brings the other points in.  The reference numbers voxels by hash-slot rank (a scan over the whole 2N-slot
// table) instead.
//
// What bounds them: a dozen megabytes of traffic behind a chain of dependent kernels, so the number of passes and the
// round trips inside each.  Nine of ten points own their voxel in a 10-sweep cloud: the numbering pass writes their
// features, coordinates and counts itself, and only the rest go through atomics.  A slot is a cell of the grid where
// that is small enough (a point then needs one result-less atomicMin), else a hash slot.
#include <math.h>

#include "common.cuh"

namespace d3d {
namespace {

constexpr int kEncThreads = 256;

// Where the voxels are: `grid` (one word per cell: -1, then the smallest point index, then kNumbered | voxel id or
// kDropped) or `slots` (key << 32 | the same word).
struct Voxels {
  int32_t* grid;
  unsigned long long* slots;
  uint32_t cap_mask;
};
constexpr int32_t kNumbered = -2147483647 - 1;
constexpr int32_t kDropped = -2;  // beyond maxNumActOut

__global__ void __launch_bounds__(256) enc_clear_kernel(uint4* table, int64_t n16) {
  pdl_release();
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (int64_t)gridDim.x * blockDim.x;
  const uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u);
  for (int64_t i = tid; i < n16; i += nth) table[i] = ones;
}

// Leaves point `i` in the voxel of `key`; returns the slot, or -1 when the hash table is full.
__device__ __forceinline__ int claim(const Voxels& v, uint32_t key, uint32_t i, int32_t* status) {
  if (v.grid) {
    atomicMin(reinterpret_cast<unsigned*>(v.grid) + key, i);
    return (int)key;
  }
  const uint32_t s = hash_insert_min_scattered(v.slots, v.cap_mask, key, i);
  if (s == 0xFFFFFFFFu) report_status(status, D3D_STATUS_HASH_FULL);
  return s == 0xFFFFFFFFu ? -1 : (int)s;
}
__device__ __forceinline__ int32_t voxel_word(const Voxels& v, int slot) {
  return v.grid ? __ldcg(v.grid + slot) : (int32_t)(uint32_t)__ldcg(v.slots + slot);
}
// Voxel id of a slot after numbering, or -1.
__device__ __forceinline__ int voxel_id(const Voxels& v, int slot) {
  const int32_t w = voxel_word(v, slot);
  return w == kDropped ? -1 : w & ~kNumbered;
}

__device__ __forceinline__ bool all_finite(const float* __restrict__ p, int c) {
  bool ok = true;
  for (int f = 0; f < c; ++f) ok = ok && isfinite(p[f]);
  return ok;
}

// trt/voxel_encoder/simple_mean_trt.cu:28-60: truncation toward zero, bounds check, insert.
__global__ void __launch_bounds__(kEncThreads)
voxelize_kernel(const Voxels vox, const float* __restrict__ pts,
                                const int32_t* __restrict__ batch, const float* __restrict__ cfg, int64_t n, int c,
                                int sb, int sz, int sy, int sx, int32_t* __restrict__ slot_of, int32_t* status) {
  pdl_release();
  pdl_wait();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* p = pts + i * c;
  int slot = -1;
  int b = batch[i];
  if (all_finite(p, c) && b >= 0 && b < sb) {
    int cx = (int)__fdiv_rn(__fsub_rn(p[0], cfg[0]), cfg[3]);
    int cy = (int)__fdiv_rn(__fsub_rn(p[1], cfg[1]), cfg[4]);
    int cz = (int)__fdiv_rn(__fsub_rn(p[2], cfg[2]), cfg[5]);
    if (cx >= 0 && cx < sx && cy >= 0 && cy < sy && cz >= 0 && cz < sz) {
      uint32_t key = (((uint32_t)b * sz + cz) * sy + cy) * sx + cx;
      slot = claim(vox, key, (uint32_t)i, status);
    }
  }
  slot_of[i] = slot;
}

// trt/voxel_encoder/cylinder_trt.cu:28-85.  cfg = (zmin, phimin, rhomin, zmax, phimax, rhomax), dims (rho, phi, z).
// The augmented rows of a block are put together in shared memory (`staged`: kEncThreads * (c + 5) floats) and leave as
// one contiguous run; rows too wide for that are written in place.
template <bool kStaged>
__global__ void __launch_bounds__(kEncThreads)
cylinderize_kernel(const Voxels vox, const float* __restrict__ pts, const int32_t* __restrict__ batch,
                   const float* __restrict__ cfg, int64_t n, int c, int sb, int sr, int sp, int sz,
                   int32_t* __restrict__ slot_of, float* __restrict__ aug) {
  extern __shared__ float staged[];
  pdl_release();
  pdl_wait();
  const int64_t i0 = (int64_t)blockIdx.x * kEncThreads, i = i0 + threadIdx.x;
  const int w = c + 5;
  if (i < n) {
    const float* p = pts + i * c;
    float* a = kStaged ? staged + threadIdx.x * w : aug + i * w;
    int slot = -1;
    bool wrote = false;
    if (all_finite(p, c)) {
      int b = batch[i];
      float x = p[0], y = p[1], z = p[2];
      float rho = sqrtf(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)));
      float phi = atan2f(y, x);
      if (b >= 0 && b < sb) {
        float zmin = cfg[0], pmin = cfg[1], rmin = cfg[2];
        float zs = __fdiv_rn(__fsub_rn(cfg[3], cfg[0]), (float)sz);
        float ps = __fdiv_rn(__fsub_rn(cfg[4], cfg[1]), (float)sp);
        float rs = __fdiv_rn(__fsub_rn(cfg[5], cfg[2]), (float)sr);
        int zc = (int)__fdiv_rn(__fsub_rn(z, zmin), zs);
        int pc = (int)__fdiv_rn(__fsub_rn(phi, pmin), ps);
        int rc = (int)__fdiv_rn(__fsub_rn(rho, rmin), rs);
        if (pc >= 0 && pc < sp && rc >= 0 && rc < sr) {
          zc = zc < 0 ? 0 : zc;  // z is clamped, not dropped (cylinder_trt.cu:64-66)
          zc = zc >= sz ? sz - 1 : zc;
          uint32_t key = (((uint32_t)b * sr + rc) * sp + pc) * sz + zc;
          slot = claim(vox, key, (uint32_t)i, nullptr);
          a[0] = z;
          a[1] = phi;
          a[2] = rho;
          a[3] = z - ((zc + 0.5f) * zs + zmin);
          a[4] = phi - ((pc + 0.5f) * ps + pmin);
          a[5] = rho - ((rc + 0.5f) * rs + rmin);
          a[6] = x;
          a[7] = y;
          for (int f = 3; f < c; ++f) a[f + 5] = p[f];
          wrote = true;
        }
      }
    }
    if (!wrote)
      for (int f = 0; f < w; ++f) a[f] = 0.f;  // the reference memsets the tensor (cylinder_trt.cu:162)
    slot_of[i] = slot;
  }
  if (kStaged) {
    __syncthreads();
    const int64_t total = (n - i0 < kEncThreads ? n - i0 : kEncThreads) * w;
    for (int64_t e = threadIdx.x; e < total; e += kEncThreads) aug[i0 * w + e] = staged[e];
  }
}

// Finds the owners and counts them per block; an owner's slot_of becomes owner_mark(slot).
constexpr int kOwner = -2;
__device__ __forceinline__ int owner_mark(int slot) { return -3 - slot; }  // its own inverse; <= -3 for slots
__global__ void __launch_bounds__(kEncThreads)
count_owners_kernel(const Voxels vox, int32_t* __restrict__ slot_of, int64_t n, int32_t* __restrict__ owners) {
  pdl_release();
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * kEncThreads + threadIdx.x;
  const int slot = i < n ? slot_of[i] : -1;
  const bool owner = slot >= 0 && voxel_word(vox, slot) == (int32_t)i;
  if (owner) slot_of[i] = owner_mark(slot);
  const int total = __syncthreads_count(owner);
  if (threadIdx.x == 0) owners[blockIdx.x] = total;
}

// Owners number their voxel in point order and write what they know of it: the coordinates (decoded from the key, last
// extent fastest), the point count (so far one) and, for the mean encoder, their features as the sum so far; for the
// cylinder encoder their own entry of the point -> voxel map.  An owner's slot_of becomes kOwner: it is done.
template <bool kMean>
__global__ void __launch_bounds__(kEncThreads)
number_voxels_kernel(const Voxels vox, int32_t* __restrict__ slot_of, int64_t n, int64_t m_max, int e1, int e2, int e3,
                     const int32_t* __restrict__ owners, bool scanned, const float* __restrict__ pts, int c,
                     int32_t* __restrict__ out_coors, int32_t* __restrict__ count, float* __restrict__ out_feats,
                     int32_t* __restrict__ scatter_to, int32_t* __restrict__ num_act_out, int32_t* status) {
  __shared__ int scratch[40], sums[kEncThreads / 32];
  pdl_release();
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * kEncThreads + threadIdx.x;
  const int mark = i < n ? slot_of[i] : -1;
  const bool owner = mark <= -3;
  const int slot = owner_mark(mark);
  const uint32_t key = !owner ? 0u : vox.grid ? (uint32_t)slot : (uint32_t)(__ldcg(vox.slots + slot) >> 32);
  const int base = preceding_sum<kEncThreads>(owners, blockIdx.x, scanned, sums);
  int total;
  const int rank = block_exclusive_scan(owner, scratch, &total);
  if (threadIdx.x == 0 && blockIdx.x == gridDim.x - 1) {
    const long long all = (long long)base + total;
    *num_act_out = (int32_t)(all < m_max ? all : m_max);
    if (all > m_max) report_status(status, D3D_STATUS_OUTPUT_OVERFLOW);
  }
  if (!owner) return;
  const int64_t vid = (int64_t)base + rank;
  const bool kept = vid < m_max;  // simple_mean_trt.cu:75, cylinder_trt.cu:101
  const int32_t word = kept ? kNumbered | (int32_t)vid : kDropped;
  if (vox.grid) vox.grid[slot] = word;
  else reinterpret_cast<int32_t*>(vox.slots + slot)[0] = word;  // the low half; the key stays
  slot_of[i] = kOwner;
  if (!kMean) scatter_to[i] = kept ? (int32_t)vid : -1;
  if (!kept) return;
  const int c3 = key % e3, k2 = key / e3;
  const int c2 = k2 % e2, k1 = k2 / e2;
  reinterpret_cast<int4*>(out_coors)[vid] = make_int4(k1 / e1, k1 % e1, c2, c3);
  count[vid] = 1;
  if (kMean) {
    const float* p = pts + i * c;
    float* o = out_feats + vid * c;
    for (int f = 0; f < c; ++f) o[f] = p[f];
  }
}

// trt/voxel_encoder/simple_mean_trt.cu:62-91: the points that do not own their voxel join its sum and count.
__global__ void __launch_bounds__(kEncThreads)
mean_accumulate_kernel(const Voxels vox, const int32_t* __restrict__ slot_of, const float* __restrict__ pts, int64_t n,
                       int c, float* __restrict__ out_feats, int32_t* __restrict__ count) {
  pdl_release();
  pdl_wait();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int slot = slot_of[i];
  if (slot < 0) return;
  int vid = voxel_id(vox, slot);
  if (vid < 0) return;
  atomicAdd(&count[vid], 1);
  const float* p = pts + i * c;
  float* o = out_feats + (int64_t)vid * c;
  int f = 0;
  if ((c & 3) == 0) {
    for (; f < c; f += 4) {
      float4 v = *reinterpret_cast<const float4*>(p + f);
      atomicAdd(reinterpret_cast<float4*>(o + f), v);  // one 16-byte reduction per four channels
    }
  }
  for (; f < c; ++f) atomicAdd(o + f, p[f]);
}

// trt/voxel_encoder/simple_mean_trt.cu:93-102: sums to means (a voxel of one point has its mean already), and zero rows
// behind the last voxel.
// With `lp` != null the mean is also written in half / bfloat16 into rows of `lp_c` >= c channels (the extra
// channels zero): the tensor the first sparse convolution reads, without a separate cast-and-pad kernel.
// One thread per voxel; the low-precision row is put together in registers and leaves as 16-byte stores where the row
// width allows.
template <class LP>
__global__ void __launch_bounds__(256)
mean_divide_kernel(float* __restrict__ out_feats, const int32_t* __restrict__ count, const int32_t* num_act_out, int64_t m_max,
                   int c, LP* __restrict__ lp, int lp_c) {
  pdl_release();
  pdl_wait();
  const int n = *num_act_out;
  const bool wide = lp && lp_c % 8 == 0 && (reinterpret_cast<uintptr_t>(lp) & 15) == 0;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = tid; v < n; v += nth) {
    const int members = count[v];
    float* row = out_feats + v * c;
    if (members > 1)
      for (int ch = 0; ch < c; ++ch) row[ch] = __fdiv_rn(row[ch], (float)members);
    if (!lp) continue;
    LP* lrow = lp + v * lp_c;
    if (wide) {
      for (int z0 = 0; z0 < lp_c; z0 += 8) {
        __align__(16) LP h[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) h[q] = LP(z0 + q < c ? row[z0 + q] : 0.f);
        *reinterpret_cast<uint4*>(lrow + z0) = *reinterpret_cast<const uint4*>(h);
      }
    } else {
      for (int z = 0; z < lp_c; ++z) lrow[z] = LP(z < c ? row[z] : 0.f);
    }
  }
  for (int64_t e = (int64_t)n * c + tid; e < m_max * c; e += nth) out_feats[e] = 0.f;
}

// trt/voxel_encoder/cylinder_trt.cu:87-111: the map of the points that do not own their voxel, their share of the
// counts, and zero counts behind the last voxel.
__global__ void __launch_bounds__(kEncThreads)
scatter_ids_kernel(const Voxels vox, const int32_t* __restrict__ slot_of, int64_t n, const int32_t* num_act_out,
                   int64_t m_max, int32_t* __restrict__ scatter_to, int32_t* __restrict__ scatter_count) {
  pdl_release();
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t v = *num_act_out + i; v < m_max; v += (int64_t)gridDim.x * blockDim.x) scatter_count[v] = 0;
  if (i >= n) return;
  const int slot = slot_of[i];
  if (slot == kOwner) return;
  const int vid = slot >= 0 ? voxel_id(vox, slot) : -1;
  scatter_to[i] = vid;
  if (vid >= 0) atomicAdd(&scatter_count[vid], 1);
}

struct EncPlan {
  int64_t n;
  int c;
  int nblk;
  int64_t table_words;  // 32-bit words of the grid or of the hash slots, a multiple of 32
  int dims[4];
  Voxels vox;
  int32_t* slot_of;
  int32_t* owners;
  int32_t* count;
  size_t bytes;
};

int make_enc_plan(const d3d_voxel_encoder_params* p, const d3d_tensor_desc* in, int n_in, void* workspace,
                  bool need_count, EncPlan* plan) {
  D3D_REQUIRE(p && in && n_in >= 4, D3D_ERR_INVALID_ARGUMENT);
  D3D_REQUIRE(in[0].nb_dims == 2 && in[1].nb_dims == 1 && in[3].nb_dims == 5, D3D_ERR_INVALID_ARGUMENT);
  D3D_REQUIRE(in[0].dtype == D3D_FLOAT, D3D_ERR_UNSUPPORTED_DTYPE);
  D3D_REQUIRE(in[1].dims[0] == in[0].dims[0] && p->max_num_act_out >= 0, D3D_ERR_INVALID_ARGUMENT);
  plan->n = in[0].dims[0];
  plan->c = (int)in[0].dims[1];
  D3D_REQUIRE(plan->c >= 3, D3D_ERR_INVALID_ARGUMENT);
  int64_t vol = 1;
  const int src[4] = {0, 2, 3, 4};
  for (int d = 0; d < 4; ++d) {
    plan->dims[d] = (int)in[3].dims[src[d]];
    D3D_REQUIRE(plan->dims[d] >= 1, D3D_ERR_INVALID_ARGUMENT);
    vol *= plan->dims[d];
    D3D_REQUIRE(vol < (1ll << 31), D3D_ERR_TOO_LARGE);
  }
  D3D_REQUIRE(plan->n < (1ll << 30), D3D_ERR_TOO_LARGE);
  plan->nblk = (int)ceil_div(plan->n > 0 ? plan->n : 1, kEncThreads);
  Carver w(workspace);
  // The grid itself while clearing it (4 bytes per cell at 5 TB/s) costs less than hashing the points would, about 0.05 ns
  // each: up to 64 cells per point.
  const bool direct = vol <= 64 * plan->n;
  const uint32_t cap = (uint32_t)next_pow2((size_t)(plan->n > 8 ? plan->n : 8) * 2);
  plan->table_words = direct ? (vol + 63) / 64 * 64 : 2ll * cap;
  int32_t* words = w.take<int32_t>((size_t)plan->table_words);
  plan->vox.grid = direct ? words : nullptr;
  plan->vox.slots = direct ? nullptr : reinterpret_cast<unsigned long long*>(words);
  plan->vox.cap_mask = cap - 1;
  plan->slot_of = w.take<int32_t>(plan->n > 0 ? plan->n : 1);
  plan->owners = w.take<int32_t>(plan->nblk);
  plan->count = need_count ? w.take<int32_t>(p->max_num_act_out > 0 ? p->max_num_act_out : 1) : nullptr;
  plan->bytes = w.off;
  return D3D_OK;
}

uint4* clear_target(const EncPlan& pl) {
  return pl.vox.grid ? reinterpret_cast<uint4*>(pl.vox.grid) : reinterpret_cast<uint4*>(pl.vox.slots);
}

}  // namespace
}  // namespace d3d

using namespace d3d;

static int parse_max_out(const void* data_s, size_t len, d3d_voxel_encoder_params* p) {
  D3D_REQUIRE(data_s && p, D3D_ERR_INVALID_ARGUMENT);
  D3D_REQUIRE(len >= 4, D3D_ERR_BAD_BLOB);
  memcpy(&p->max_num_act_out, data_s, 4);
  return D3D_OK;
}

extern "C" int d3d_simple_mean_encoder_parse(const void* data_s, size_t len, d3d_voxel_encoder_params* p) {
  return parse_max_out(data_s, len, p);
}
extern "C" int d3d_cylinder_encoder_parse(const void* data_s, size_t len, d3d_voxel_encoder_params* p) {
  return parse_max_out(data_s, len, p);
}

extern "C" int d3d_simple_mean_encoder_workspace(const d3d_voxel_encoder_params* p, const d3d_tensor_desc* in,
                                                 int n_in, size_t* bytes) {
  D3D_REQUIRE(bytes, D3D_ERR_INVALID_ARGUMENT);
  EncPlan plan;
  int rc = make_enc_plan(p, in, n_in, nullptr, true, &plan);
  if (rc == D3D_OK) *bytes = plan.bytes;
  return rc;
}
extern "C" int d3d_cylinder_encoder_workspace(const d3d_voxel_encoder_params* p, const d3d_tensor_desc* in, int n_in,
                                              size_t* bytes) {
  D3D_REQUIRE(bytes, D3D_ERR_INVALID_ARGUMENT);
  EncPlan plan;
  int rc = make_enc_plan(p, in, n_in, nullptr, false, &plan);
  if (rc == D3D_OK) *bytes = plan.bytes;
  return rc;
}

// `coors_event` (may be null): recorded where coordinates and count are final.
static int enqueue_mean(const d3d_voxel_encoder_params* p, const d3d_tensor_desc* in, int n_in, const d3d_tensor_desc* out,
                        int n_out, const void* const* inputs, void* const* outputs, void* workspace,
                        size_t workspace_bytes, void* stream, const d3d_mean_encoder_extras* extras,
                        cudaEvent_t coors_event) {
  D3D_REQUIRE(inputs && outputs && out && n_out >= 3, D3D_ERR_INVALID_ARGUMENT);
  void* lp = extras ? extras->lp_feats : nullptr;
  int32_t* status = extras ? extras->status : nullptr;
  D3D_REQUIRE(!lp || ((extras->lp_dtype == D3D_HALF || extras->lp_dtype == D3D_BF16) &&
                      extras->lp_channels >= in[0].dims[1]),
              D3D_ERR_INVALID_ARGUMENT);
  EncPlan pl;
  int rc = make_enc_plan(p, in, n_in, workspace, true, &pl);
  if (rc != D3D_OK) return rc;
  D3D_REQUIRE(workspace && workspace_bytes >= pl.bytes, D3D_ERR_WORKSPACE_TOO_SMALL);
  D3D_REQUIRE(out[0].dims[0] == p->max_num_act_out && out[0].dims[1] == pl.c, D3D_ERR_INVALID_ARGUMENT);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const float* pts = reinterpret_cast<const float*>(inputs[0]);
  const int32_t* batch = reinterpret_cast<const int32_t*>(inputs[1]);
  const float* cfg = reinterpret_cast<const float*>(inputs[2]);
  float* out_feats = reinterpret_cast<float*>(outputs[0]);
  int32_t* out_coors = reinterpret_cast<int32_t*>(outputs[1]);
  int32_t* num_act_out = reinterpret_cast<int32_t*>(outputs[2]);
  const int64_t m_max = p->max_num_act_out;
  if (pl.n == 0) {
    cudaMemsetAsync(num_act_out, 0, sizeof(int32_t), st);
    if (m_max > 0) cudaMemsetAsync(out_feats, 0, (size_t)m_max * pl.c * sizeof(float), st);
    if (coors_event && cudaEventRecord(coors_event, st) != cudaSuccess) return D3D_ERR_CUDA;
    D3D_CHECK_LAUNCH();
    return D3D_OK;
  }
  // a caller with extras runs other work beside this one: its kernels do not wait early for each other
  const bool chained = !extras;
  D3D_LAUNCH(false, enc_clear_kernel, stream_grid(pl.table_words / 16, 256), 256, 0, st, clear_target(pl),
             pl.table_words / 4);
  D3D_LAUNCH(chained, voxelize_kernel, pl.nblk, kEncThreads, 0, st, pl.vox, pts, batch, cfg, pl.n, pl.c, pl.dims[0],
             pl.dims[1], pl.dims[2], pl.dims[3], pl.slot_of, status);
  D3D_LAUNCH(chained, count_owners_kernel, pl.nblk, kEncThreads, 0, st, pl.vox, pl.slot_of, pl.n, pl.owners);
  bool scanned;
  rc = scan_counts(pl.owners, pl.nblk, chained, st, &scanned);
  if (rc != D3D_OK) return rc;
  D3D_LAUNCH(chained, number_voxels_kernel<true>, pl.nblk, kEncThreads, 0, st, pl.vox, pl.slot_of, pl.n, m_max,
             pl.dims[1], pl.dims[2], pl.dims[3], pl.owners, scanned, pts, pl.c, out_coors, pl.count, out_feats, nullptr,
             num_act_out, status);
  if (coors_event && cudaEventRecord(coors_event, st) != cudaSuccess) return D3D_ERR_CUDA;
  if (m_max > 0) {
    D3D_LAUNCH(chained, mean_accumulate_kernel, pl.nblk, kEncThreads, 0, st, pl.vox, pl.slot_of, pts, pl.n, pl.c,
               out_feats, pl.count);
    const int grid = stream_grid(m_max, 256);
    if (lp && extras->lp_dtype == D3D_BF16)
      D3D_LAUNCH(chained, mean_divide_kernel<__nv_bfloat16>, grid, 256, 0, st, out_feats, pl.count, num_act_out, m_max,
                 pl.c, reinterpret_cast<__nv_bfloat16*>(lp), extras->lp_channels);
    else
      D3D_LAUNCH(chained, mean_divide_kernel<__half>, grid, 256, 0, st, out_feats, pl.count, num_act_out, m_max, pl.c,
                 reinterpret_cast<__half*>(lp), lp ? extras->lp_channels : 0);
  }
  D3D_CHECK_LAUNCH();
  return D3D_OK;
}

extern "C" int d3d_simple_mean_encoder_enqueue(const d3d_voxel_encoder_params* p, const d3d_tensor_desc* in, int n_in,
                                               const d3d_tensor_desc* out, int n_out, const void* const* inputs,
                                               void* const* outputs, void* workspace, size_t workspace_bytes,
                                               void* stream) {
  D3D_NVTX_RANGE("d3d_simple_mean_encoder_enqueue");
  return enqueue_mean(p, in, n_in, out, n_out, inputs, outputs, workspace, workspace_bytes, stream, nullptr, nullptr);
}

extern "C" int d3d_simple_mean_encoder_enqueue_ex(const d3d_voxel_encoder_params* p, const d3d_tensor_desc* in, int n_in,
                                                  const d3d_tensor_desc* out, int n_out, const void* const* inputs,
                                                  void* const* outputs, void* workspace, size_t workspace_bytes,
                                                  void* stream, const d3d_mean_encoder_extras* extras) {
  D3D_NVTX_RANGE("d3d_simple_mean_encoder_enqueue_ex");
  return enqueue_mean(p, in, n_in, out, n_out, inputs, outputs, workspace, workspace_bytes, stream, extras, nullptr);
}

extern "C" int d3d_simple_mean_encoder_enqueue_event(const d3d_voxel_encoder_params* p, const d3d_tensor_desc* in, int n_in,
                                                     const d3d_tensor_desc* out, int n_out, const void* const* inputs,
                                                     void* const* outputs, void* workspace, size_t workspace_bytes,
                                                     void* stream, const d3d_mean_encoder_extras* extras,
                                                     void* coors_event) {
  D3D_NVTX_RANGE("d3d_simple_mean_encoder_enqueue_event");
  return enqueue_mean(p, in, n_in, out, n_out, inputs, outputs, workspace, workspace_bytes, stream, extras,
                      reinterpret_cast<cudaEvent_t>(coors_event));
}

extern "C" int d3d_cylinder_encoder_enqueue(const d3d_voxel_encoder_params* p, const d3d_tensor_desc* in, int n_in,
                                            const d3d_tensor_desc* out, int n_out, const void* const* inputs,
                                            void* const* outputs, void* workspace, size_t workspace_bytes,
                                            void* stream) {
  D3D_NVTX_RANGE("d3d_cylinder_encoder_enqueue");
  D3D_REQUIRE(inputs && outputs && out && n_out >= 5, D3D_ERR_INVALID_ARGUMENT);
  EncPlan pl;
  int rc = make_enc_plan(p, in, n_in, workspace, false, &pl);
  if (rc != D3D_OK) return rc;
  D3D_REQUIRE(workspace && workspace_bytes >= pl.bytes, D3D_ERR_WORKSPACE_TOO_SMALL);
  D3D_REQUIRE(out[0].dims[0] == pl.n && out[0].dims[1] == pl.c + 5, D3D_ERR_INVALID_ARGUMENT);
  D3D_REQUIRE(out[2].dims[0] == p->max_num_act_out, D3D_ERR_INVALID_ARGUMENT);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const float* pts = reinterpret_cast<const float*>(inputs[0]);
  const int32_t* batch = reinterpret_cast<const int32_t*>(inputs[1]);
  const float* cfg = reinterpret_cast<const float*>(inputs[2]);
  float* aug = reinterpret_cast<float*>(outputs[0]);
  int32_t* scatter_to = reinterpret_cast<int32_t*>(outputs[1]);
  int32_t* scatter_count = reinterpret_cast<int32_t*>(outputs[2]);
  int32_t* out_coors = reinterpret_cast<int32_t*>(outputs[3]);
  int32_t* num_act_out = reinterpret_cast<int32_t*>(outputs[4]);
  const int64_t m_max = p->max_num_act_out;
  if (pl.n == 0) {
    cudaMemsetAsync(num_act_out, 0, sizeof(int32_t), st);
    if (m_max > 0) cudaMemsetAsync(scatter_count, 0, (size_t)m_max * sizeof(int32_t), st);
    D3D_CHECK_LAUNCH();
    return D3D_OK;
  }
  D3D_LAUNCH(false, enc_clear_kernel, stream_grid(pl.table_words / 16, 256), 256, 0, st, clear_target(pl),
             pl.table_words / 4);
  const size_t staged = (size_t)kEncThreads * (pl.c + 5) * sizeof(float);
  const bool fits = staged <= 40 * 1024;
  D3D_LAUNCH(true, (fits ? cylinderize_kernel<true> : cylinderize_kernel<false>), pl.nblk, kEncThreads,
             fits ? staged : 0, st, pl.vox, pts, batch, cfg, pl.n, pl.c, pl.dims[0], pl.dims[1], pl.dims[2], pl.dims[3],
             pl.slot_of, aug);
  D3D_LAUNCH(true, count_owners_kernel, pl.nblk, kEncThreads, 0, st, pl.vox, pl.slot_of, pl.n, pl.owners);
  bool scanned;
  rc = scan_counts(pl.owners, pl.nblk, true, st, &scanned);
  if (rc != D3D_OK) return rc;
  D3D_LAUNCH(true, number_voxels_kernel<false>, pl.nblk, kEncThreads, 0, st, pl.vox, pl.slot_of, pl.n, m_max, pl.dims[1],
             pl.dims[2], pl.dims[3], pl.owners, scanned, pts, pl.c, out_coors, scatter_count, nullptr, scatter_to, num_act_out,
             nullptr);
  D3D_LAUNCH(true, scatter_ids_kernel, pl.nblk, kEncThreads, 0, st, pl.vox, pl.slot_of, pl.n, num_act_out, m_max,
             scatter_to, scatter_count);
  D3D_CHECK_LAUNCH();
  return D3D_OK;
}
