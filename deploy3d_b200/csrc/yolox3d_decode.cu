// YoloX3dDecode: per (batch row, class) the K best BEV cells by class score, decoded into boxes.
//
// Replaces decoder::YoloX3dDecodePlugin of the reference (trt/decoder/yolox3d_decode.cu:147-412): there a
// segmented radix sort of all B*C*Y*X scores (cub, :341-355) followed by one decode launch per class (:357-367).
// Only the first K entries of every sorted segment are ever read, so here one cluster of eight CTAs per (class, batch
// row) selects them directly: each CTA keeps the keys of its eighth of the map in shared memory; a three-pass radix
// select over the cluster's histograms finds the K-th largest key; the cells above it (and, among equal scores, the
// lowest positions, which is what the stable sort of the reference yields) are collected, every CTA ranks an eighth of
// them by counting the larger ones, and decodes its boxes to their ranks.  No workspace, one launch for all classes.
//
// What bounds it: a head has few (class, row) pairs -- six of 180 x 180 cells fill six CTAs of the former one-CTA
// version, which read the map five times, searched its histograms serially and sorted with a barrier per step.  The
// chain that is left is one pass over the map, five cluster barriers and the decode (2 x 3 x 180 x 180, top 500, fp16:
// 62.6 -> 19.7 us).
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <string.h>

#include <atomic>

#include "common.cuh"

namespace d3d {
namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 512;
constexpr int kCluster = 8;     // CTAs per (class, batch row); the largest portable cluster
constexpr int kMaxTopK = 4096;  // candidates are ranked in shared memory
constexpr int kBins = 2048;     // digits of 11, 11 and 10 bits
constexpr int kMaxHeldKeys = 24 * 1024;  // keys a CTA keeps in shared memory; larger maps are read again (from L2)

// Order-preserving map of a float to an unsigned key (larger score = larger key); -0 and +0 share a key.
__device__ __forceinline__ uint32_t score_key(float f) {
  uint32_t u = __float_as_uint(f);
  if ((u << 1) == 0u) u = 0u;
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
template <class T> __device__ __forceinline__ float load_f32(const T* p);
template <> __device__ __forceinline__ float load_f32<float>(const float* p) { return __ldg(p); }
template <> __device__ __forceinline__ float load_f32<__half>(const __half* p) { return __half2float(__ldg(p)); }

struct DecodeArgs {
  const void* cls_scores;  // [B, C, Y, X]
  const void* bbox_preds;  // [B, 9 + a, Y, X]
  const float* pillar_config;
  int num_class, size_y, size_x, box_in_params, topk;
  int stride;
  int class_ids[8];
  int32_t* out_ids[8];  // [B, K]
  float* out_scores[8];  // [B, K]
  float* out_boxes[8];   // [B, K, 7 + a]
};

// Box of BEV cell `pos` (trt/decoder/yolox3d_decode.cu:46-125, same arithmetic in the same precision).
template <class T>
__device__ __forceinline__ void decode_cell(const DecodeArgs& a, const T* preds_b, int pos, float score, int32_t* id_out,
                                            float* score_out, float* box_out, int cls) {
  const int n = a.size_y * a.size_x;
  const float x_min = a.pillar_config[0], y_min = a.pillar_config[1];
  const float feat_stride = static_cast<float>(a.stride) * a.pillar_config[3];
  const float x_base = static_cast<float>(pos % a.size_x), y_base = static_cast<float>(pos / a.size_x);
  const T* pred = preds_b + pos;
  float cx = load_f32(pred) + x_base;
  const bool cx_valid = (cx <= a.size_x && cx >= 0);
  cx = x_min + feat_stride * cx;
  float cy = load_f32(pred + n) + y_base;
  const bool cy_valid = (cy <= a.size_y && cy >= 0);
  cy = y_min + feat_stride * cy;
  float cz = load_f32(pred + 2 * n);
  float dx = feat_stride * expf(load_f32(pred + 3 * n));
  float dy = feat_stride * expf(load_f32(pred + 4 * n));
  float dz = expf(load_f32(pred + 5 * n));
  float yaw = load_f32(pred + 6 * n);
  const float dir_sine = load_f32(pred + 7 * n), dir_cosine = load_f32(pred + 8 * n);
  const float dir = atan2f(dir_sine, dir_cosine);
  const bool yaw_valid = (dir_sine != 0) || (dir_cosine != 0);
  if (!(isfinite(cx) && isfinite(cy) && isfinite(cz) && isfinite(dx) && isfinite(dy) && isfinite(dz) && isfinite(yaw) &&
        dx > 0 && dy > 0 && dz > 0 && yaw_valid && cx_valid && cy_valid)) {
    score = -1.0f;
    cx = cy = cz = 10000.0f;
    dx = dy = dz = 1.f;
    yaw = 0.f;
  } else if (0.9f * dx < dy && dy < 1.11f * dx) {  // nearly square: the direction head decides the heading
    yaw = dir;
    const float t = fmaxf(dx, dy);
    dx = t, dy = t;
  } else {  // elongated: yaw, flipped to the half-plane of the direction head
    if (dy > dx) {
      yaw += M_PI_2;
      const float t = dy;
      dy = dx, dx = t;
    }
    yaw += floorf((dir - yaw) / M_PI + 0.5) * M_PI;
    yaw -= floorf(yaw / (2 * M_PI) + 0.5) * (2 * M_PI);
  }
  *id_out = cls;
  *score_out = score;
  box_out[0] = cx, box_out[1] = cy, box_out[2] = cz, box_out[3] = dx, box_out[4] = dy, box_out[5] = dz, box_out[6] = yaw;
  for (int e = 9; e < a.box_in_params; ++e) box_out[e - 2] = load_f32(pred + (int64_t)e * n);
}

// Cluster rank r owns the cells [r * per, (r + 1) * per).  Dynamic shared memory: candidates [topk], then (kHold) keys.
template <class T, bool kHold>
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kThreads)
topk_decode_kernel(const DecodeArgs a, const int per) {
  extern __shared__ unsigned long long cand[];  // (key << 32) | ~position: descending = the output order
  __shared__ int hist[3][kBins];
  __shared__ int warp_sum[kThreads / 32];
  __shared__ int sel_digit, sel_need, n_greater;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c = blockIdx.x / kCluster, b = blockIdx.y;
  const int n = a.size_y * a.size_x, k_out = a.topk;
  const T* scores = reinterpret_cast<const T*>(a.cls_scores) + ((int64_t)b * a.num_class + c) * n;
  const T* preds_b = reinterpret_cast<const T*>(a.bbox_preds) + (int64_t)b * a.box_in_params * n;
  uint32_t* held = reinterpret_cast<uint32_t*>(cand + k_out);
  const int first = min(rank * per, n), count = min(per, n - first);
  auto key_at = [&](int i) -> uint32_t { return kHold ? held[i] : score_key(load_f32(scores + first + i)); };
  for (int i = tid; i < 3 * kBins; i += kThreads) (&hist[0][0])[i] = 0;
  if (tid == 0) n_greater = 0;
  if (kHold)
    for (int i = tid; i < count; i += kThreads) held[i] = score_key(load_f32(scores + first + i));
  __syncthreads();
  // ---- radix select: after the three passes `prefix` is the K-th largest key, `need` how many cells with exactly
  // that key belong to the top K
  uint32_t prefix = 0u, mask = 0u;
  int need = k_out;
#pragma unroll
  for (int pass = 0; pass < 3; ++pass) {
    const int shift = pass == 0 ? 21 : pass == 1 ? 10 : 0;
    const uint32_t digits = pass == 2 ? 1023u : 2047u;
    for (int i = tid; i < count; i += kThreads) {
      const uint32_t key = key_at(i);
      if ((key & mask) == prefix) atomicAdd(&hist[pass][(key >> shift) & digits], 1);
    }
    cluster.sync();
    // every CTA adds up the cluster's bins for itself: thread t holds the bins [4 t, 4 t + 4)
    int v[4] = {0, 0, 0, 0};
#pragma unroll
    for (int r = 0; r < kCluster; ++r) {
      const int4 w = *reinterpret_cast<const int4*>(cluster.map_shared_rank(&hist[pass][4 * tid], r));
      v[0] += w.x, v[1] += w.y, v[2] += w.z, v[3] += w.w;
    }
    const int mine = v[0] + v[1] + v[2] + v[3];
    int above = mine;  // cells in this thread's bins and all higher ones: suffix sum over the CTA
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_down_sync(0xffffffffu, above, d);
      if (lane + d < 32) above += t;
    }
    if (lane == 0) warp_sum[warp] = above;
    __syncthreads();
    for (int w = warp + 1; w < kThreads / 32; ++w) above += warp_sum[w];
    above -= mine;  // strictly higher bins
#pragma unroll
    for (int q = 3; q >= 0; --q) {
      if (above < need && above + v[q] >= need) sel_digit = 4 * tid + q, sel_need = need - above;  // one thread, one q
      above += v[q];
    }
    __syncthreads();
    prefix |= (uint32_t)sel_digit << shift;
    mask |= digits << shift;
    need = sel_need;
    __syncthreads();
  }
  const uint32_t threshold = prefix;
  const int greater = k_out - need;
  // ---- collect into CTA 0: everything above the threshold (any order), then the `need` lowest positions at it
  unsigned long long* all = cluster.map_shared_rank(cand, 0);
  int* taken = cluster.map_shared_rank(&n_greater, 0);
  int tie_base = 0;  // ties of the lower ranks: their last histogram knows them
  for (int r = 0; r < rank; ++r) tie_base += *cluster.map_shared_rank(&hist[2][threshold & 1023u], r);
  // a warp owns a run of cells; its ties are counted first so that they can be numbered by position
  const int run = (count + kThreads / 32 - 1) / (kThreads / 32);
  const int w0 = min(warp * run, count), w1 = min(w0 + run, count);
  int ties = 0;
  for (int i0 = w0; i0 < w1; i0 += 32) {
    const bool in = i0 + lane < w1;
    ties += __popc(__ballot_sync(0xffffffffu, in && key_at(in ? i0 + lane : 0) == threshold));
  }
  if (lane == 0) warp_sum[warp] = ties;
  __syncthreads();
  for (int w = 0; w < warp; ++w) tie_base += warp_sum[w];
  for (int i0 = w0; i0 < w1; i0 += 32) {
    const bool in = i0 + lane < w1;
    const uint32_t key = in ? key_at(i0 + lane) : 0u;
    const unsigned long long entry = ((unsigned long long)key << 32) | (0xFFFFFFFFu - (uint32_t)(first + i0 + lane));
    const unsigned up = __ballot_sync(0xffffffffu, in && key > threshold);
    const unsigned tie = __ballot_sync(0xffffffffu, in && key == threshold);
    int base = 0;
    if (up) {
      if (lane == 0) base = atomicAdd(taken, __popc(up));
      base = __shfl_sync(0xffffffffu, base, 0);
      if ((up >> lane) & 1u) all[base + __popc(up & lanemask_lt())] = entry;
    }
    if ((tie >> lane) & 1u) {
      const int t = tie_base + __popc(tie & lanemask_lt());
      if (t < need) all[greater + t] = entry;
    }
    tie_base += __popc(tie);
  }
  cluster.sync();
  if (rank != 0)
    for (int i = tid; i < k_out; i += kThreads) cand[i] = all[i];
  cluster.sync();  // CTA 0 may leave once the others have their copies
  // ---- rank and decode: the entries are distinct, so an entry's rank is the number of larger ones; eight lanes count
  // for one entry
  const int share = (k_out + kCluster - 1) / kCluster;
  const int e0 = min(rank * share, k_out), e1 = min(e0 + share, k_out);
  for (int e = e0 + (tid >> 3); e < ((e1 - e0 + 3) & ~3) + e0; e += kThreads / 8) {  // whole warps
    const unsigned long long me = cand[e < e1 ? e : e0];
    int larger = 0;
    for (int i = tid & 7; i < k_out; i += 8) larger += cand[i] > me;
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) larger += __shfl_xor_sync(0xffffffffu, larger, d);
    if ((tid & 7) == 0 && e < e1) {
      const int pos = (int)(0xFFFFFFFFu - (uint32_t)me);
      const int64_t o = (int64_t)b * k_out + larger;
      decode_cell<T>(a, preds_b, pos, load_f32(scores + pos), a.out_ids[c] + o, a.out_scores[c] + o,
                     a.out_boxes[c] + o * (a.box_in_params - 2), a.class_ids[c]);
    }
  }
}

template <class T> int launch_topk(const DecodeArgs& a, int b, cudaStream_t st) {
  const int n = a.size_y * a.size_x, per = (n + kCluster - 1) / kCluster;
  const bool hold = per <= kMaxHeldKeys;
  const size_t smem = (size_t)a.topk * sizeof(unsigned long long) + (hold ? (size_t)per * sizeof(uint32_t) : 0);
  auto kern = hold ? topk_decode_kernel<T, true> : topk_decode_kernel<T, false>;
  if (smem > 20 * 1024) {  // beside the histograms' 24 KB
    static std::atomic<bool> raised[64][2];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return D3D_ERR_CUDA;
    if (!raised[dev][hold].load(std::memory_order_acquire)) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxTopK * 8 + kMaxHeldKeys * 4) !=
          cudaSuccess)
        return D3D_ERR_CUDA;
      raised[dev][hold].store(true, std::memory_order_release);
    }
  }
  kern<<<dim3(a.num_class * kCluster, b), kThreads, smem, st>>>(a, per);
  D3D_CHECK_LAUNCH();
  return D3D_OK;
}

int num_classes(const d3d_yolox3d_decode_params* p) {
  for (int i = 0; i < 8; ++i)
    if (p->class_ids[i] < 0) return i;
  return 8;
}

}  // namespace
}  // namespace d3d

using namespace d3d;

extern "C" int d3d_yolox3d_decode_parse(const void* data_s, size_t len, d3d_yolox3d_decode_params* p) {
  D3D_REQUIRE(p && (data_s || len == 0), D3D_ERR_INVALID_ARGUMENT);
  D3D_REQUIRE(len >= sizeof(int32_t) * 10, D3D_ERR_BAD_BLOB);
  const unsigned char* s = reinterpret_cast<const unsigned char*>(data_s);
  memcpy(&p->stride, s, 4);
  memcpy(&p->topk, s + 4, 4);
  memcpy(p->class_ids, s + 8, 32);
  D3D_REQUIRE(p->stride >= 1 && p->topk >= 1, D3D_ERR_BAD_BLOB);
  return D3D_OK;
}

extern "C" int d3d_yolox3d_decode_num_outputs(const d3d_yolox3d_decode_params* p) {
  return p ? 3 * num_classes(p) : D3D_ERR_INVALID_ARGUMENT;
}

static int decode_dims(const d3d_yolox3d_decode_params* p, const d3d_tensor_desc* in, int n_in, int* b, int* c, int* y,
                       int* x, int* box_in, int* k) {
  D3D_REQUIRE(p && in && n_in >= 3 && in[0].nb_dims == 4 && in[1].nb_dims == 4 && in[2].nb_dims == 1,
              D3D_ERR_INVALID_ARGUMENT);
  D3D_REQUIRE((in[0].dtype == D3D_FLOAT || in[0].dtype == D3D_HALF) && in[1].dtype == in[0].dtype &&
                  in[2].dtype == D3D_FLOAT,
              D3D_ERR_UNSUPPORTED_DTYPE);
  *b = (int)in[0].dims[0], *c = (int)in[0].dims[1], *y = (int)in[0].dims[2], *x = (int)in[0].dims[3];
  *box_in = (int)in[1].dims[1];
  D3D_REQUIRE(in[1].dims[0] == *b && in[1].dims[2] == *y && in[1].dims[3] == *x && *box_in >= 9 && in[2].dims[0] >= 4,
              D3D_ERR_INVALID_ARGUMENT);
  D3D_REQUIRE(*c >= 0 && *c <= num_classes(p), D3D_ERR_INVALID_ARGUMENT);
  const int64_t n = (int64_t)*y * *x;
  D3D_REQUIRE(n < (1ll << 31) && *b <= 65535, D3D_ERR_TOO_LARGE);
  *k = (int)(n < p->topk ? n : p->topk);
  return D3D_OK;
}

extern "C" int d3d_yolox3d_decode_output_desc(const d3d_yolox3d_decode_params* p, const d3d_tensor_desc* in, int n_in,
                                              int index, d3d_tensor_desc* out) {
  D3D_REQUIRE(out && index >= 0, D3D_ERR_INVALID_ARGUMENT);
  int b, c, y, x, box_in, k;
  int rc = decode_dims(p, in, n_in, &b, &c, &y, &x, &box_in, &k);
  if (rc != D3D_OK) return rc;
  D3D_REQUIRE(index < 3 * num_classes(p), D3D_ERR_INVALID_ARGUMENT);
  memset(out, 0, sizeof(*out));
  out->dtype = index % 3 == 0 ? D3D_INT32 : D3D_FLOAT;
  out->nb_dims = index % 3 == 2 ? 3 : 2;
  out->dims[0] = b, out->dims[1] = k;
  if (index % 3 == 2) out->dims[2] = box_in - 2;
  return D3D_OK;
}

extern "C" int d3d_yolox3d_decode_workspace(const d3d_yolox3d_decode_params* p, const d3d_tensor_desc* in, int n_in,
                                            size_t* bytes) {
  D3D_REQUIRE(p && bytes, D3D_ERR_INVALID_ARGUMENT);
  (void)in, (void)n_in;
  *bytes = 0;  // the reference needs the radix-sort scratch (yolox3d_decode.cu:255-298); the top-K select needs none
  return D3D_OK;
}

extern "C" int d3d_yolox3d_decode_enqueue(const d3d_yolox3d_decode_params* p, const d3d_tensor_desc* in, int n_in,
                                          const d3d_tensor_desc* out, int n_out, const void* const* inputs,
                                          void* const* outputs, void* workspace, size_t workspace_bytes,
                                          void* stream) {
  D3D_NVTX_RANGE("d3d_yolox3d_decode_enqueue");
  (void)workspace, (void)workspace_bytes;
  D3D_REQUIRE(out && inputs && outputs, D3D_ERR_INVALID_ARGUMENT);
  int b, c, y, x, box_in, k;
  int rc = decode_dims(p, in, n_in, &b, &c, &y, &x, &box_in, &k);
  if (rc != D3D_OK) return rc;
  D3D_REQUIRE(n_out >= 3 * c, D3D_ERR_INVALID_ARGUMENT);
  if (b == 0 || c == 0 || k == 0) return D3D_OK;
  D3D_REQUIRE(k <= kMaxTopK, D3D_ERR_TOO_LARGE);
  DecodeArgs a;
  a.cls_scores = inputs[0], a.bbox_preds = inputs[1], a.pillar_config = reinterpret_cast<const float*>(inputs[2]);
  a.num_class = c, a.size_y = y, a.size_x = x, a.box_in_params = box_in, a.topk = k, a.stride = p->stride;
  for (int i = 0; i < 8; ++i) {
    a.class_ids[i] = p->class_ids[i];
    a.out_ids[i] = i < c ? reinterpret_cast<int32_t*>(outputs[3 * i]) : nullptr;
    a.out_scores[i] = i < c ? reinterpret_cast<float*>(outputs[3 * i + 1]) : nullptr;
    a.out_boxes[i] = i < c ? reinterpret_cast<float*>(outputs[3 * i + 2]) : nullptr;
    D3D_REQUIRE(i >= c || (a.out_ids[i] && a.out_scores[i] && a.out_boxes[i]), D3D_ERR_INVALID_ARGUMENT);
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return in[0].dtype == D3D_FLOAT ? launch_topk<float>(a, b, st) : launch_topk<__half>(a, b, st);
}
