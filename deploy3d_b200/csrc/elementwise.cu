// The layers an engine runs between and behind the plugins of a network, each as one pass over its tensors: they move
// bytes and nothing else, so what counts is that every tensor is read and written once.
//   activation      residual sum and ReLU of a plugin-order graph
//   recon           (sigmoid(a) + sigmoid(b) + sigmoid(c)) * x, with x copied behind it: ReconBlock and concatenation of the
//                   Cylinder3D-shaped network (tests/cylinder/test_cylinder3d.py:181-205, :262-263).  As tensor operations
//                   in fp32 these are 26 kernels, 290 us of the 120 k-point frame; one pass over 5 x 13 MB takes 15
//   gather labels   voxel -> point gather of the logits together with their arg-max (:322)
#include "common.cuh"

// The element-wise layer that follows an SPConvMM node in a graph (residual sum and ReLU, in that order or the other):
// one pass over the tensor where a sum and an activation layer are two.  The sum is rounded once: ReLU commutes with
// rounding, so the bytes are those of the two layers.
namespace d3d {
namespace {
template <class T>
__global__ void __launch_bounds__(256) activation_kernel(T* __restrict__ x, const T* __restrict__ residual, int64_t n, int relu) {
  constexpr int kVec = 16 / sizeof(T);
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (int64_t)gridDim.x * blockDim.x;
  auto one = [&](T v, T r) -> T {
    float f = to_f32(v);
    if (relu == 2) f = f < 0.f ? 0.f : f;  // NaN stays NaN, as in an activation layer
    if (residual) f += to_f32(r);
    if (relu == 1) f = f < 0.f ? 0.f : f;
    return from_f32<T>(f);
  };
  const int64_t nv = n / kVec;
  for (int64_t i = tid; i < nv; i += nth) {
    uint4 a = reinterpret_cast<uint4*>(x)[i], b = make_uint4(0u, 0u, 0u, 0u);
    if (residual) b = __ldg(reinterpret_cast<const uint4*>(residual) + i);
    T* pa = reinterpret_cast<T*>(&a);
    const T* pb = reinterpret_cast<const T*>(&b);
#pragma unroll
    for (int e = 0; e < kVec; ++e) pa[e] = one(pa[e], pb[e]);
    reinterpret_cast<uint4*>(x)[i] = a;
  }
  for (int64_t i = nv * kVec + tid; i < n; i += nth) x[i] = one(x[i], residual ? residual[i] : x[i]);
}
}  // namespace
}  // namespace d3d

using namespace d3d;

extern "C" int d3d_activation(int dtype, void* x, const void* residual, int64_t elements, int relu, void* stream) {
  D3D_NVTX_RANGE("d3d_activation");
  D3D_REQUIRE(elements >= 0 && relu >= 0 && relu <= 2, D3D_ERR_INVALID_ARGUMENT);
  if (elements == 0 || (relu == 0 && !residual)) return D3D_OK;
  D3D_REQUIRE(x && reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(residual) % 16 == 0,
              D3D_ERR_INVALID_ARGUMENT);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int grid = stream_grid(elements * (int64_t)dtype_size(dtype) / 16, 256);
  switch (dtype) {
    case D3D_FLOAT:
      activation_kernel<float><<<grid, 256, 0, st>>>((float*)x, (const float*)residual, elements, relu);
      break;
    case D3D_HALF:
      activation_kernel<__half><<<grid, 256, 0, st>>>((__half*)x, (const __half*)residual, elements, relu);
      break;
    case D3D_BF16:
      activation_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((__nv_bfloat16*)x, (const __nv_bfloat16*)residual, elements, relu);
      break;
    default: return D3D_ERR_UNSUPPORTED_DTYPE;
  }
  D3D_CHECK_LAUNCH();
  return D3D_OK;
}

namespace d3d {
namespace {

// One thread per 16 bytes of a row; out rows have `out_ld` elements: [result | x if copy_x].
template <class T>
__global__ void __launch_bounds__(256)
recon_kernel(const T* __restrict__ a, const T* __restrict__ b, const T* __restrict__ c, const T* __restrict__ x, int64_t rows,
             int channels, T* __restrict__ out, int64_t out_ld, int copy_x) {
  constexpr int kVec = 16 / sizeof(T);
  const int per_row = channels / kVec;
  const int64_t n = rows * per_row, nth = (int64_t)gridDim.x * blockDim.x;
  auto sigmoid = [](float t) { return 1.0f / (1.0f + expf(-t)); };
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nth) {
    const int64_t row = i / per_row;
    const int piece = (int)(i - row * per_row);
    const uint4 va = __ldg(reinterpret_cast<const uint4*>(a) + i), vb = __ldg(reinterpret_cast<const uint4*>(b) + i);
    const uint4 vc = __ldg(reinterpret_cast<const uint4*>(c) + i), vx = __ldg(reinterpret_cast<const uint4*>(x) + i);
    uint4 r;
#pragma unroll
    for (int e = 0; e < kVec; ++e) {
      const float g = sigmoid(to_f32(reinterpret_cast<const T*>(&va)[e])) + sigmoid(to_f32(reinterpret_cast<const T*>(&vb)[e])) +
                      sigmoid(to_f32(reinterpret_cast<const T*>(&vc)[e]));
      reinterpret_cast<T*>(&r)[e] = from_f32<T>(g * to_f32(reinterpret_cast<const T*>(&vx)[e]));
    }
    uint4* o = reinterpret_cast<uint4*>(out + row * out_ld) + piece;
    o[0] = r;
    if (copy_x) o[per_row] = vx;
  }
}

// 64 points per CTA: their rows come in as 16-byte pieces, the arg-max is taken in shared memory, the logits leave as one
// contiguous run.
constexpr int kLabelPoints = 64;
template <class T>
__global__ void __launch_bounds__(256)
gather_labels_kernel(const T* __restrict__ feats, int64_t ld, bool wide, int classes, int64_t m, const int32_t* __restrict__ ids,
                     int64_t n, float fill, float* __restrict__ logits, int32_t* __restrict__ labels) {
  extern __shared__ float rows[];  // [kLabelPoints][pitch]
  constexpr int kVec = 16 / sizeof(T);
  const int pieces = (classes + kVec - 1) / kVec, pitch = classes | 1;
  const int64_t p0 = (int64_t)blockIdx.x * kLabelPoints;
  const int here = (int)(n - p0 < kLabelPoints ? n - p0 : kLabelPoints);
  for (int e = threadIdx.x; e < here * pieces; e += 256) {
    const int p = e / pieces, piece = e - p * pieces;
    const int v = __ldg(ids + p0 + p);
    const bool ok = v >= 0 && D3D_BOUNDS_OK(v, 0, m, kSiteGatherBack) && v < m;
    const T* src = feats + (int64_t)v * ld + piece * kVec;
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
    if (ok && wide) w = __ldg(reinterpret_cast<const uint4*>(src));
#pragma unroll
    for (int q = 0; q < kVec; ++q)
      if (piece * kVec + q < classes)
        rows[p * pitch + piece * kVec + q] = !ok ? fill : wide ? to_f32(reinterpret_cast<const T*>(&w)[q]) : to_f32(src[q]);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < here * classes; e += 256) logits[p0 * classes + e] = rows[e / classes * pitch + e % classes];
  if ((int)threadIdx.x < here) {
    float best = rows[threadIdx.x * pitch];
    int at = 0;
    for (int c = 1; c < classes; ++c) {  // the first of equal values; a NaN counts as the largest
      const float v = rows[threadIdx.x * pitch + c];
      if (v > best || (isnan(v) && !isnan(best))) best = v, at = c;
    }
    labels[p0 + threadIdx.x] = at;
  }
}

}  // namespace
}  // namespace d3d

using namespace d3d;

extern "C" int d3d_recon(int dtype, const void* a, const void* b, const void* c, const void* x, int64_t rows, int channels,
                         void* out, int64_t out_ld, int copy_x, void* stream) {
  D3D_NVTX_RANGE("d3d_recon");
  const int esize = (int)dtype_size(dtype);
  D3D_REQUIRE(dtype == D3D_FLOAT || dtype == D3D_HALF || dtype == D3D_BF16, D3D_ERR_UNSUPPORTED_DTYPE);
  D3D_REQUIRE(rows >= 0 && channels >= 1 && channels * esize % 16 == 0 && out_ld * esize % 16 == 0 &&
                  out_ld >= (int64_t)channels * (copy_x ? 2 : 1),
              D3D_ERR_INVALID_ARGUMENT);
  if (rows == 0) return D3D_OK;
  const uintptr_t all = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
                        reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out);
  D3D_REQUIRE(a && b && c && x && out && all % 16 == 0, D3D_ERR_INVALID_ARGUMENT);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int grid = stream_grid(rows * (channels * esize / 16), 256);
#define D3D_RECON(T) \
  recon_kernel<T><<<grid, 256, 0, st>>>((const T*)a, (const T*)b, (const T*)c, (const T*)x, rows, channels, (T*)out, out_ld, copy_x)
  if (dtype == D3D_FLOAT) D3D_RECON(float);
  else if (dtype == D3D_HALF) D3D_RECON(__half);
  else D3D_RECON(__nv_bfloat16);
#undef D3D_RECON
  D3D_CHECK_LAUNCH();
  return D3D_OK;
}

extern "C" int d3d_gather_labels(int dtype, const void* feats, int64_t ld, int classes, int64_t m, const int32_t* ids,
                                 int64_t n, float fill, float* logits, int32_t* labels, void* stream) {
  D3D_NVTX_RANGE("d3d_gather_labels");
  D3D_REQUIRE(dtype == D3D_FLOAT || dtype == D3D_HALF || dtype == D3D_BF16, D3D_ERR_UNSUPPORTED_DTYPE);
  const int vec = 16 / (int)dtype_size(dtype);
  D3D_REQUIRE(classes >= 1 && classes <= 128 && m >= 0 && n >= 0 && ld >= classes, D3D_ERR_INVALID_ARGUMENT);
  if (n == 0) return D3D_OK;
  D3D_REQUIRE(ids && logits && labels && (feats || m == 0), D3D_ERR_INVALID_ARGUMENT);
  // 16-byte pieces where the rows allow them (a padded row may be read up to its end)
  const bool wide = ld % vec == 0 && reinterpret_cast<uintptr_t>(feats) % 16 == 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)ceil_div(n, kLabelPoints);
  const size_t smem = (size_t)kLabelPoints * (classes | 1) * sizeof(float);  // at most 33 KB
#define D3D_LABELS(T) gather_labels_kernel<T><<<grid, 256, smem, st>>>((const T*)feats, ld, wide, classes, m, ids, n, fill, logits, labels)
  if (dtype == D3D_FLOAT) D3D_LABELS(float);
  else if (dtype == D3D_HALF) D3D_LABELS(__half);
  else D3D_LABELS(__nv_bfloat16);
#undef D3D_LABELS
  D3D_CHECK_LAUNCH();
  return D3D_OK;
}
