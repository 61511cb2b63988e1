// NMS3d: rotated-BEV non-maximum suppression.
//
// Replaces decoder::NMS3dPlugin (trt/decoder/nms3d.cu:58-127, :200-236) with the IoU arithmetic of
// trt/decoder/iou_rotated.cuh:36-234 restated operation by operation (this file is compiled with -fmad=false so
// that no multiply-add is fused and the keep-set is bit-identical to a strict IEEE-754 evaluation).
//
// Two kernels:
//   overlap mask : 64 rows x 64 (or, for few boxes, 16) columns of box pairs per CTA, upper triangle only.  A
//                  bounding-circle test and an upper bound of the overlap reject most pairs before the exact polygon
//                  clipping; the pairs that are left are dealt out evenly over the 256 threads.
//   suppression  : one CTA per batch row.  The greedy order is resolved 64 boxes at a time: a box is kept as soon as
//                  no undecided box before it suppresses it, so a block takes as many rounds as its longest chain
//                  of suppressions (2-5 on detector output), not 64 steps; the mask words of the kept boxes are then
//                  OR-ed into the later words by all warps while the rows of the next blocks are in flight.
//                  The reference runs this step on a single thread per row (nms3d.cu:106-127, launched <<<B, 1>>>).
#include <math.h>

#include <atomic>

#include "common.cuh"

namespace d3d {
namespace {

struct Pt {
  float x, y;
};
__device__ __forceinline__ Pt sub(Pt a, Pt b) { return Pt{a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ float cross2(Pt a, Pt b) { return a.x * b.y - b.x * a.y; }
__device__ __forceinline__ float dot2(Pt a, Pt b) { return a.x * b.x + a.y * b.y; }

struct Box {
  Pt p[4];     // corners (iou_rotated.cuh:30-49)
  float area;  // dx * dy
  float cx, cy, rad;
  float c2, s2, w, h;  // half cosine / sine of the heading, extents
  float pad;           // 17 words: a warp reading one field of 32 boxes hits 32 banks
};

__device__ __forceinline__ Box make_box(const float* b) {
  Box r;
  float cx = b[0], cy = b[1], w = b[3], h = b[4];
  double theta = b[6];
  float c2 = (float)cos(theta) * 0.5f;
  float s2 = (float)sin(theta) * 0.5f;
  r.p[0].x = cx - s2 * h - c2 * w;
  r.p[0].y = cy + c2 * h - s2 * w;
  r.p[1].x = cx + s2 * h - c2 * w;
  r.p[1].y = cy - c2 * h - s2 * w;
  r.p[2].x = 2 * cx - r.p[0].x;
  r.p[2].y = 2 * cy - r.p[0].y;
  r.p[3].x = 2 * cx - r.p[1].x;
  r.p[3].y = 2 * cy - r.p[1].y;
  r.area = w * h;
  r.cx = cx, r.cy = cy;
  r.c2 = c2, r.s2 = s2, r.w = w, r.h = h;
  r.rad = 0.5f * sqrtf(w * w + h * h);
  return r;
}

// The reference compares floats with double constants.  For a float x and a double constant c, x < c is x <= F or x < F
// with F the constant rounded to float, whichever side it was rounded to: the same truth value without a conversion.
#define D3D_F32_LT(x, c) ((double)(float)(c) < (c) ? (x) <= (float)(c) : (x) < (float)(c))
#define D3D_F32_LE(x, c) ((double)(float)(c) > (c) ? (x) < (float)(c) : (x) <= (float)(c))
#define D3D_F32_GT(x, c) ((double)(float)(c) > (c) ? (x) >= (float)(c) : (x) > (float)(c))

// Whether num / den, rounded to float, certainly lies outside [0, 1]: the signs differ (and the quotient cannot
// underflow to zero), or |num| > |den| (neighbouring floats already have a quotient that rounds above 1).  Of the 16
// edge pairs of two boxes at most a few cross; the others need no division.
__device__ __forceinline__ bool quotient_outside(float num, float den) {
  if (fabsf(num) > fabsf(den)) return true;
  return ((num < 0.f) != (den < 0.f)) && fabsf(num) > 1e-25f && fabsf(den) < 1e12f;
}

// Area of the convex hull of `num` points (iou_rotated.cuh:124-234) for 3 <= num <= 8, which is what two rectangles
// give unless corners or edges coincide: the same steps on the same values as the general loop in clipped_area, with
// every point in registers: the exchange sort has static indices then (with its 28 steps in local memory the mask
// kernel took 11.3 instead of 9.1 us at 3 x 257 boxes, 33 instead of 29 at 10 x 1000).
__device__ __forceinline__ float hull_area_small(const Pt* pts, int num) {
  Pt q[8];
  float dist[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) q[i] = pts[i];
  int t = 0;
  Pt start = q[0];
#pragma unroll
  for (int i = 1; i < 8; ++i)
    if (i < num && (q[i].y < start.y || (q[i].y == start.y && q[i].x < start.x))) t = i, start = q[i];
#pragma unroll
  for (int i = 0; i < 8; ++i) q[i] = sub(q[i], start);
  const Pt head = q[0];
#pragma unroll
  for (int i = 1; i < 8; ++i)
    if (i == t) q[0] = q[i], q[i] = head;
#pragma unroll
  for (int i = 0; i < 8; ++i) dist[i] = dot2(q[i], q[i]);
#pragma unroll
  for (int i = 1; i < 7; ++i) {
#pragma unroll
    for (int j = i + 1; j < 8; ++j) {
      const float cr = cross2(q[i], q[j]);
      if (j < num && (D3D_F32_LT(cr, -1e-6) || (D3D_F32_LT(fabsf(cr), 1e-6) && dist[i] > dist[j]))) {
        const Pt qt = q[i];
        q[i] = q[j], q[j] = qt;
        const float dt = dist[i];
        dist[i] = dist[j], dist[j] = dt;
      }
    }
  }
  Pt stack[8];  // the hull so far; its two topmost points also in registers
  stack[0] = q[0];
  Pt below = q[0], top = q[0];
  int m = 1;  // points on the stack
#pragma unroll
  for (int i = 1; i < 8; ++i) {
    if (i >= num) break;
    if (m == 1) {  // the first point apart from the start
      if (!D3D_F32_GT(dist[i], 1e-8)) continue;
    } else {
      while (m > 1 && cross2(sub(q[i], below), sub(top, below)) >= 0) {
        --m;
        top = below;
        if (m > 1) below = stack[m - 2];
      }
    }
    below = top, top = q[i];
    stack[m++] = q[i];
  }
  if (m <= 2) return 0.0f;
  float area = 0;
  for (int i = 1; i < m - 1; ++i) area += fabsf(cross2(sub(stack[i], q[0]), sub(stack[i + 1], q[0])));
  return area * 0.5f;
}

// Area of the intersection polygon (iou_rotated.cuh:51-234).
__device__ float clipped_area(const Box& A, const Box& B) {
  Pt ea[4], eb[4], pts[24], q[24];
  float dist[24];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    ea[i] = sub(A.p[(i + 1) & 3], A.p[i]);
    eb[i] = sub(B.p[(i + 1) & 3], B.p[i]);
  }
  int num = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float det = cross2(eb[j], ea[i]);
      if (D3D_F32_LE(fabsf(det), 1e-14)) continue;
      Pt d = sub(B.p[j], A.p[i]);
      const float n1 = cross2(eb[j], d), n2 = cross2(ea[i], d);
      if (quotient_outside(n1, det) || quotient_outside(n2, det)) continue;
      float t1 = n1 / det;
      float t2 = n2 / det;
      if (t1 >= 0.0f && t1 <= 1.0f && t2 >= 0.0f && t2 <= 1.0f) {
        pts[num].x = A.p[i].x + ea[i].x * t1;
        pts[num].y = A.p[i].y + ea[i].y * t1;
        ++num;
      }
    }
  }
  {
    Pt ab = eb[0], da = eb[3];
    float abab = dot2(ab, ab), adad = dot2(da, da);
    for (int i = 0; i < 4; ++i) {
      Pt ap = sub(A.p[i], B.p[0]);
      float apab = dot2(ap, ab), apad = -dot2(ap, da);
      if (apab >= 0 && apad >= 0 && apab <= abab && apad <= adad) pts[num++] = A.p[i];
    }
  }
  {
    Pt ab = ea[0], da = ea[3];
    float abab = dot2(ab, ab), adad = dot2(da, da);
    for (int i = 0; i < 4; ++i) {
      Pt ap = sub(B.p[i], A.p[0]);
      float apab = dot2(ap, ab), apad = -dot2(ap, da);
      if (apab >= 0 && apad >= 0 && apab <= abab && apad <= adad) pts[num++] = B.p[i];
    }
  }
  if (num <= 2) return 0.0f;
  if (num <= 8) return hull_area_small(pts, num);
  // Graham scan around the lowest point (iou_rotated.cuh:124-199)
  int t = 0;
  for (int i = 1; i < num; ++i)
    if (pts[i].y < pts[t].y || (pts[i].y == pts[t].y && pts[i].x < pts[t].x)) t = i;
  Pt start = pts[t];
  for (int i = 0; i < num; ++i) q[i] = sub(pts[i], start);
  Pt tmp = q[0];
  q[0] = q[t];
  q[t] = tmp;
  for (int i = 0; i < num; ++i) dist[i] = dot2(q[i], q[i]);
  for (int i = 1; i < num - 1; ++i) {
    for (int j = i + 1; j < num; ++j) {
      float cr = cross2(q[i], q[j]);
      if (D3D_F32_LT(cr, -1e-6) || (D3D_F32_LT(fabsf(cr), 1e-6) && dist[i] > dist[j])) {
        Pt qt = q[i];
        q[i] = q[j];
        q[j] = qt;
        float dt = dist[i];
        dist[i] = dist[j];
        dist[j] = dt;
      }
    }
  }
  int k;
  for (k = 1; k < num; ++k)
    if (D3D_F32_GT(dist[k], 1e-8)) break;
  if (k == num) return 0.0f;  // a single point
  q[1] = q[k];
  int m = 2;
  for (int i = k + 1; i < num; ++i) {
    while (m > 1 && cross2(sub(q[i], q[m - 2]), sub(q[m - 1], q[m - 2])) >= 0) --m;
    q[m++] = q[i];
  }
  if (m <= 2) return 0.0f;
  float area = 0;
  for (int i = 1; i < m - 1; ++i) area += fabsf(cross2(sub(q[i], q[0]), sub(q[i + 1], q[0])));
  return area * 0.5f;
}

// nms3d.cu:42-56: BEV IoU, z ignored.  Two boxes whose bounding circles are disjoint cannot overlap (their clipped
// area is exactly 0, and 0 >= thr fails for thr > 0): such pairs never reach the polygon clipping.
__device__ __forceinline__ bool circles_touch(const Box& a, const Box& b) {
  float dx = a.cx - b.cx, dy = a.cy - b.cy, r = a.rad + b.rad;
  return !(dx * dx + dy * dy > r * r * 1.0001f + 1e-6f);
}
// Whether the pair can be dropped without clipping: the intersection lies inside the rectangle that box `b`'s extent
// along box `a`'s axes leaves of box `a`; when even that area -- with a margin far above the rounding of either
// computation -- stays below the threshold, the exact IoU does too.  Boxes that are tiny, far out or not finite are
// never dropped here.  (Detector output: of the pairs whose circles touch, one in two to three is left.)
__device__ __forceinline__ float overlap_bound(const Box& a, const Box& b) {
  const float ca = 2.f * a.c2, sa = 2.f * a.s2, dx = b.cx - a.cx, dy = b.cy - a.cy;
  const float u = dx * ca + dy * sa, v = dy * ca - dx * sa;  // centre of b in the frame of a
  const float cr = 2.f * fabsf(ca * b.c2 + sa * b.s2), sr = 2.f * fabsf(sa * b.c2 - ca * b.s2);
  const float eu = 0.5f * (cr * b.w + sr * b.h), ev = 0.5f * (sr * b.w + cr * b.h);
  const float hw = 0.5f * a.w, hh = 0.5f * a.h;
  const float ou = fminf(hw, u + eu) - fmaxf(-hw, u - eu), ov = fminf(hh, v + ev) - fmaxf(-hh, v - ev);
  return (fmaxf(ou, 0.f) + 1e-3f) * (fmaxf(ov, 0.f) + 1e-3f);
}
__device__ __forceinline__ bool surely_below(const Box& a, const Box& b, float thr) {
  // the margins are absolute lengths: for boxes of millimetres they say nothing (and the clipping's own tolerances
  // decide), and positions far from the origin round coarser than they allow for
  if (!(a.w > 0.02f && a.h > 0.02f && b.w > 0.02f && b.h > 0.02f)) return false;
  if (!(fabsf(a.cx) + fabsf(a.cy) + a.w + a.h < 1000.f && fabsf(b.cx) + fabsf(b.cy) + b.w + b.h < 1000.f)) return false;
  const float m = fminf(overlap_bound(a, b), overlap_bound(b, a)) * 1.001f;
  return m < thr * 0.99f * (a.area + b.area - m);
}
__device__ __forceinline__ bool iou_reaches(const Box& a, const Box& b, float thr) {
  float ov = clipped_area(a, b);
  return ov / fmaxf(a.area + b.area - ov, 1e-8f) >= thr;
}

constexpr int kNmsBlock = 64;

// grid (col block * kSplit + column part, row block, batch); upper triangle only.  mask[b][row][col block] bit j = row
// suppresses col*64+j; with kSplit = 4 a CTA writes the 16-bit quarter of its columns.
// Two passes over the pairs of a CTA: the cheap rejections for every pair (uniform work), then the polygon clipping
// for the pairs that passed, dealt out evenly over the 256 threads -- taken pair by pair inside the first loop, the
// few survivors would each hold up their whole warp.  The clipping of one pair is a serial chain of 4-5 us, so
// a call with few boxes is spread over four times the CTAs (kSplit = 4): no thread then clips two pairs in turn.
template <int kSplit>
__global__ void __launch_bounds__(256)
overlap_mask_kernel(const float* __restrict__ boxes, int k, int box_dim, float thr, int nw,
                    unsigned long long* __restrict__ mask) {
  constexpr int kCols = kNmsBlock / kSplit, kPerThread = kCols / 4;  // columns of the CTA, of a thread
  pdl_release();
  const int cb = blockIdx.x / kSplit, part = blockIdx.x % kSplit, rb = blockIdx.y, b = blockIdx.z;
  if (rb > cb) return;
  __shared__ Box cols[kCols], rows[kNmsBlock];
  __shared__ unsigned int hit[kNmsBlock][kCols / 16];           // 16 columns per word
  __shared__ unsigned short cand[kNmsBlock * kCols];            // row << 8 | column of a pair to clip
  __shared__ int warp_base[9];
  const float* bx = boxes + (int64_t)b * k * box_dim;
  const int tid = threadIdx.x, r = tid & 63, quarter = tid >> 6;
  const int col0 = cb * kNmsBlock + part * kCols;
  if (tid < kCols) {
    if (col0 + tid < k) cols[tid] = make_box(bx + (int64_t)(col0 + tid) * box_dim);
  } else if (tid >= 64 && tid < 64 + kNmsBlock) {
    const int rr = rb * kNmsBlock + tid - 64;
    if (rr < k) rows[tid - 64] = make_box(bx + (int64_t)rr * box_dim);
  }
  if (tid < kNmsBlock)
    for (int w = 0; w < kCols / 16; ++w) hit[tid][w] = 0u;
  __syncthreads();
  const int row = rb * kNmsBlock + r;
  const int ncol = min(k - col0, kCols);
  unsigned int near = 0;  // bit j - kPerThread * quarter: column j is to be clipped
  if (row < k) {
    int j0 = quarter * kPerThread;
    const int j1 = min(j0 + kPerThread, ncol);
    if (rb == cb) j0 = max(j0, r + 1 - part * kCols);
    for (int j = j0; j < j1; ++j)
      if (thr <= 0.f || (circles_touch(rows[r], cols[j]) && !surely_below(rows[r], cols[j], thr)))
        near |= 1u << (j - quarter * kPerThread);
  }
  // positions of this thread's pairs in the CTA's list: warp scan, then the eight warp totals
  const int lane = tid & 31, warp = tid >> 5;
  const int mine = __popc(near);
  int inc = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += t;
  }
  if (lane == 31) warp_base[warp + 1] = inc;
  __syncthreads();
  if (tid == 0) {
    warp_base[0] = 0;
    for (int w = 1; w <= 8; ++w) warp_base[w] += warp_base[w - 1];
  }
  __syncthreads();
  int pos = warp_base[warp] + inc - mine;
  for (unsigned int m = near; m; m &= m - 1)
    cand[pos++] = (unsigned short)((r << 8) | (quarter * kPerThread + __ffs(m) - 1));
  __syncthreads();
  const int total = warp_base[8];
  for (int i = tid; i < total; i += 256) {
    const int pr = cand[i] >> 8, pj = cand[i] & 255;
    if (iou_reaches(rows[pr], cols[pj], thr)) atomicOr(&hit[pr][pj >> 4], 1u << (pj & 15));
  }
  __syncthreads();
  if (tid < kNmsBlock && row < k) {
    unsigned long long* word = mask + ((int64_t)b * k + row) * nw + cb;
    if constexpr (kSplit == 1)
      *word = (unsigned long long)hit[r][0] | ((unsigned long long)hit[r][1] << 16) |
              ((unsigned long long)hit[r][2] << 32) | ((unsigned long long)hit[r][3] << 48);
    else
      reinterpret_cast<unsigned short*>(word)[part] = (unsigned short)hit[r][0];
  }
}

// One warp per batch row (nms3d.cu:106-127).  remv words are lane-distributed: lane l owns words l, l+32, ...
constexpr int kMaxWordsPerLane = 8;  // K <= 64 * 32 * 8 = 16384 boxes per row

__global__ void __launch_bounds__(32)
suppress_kernel(const unsigned long long* __restrict__ mask, const float* __restrict__ in_scores, int k, int nw,
                float* __restrict__ out_scores) {
  const int b = blockIdx.x, lane = threadIdx.x;
  const unsigned long long* mk = mask + (int64_t)b * k * nw;
  unsigned long long remv[kMaxWordsPerLane];
#pragma unroll
  for (int s = 0; s < kMaxWordsPerLane; ++s) remv[s] = 0ull;
  for (int blk = 0; blk < nw; ++blk) {
    const int base = blk * kNmsBlock;
    const int nbox = min(k - base, kNmsBlock);
    // diagonal words of the 64 boxes of this block: lane holds boxes lane and lane + 32
    unsigned long long d0 = lane < nbox ? mk[(int64_t)(base + lane) * nw + blk] : 0ull;
    unsigned long long d1 = lane + 32 < nbox ? mk[(int64_t)(base + lane + 32) * nw + blk] : 0ull;
    unsigned long long cur = 0ull;
#pragma unroll
    for (int s = 0; s < kMaxWordsPerLane; ++s)
      if ((blk >> 5) == s) cur = remv[s];
    cur = __shfl_sync(0xffffffffu, cur, blk & 31);
    for (int i = 0; i < nbox; ++i) {
      unsigned long long di = __shfl_sync(0xffffffffu, i < 32 ? d0 : d1, i & 31);
      if (!((cur >> i) & 1ull)) cur |= di;
    }
    unsigned long long valid = nbox == 64 ? ~0ull : ((1ull << nbox) - 1ull);
    unsigned long long kept = ~cur & valid;
    // scores of this block
    for (int i = lane; i < nbox; i += 32) {
      float s = in_scores[(int64_t)b * k + base + i];
      out_scores[(int64_t)b * k + base + i] = ((cur >> i) & 1ull) ? -1.0f : s;
    }
    // OR the rows of the kept boxes into the words behind this block
    while (kept) {
      int i = __ffsll((long long)kept) - 1;
      kept &= kept - 1;
      const unsigned long long* row = mk + (int64_t)(base + i) * nw;
#pragma unroll
      for (int s = 0; s < kMaxWordsPerLane; ++s) {
        int w = s * 32 + lane;
        if (w > blk && w < nw) remv[s] |= row[w];
      }
    }
  }
}

// The sweep for K <= 2048 boxes (nw <= 32 words per row).  The rows of a 64-box block are consecutive words of the
// mask; they come in with cp.async, up to kRing blocks ahead, so that the serial part touches shared memory only.
// What is left is the chain over the blocks: two barriers, a few rounds of warp reductions and eight shared-memory
// reads each (one CTA-wide pass over 16 blocks: 100 -> 21 us at 10 x 1000 boxes, 25 -> 4 us at 3 x 257; every box
// cost a step before).
constexpr int kSweepMaxWords = 32;
constexpr int kSweepThreads = 256;
constexpr int kRing = 6;

__device__ __forceinline__ unsigned long long warp_or(unsigned long long v) {
  const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)v);
  const unsigned hi = __reduce_or_sync(0xffffffffu, (unsigned)(v >> 32));
  return ((unsigned long long)hi << 32) | lo;
}

__global__ void __launch_bounds__(kSweepThreads)
suppress_blocks_kernel(const unsigned long long* __restrict__ mask, const float* __restrict__ in_scores, int k, int nw,
                       float* __restrict__ out_scores) {
  extern __shared__ unsigned long long ring[];  // [kRing][64 * nw]
  __shared__ unsigned long long removed[kSweepMaxWords];
  __shared__ unsigned long long kept_s[kSweepMaxWords];
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned long long* mk = mask + (int64_t)b * k * nw;
  const int slot_words = kNmsBlock * nw;
  auto load = [&](int blk) {  // one commit group per block, also beyond the last one: the waits below count groups
    if (blk < nw) {
      const int words = min(k - blk * kNmsBlock, kNmsBlock) * nw;
      const unsigned long long* src = mk + (int64_t)blk * kNmsBlock * nw;
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ring + (blk % kRing) * slot_words);
      for (int f = tid; f < words; f += kSweepThreads)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + f * 8), "l"(src + f) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (tid < kSweepMaxWords) removed[tid] = 0ull;
  pdl_wait();  // the mask of the preceding kernel
  for (int blk = 0; blk < kRing - 1; ++blk) load(blk);
  for (int blk = 0; blk < nw; ++blk) {
    load(blk + kRing - 1);  // its slot was last read before the barrier at the end of the previous turn
    asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 1) : "memory");
    __syncthreads();
    const unsigned long long* rows = ring + (blk % kRing) * slot_words;
    const int nbox = min(k - blk * kNmsBlock, kNmsBlock);
    if (warp == 0) {
      const unsigned long long d0 = lane < nbox ? rows[lane * nw + blk] : 0ull;
      const unsigned long long d1 = lane + 32 < nbox ? rows[(lane + 32) * nw + blk] : 0ull;
      const unsigned long long valid = nbox == 64 ? ~0ull : ((1ull << nbox) - 1ull);
      unsigned long long open = ~removed[blk] & valid, kept = 0ull;  // not decided yet / kept
      while (open) {
        // suppressed by some undecided box: wait; the others are kept, and what they suppress is removed.  (The first
        // undecided box is always among the kept ones.)
        const unsigned long long by_open =
            warp_or((((open >> lane) & 1ull) ? d0 : 0ull) | (((open >> (lane + 32)) & 1ull) ? d1 : 0ull));
        const unsigned long long fresh = open & ~by_open;
        const unsigned long long by_fresh =
            warp_or((((fresh >> lane) & 1ull) ? d0 : 0ull) | (((fresh >> (lane + 32)) & 1ull) ? d1 : 0ull));
        kept |= fresh;
        open &= ~(fresh | by_fresh);
      }
      if (lane == 0) kept_s[blk] = kept;
    }
    __syncthreads();
    // the kept boxes' rows into the words behind this block: warp w takes rows 8 w .. 8 w + 7, a lane one word
    const unsigned long long kept = kept_s[blk];
    const unsigned mine = (unsigned)(kept >> (8 * warp)) & 255u;
    if (mine && lane > blk && lane < nw) {
      unsigned long long acc = 0ull;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if ((mine >> i) & 1u) acc |= rows[(8 * warp + i) * nw + lane];
      if (acc) atomicOr(&removed[lane], acc);
    }
    __syncthreads();
  }
  for (int i = tid; i < k; i += kSweepThreads) {
    const float s = in_scores[(int64_t)b * k + i];
    out_scores[(int64_t)b * k + i] = ((kept_s[i >> 6] >> (i & 63)) & 1ull) ? s : -1.0f;
  }
}

}  // namespace
}  // namespace d3d

using namespace d3d;

extern "C" int d3d_nms3d_parse(const void* data_s, size_t len, d3d_nms3d_params* p) {
  (void)data_s, (void)len;  // the reference plugin carries no parameters (nms3d.cu:143-144)
  D3D_REQUIRE(p, D3D_ERR_INVALID_ARGUMENT);
  p->iou_threshold = 0.1f;  // nms3d.cu:138
  return D3D_OK;
}

static int nms_dims(const d3d_tensor_desc* in, int n_in, int* b, int* k, int* box_dim) {
  D3D_REQUIRE(in && n_in >= 2 && in[0].nb_dims == 2 && in[1].nb_dims == 3, D3D_ERR_INVALID_ARGUMENT);
  D3D_REQUIRE(in[0].dtype == D3D_FLOAT && in[1].dtype == D3D_FLOAT, D3D_ERR_UNSUPPORTED_DTYPE);
  *b = (int)in[1].dims[0], *k = (int)in[1].dims[1], *box_dim = (int)in[1].dims[2];
  D3D_REQUIRE(in[0].dims[0] == *b && in[0].dims[1] == *k && *box_dim >= 7, D3D_ERR_INVALID_ARGUMENT);
  D3D_REQUIRE(*k <= kNmsBlock * 32 * kMaxWordsPerLane && *b <= 65535, D3D_ERR_TOO_LARGE);
  return D3D_OK;
}

extern "C" int d3d_nms3d_workspace(const d3d_nms3d_params* p, const d3d_tensor_desc* in, int n_in, size_t* bytes) {
  D3D_REQUIRE(p && bytes, D3D_ERR_INVALID_ARGUMENT);
  int b, k, bd;
  int rc = nms_dims(in, n_in, &b, &k, &bd);
  if (rc != D3D_OK) return rc;
  *bytes = align_up((size_t)b * k * ceil_div(k, kNmsBlock) * sizeof(unsigned long long), 256);
  return D3D_OK;
}

// The two launches of an NMS3d call over a mask scratch of b * k * nw words.  Neither sweep reads a word the mask
// kernel did not write in the same call (the diagonal word and the words behind it; the block sweep copies whole
// rows into shared memory but uses the same words), so the scratch needs no initialisation.
static int launch_nms(const d3d_nms3d_params* p, int b, int k, int bd, int nw, const void* const* inputs,
                      void* const* outputs, unsigned long long* mask, void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const float* boxes = reinterpret_cast<const float*>(inputs[1]);
  // as long as the finer grid still fits the GPU in about two rounds of CTAs (four of them per SM)
  if ((int64_t)nw * (nw + 1) / 2 * b * 4 <= kNumSMs * 8)
    overlap_mask_kernel<4><<<dim3(nw * 4, nw, b), 256, 0, st>>>(boxes, k, bd, p->iou_threshold, nw, mask);
  else
    overlap_mask_kernel<1><<<dim3(nw, nw, b), 256, 0, st>>>(boxes, k, bd, p->iou_threshold, nw, mask);
  const float* scores = reinterpret_cast<const float*>(inputs[0]);
  float* out = reinterpret_cast<float*>(outputs[0]);
  if (nw <= kSweepMaxWords) {
    static std::atomic<bool> raised[64];
    const size_t smem = (size_t)kRing * kNmsBlock * nw * sizeof(unsigned long long);  // at most 96 KB
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return D3D_ERR_CUDA;
    if (smem > 40 * 1024 && !raised[dev].load(std::memory_order_acquire)) {
      if (cudaFuncSetAttribute(suppress_blocks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kRing * kNmsBlock * kSweepMaxWords * 8) != cudaSuccess)
        return D3D_ERR_CUDA;
      raised[dev].store(true, std::memory_order_release);
    }
    // started while the mask kernel drains; it waits for the mask itself
    D3D_LAUNCH(true, suppress_blocks_kernel, (unsigned)b, kSweepThreads, smem, st, mask, scores, k, nw, out);
  } else {
    suppress_kernel<<<b, 32, 0, st>>>(mask, scores, k, nw, out);
  }
  D3D_CHECK_LAUNCH();
  return D3D_OK;
}

extern "C" int d3d_nms3d_enqueue(const d3d_nms3d_params* p, const d3d_tensor_desc* in, int n_in,
                                 const d3d_tensor_desc* out, int n_out, const void* const* inputs,
                                 void* const* outputs, void* workspace, size_t workspace_bytes, void* stream) {
  D3D_NVTX_RANGE("d3d_nms3d_enqueue");
  D3D_REQUIRE(p && out && inputs && outputs && n_out >= 1, D3D_ERR_INVALID_ARGUMENT);
  int b, k, bd;
  int rc = nms_dims(in, n_in, &b, &k, &bd);
  if (rc != D3D_OK) return rc;
  if (b == 0 || k == 0) return D3D_OK;
  const int nw = (int)ceil_div(k, kNmsBlock);
  D3D_REQUIRE(workspace && workspace_bytes >= (size_t)b * k * nw * sizeof(unsigned long long),
              D3D_ERR_WORKSPACE_TOO_SMALL);
  return launch_nms(p, b, k, bd, nw, inputs, outputs, reinterpret_cast<unsigned long long*>(workspace), stream);
}

// ---------------------------------------------------------------------------------------------
// NMS3d without a caller-provided workspace.
//
// Some hosts of this library hand a plugin nothing but its input and output pointers and a stream, and are not
// allowed to obtain device memory themselves: a real-time perception loop that bans allocator calls once it is
// running, an engine that was built before the plugin asked for workspace, a thin C caller that owns no memory
// pool.  For them the overlap-mask scratch of NMS3d lives in the library image itself: a file-scope device
// array of fixed size.  Every GPU that loads the library keeps those 2 MiB until the process exits.
//
// `g_nms_static_mask` below is, in host code, only a handle for the symbol -- not a device address.  The address
// a kernel can use is looked up once per device with cudaGetSymbolAddress (with that device current) and cached;
// that look-up happens inside the first call on a device, which therefore should be made before any stream
// capture is started.  Nothing in the array has to start at zero: the mask kernel overwrites every word the
// suppression kernel reads, so stale contents of an earlier call are harmless.  All calls on one GPU share the
// one array: two calls that overlap on the GPU (different streams, or different threads) race on it.
// ---------------------------------------------------------------------------------------------
// D3D_NMS3D_STATIC_MAX_WORDS (include/deploy3d_b200.h): 256 Ki 64-bit mask words = 2 MiB; 10 x 1000 boxes need 160 000
static __device__ __align__(256) unsigned long long g_nms_static_mask[D3D_NMS3D_STATIC_MAX_WORDS];

namespace {
constexpr int kMaxStaticDevices = 64;
// per-device address of g_nms_static_mask, null = not yet known; atomic because any host thread may be the first
std::atomic<unsigned long long*> g_nms_static_ptr[kMaxStaticDevices];
}  // namespace

extern "C" int d3d_nms3d_enqueue_static(const d3d_nms3d_params* p, const d3d_tensor_desc* in, int n_in,
                                        const d3d_tensor_desc* out, int n_out, const void* const* inputs,
                                        void* const* outputs, void* stream) {
  D3D_NVTX_RANGE("d3d_nms3d_enqueue_static");
  D3D_REQUIRE(p && out && inputs && outputs && n_out >= 1, D3D_ERR_INVALID_ARGUMENT);
  int b, k, bd;
  int rc = nms_dims(in, n_in, &b, &k, &bd);
  if (rc != D3D_OK) return rc;
  if (b == 0 || k == 0) return D3D_OK;
  const int nw = (int)ceil_div(k, kNmsBlock);
  // the scratch is fixed: larger problems are refused, never truncated
  D3D_REQUIRE((size_t)b * k * nw <= (size_t)D3D_NMS3D_STATIC_MAX_WORDS, D3D_ERR_TOO_LARGE);
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxStaticDevices) return D3D_ERR_CUDA;
  unsigned long long* mask = g_nms_static_ptr[dev].load(std::memory_order_acquire);
  if (!mask) {
    void* addr = nullptr;
    if (cudaGetSymbolAddress(&addr, g_nms_static_mask) != cudaSuccess || !addr) return D3D_ERR_CUDA;
    mask = reinterpret_cast<unsigned long long*>(addr);
    g_nms_static_ptr[dev].store(mask, std::memory_order_release);  // the same value whichever thread stores it
  }
  // the same launches as the workspace variant, over the built-in scratch
  return launch_nms(p, b, k, bd, nw, inputs, outputs, mask, stream);
}
