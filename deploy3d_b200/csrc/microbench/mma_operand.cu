// Stand-alone measurement, not part of the library:
//     nvcc -gencode arch=compute_100a,code=sm_100a -O2 -o mma_operand mma_operand.cu && ./mma_operand
// Two properties the SPConvMM kernel is built on, for tcgen05.mma of M = 128, K = 16 (fp16, fp32 accumulator):
//   * what an MMA takes with its A operand in shared memory and in tensor memory, for N = 16 to 256 (16 issued in a row);
//   * what a warp needs to issue four MMAs and a commit when the whole warp runs the loop and one elected lane issues
//     (every operand is the same for the warp in a way the compiler can see), and when one lane runs the loop by itself.
// All 148 SMs run it, operands are zeros; one warp per SM issues `kStages` groups of MMAs.  Every wait is bounded.
// Prints cycles per MMA, from the first issue to the last completion, and cycles to issue a group.
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

constexpr int kStages = 512, kSmem = 96 * 1024;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred P;\n\t.reg .b32 r;\n\telect.sync r|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ bool try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mma_tensor(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.b32 p, 0, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc) : "memory");
}
__device__ __forceinline__ void mma_shared(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.b32 p, 0, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc) : "memory");
}

struct Result {
  long long total, issue;
  int gave_up;
};

// kTensor: A in tensor memory; kLane: one lane runs the loop; groups of kMmas, those of four with a commit each.
template <bool kTensor, bool kLane, int kMmas> __global__ void __launch_bounds__(128, 1) issue_kernel(int n, Result* out) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint64_t done, slot;
  __shared__ uint32_t base;
  const int warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < kSmem / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(smem)[i] = 0u;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&done)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&slot)));
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&base)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = base;
  for (int c = 0; c < 512; c += 16)  // zeros everywhere
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};"
                 ::"r"(tmem + ((uint32_t)(warp * 32) << 16) + c), "r"(0u) : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0) {
    const uint32_t idesc = (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
    const uint64_t hi = (uint64_t)((1024u >> 4) | (1u << 14) | (2u << 29)) << 32;  // 128-byte swizzle
    const uint32_t a_lo = ((smem_u32(smem) & 0x3FFFFu) >> 4) | (1u << 16), b_lo = a_lo + (32 * 1024 >> 4);
    const uint32_t a_tmem = tmem + 256;  // four units of 32 columns behind the accumulator
    auto group = [&](int s) {
#pragma unroll
      for (int m = 0; m < kMmas; ++m) {
        if (kTensor) mma_tensor(tmem, a_tmem + (s & 3) * 32 + m % 4 * 8, hi | (b_lo + m % 4 * 2), idesc);
        else mma_shared(tmem, hi | (a_lo + (s & 1) * 1024 + m % 4 * 2), hi | (b_lo + m % 4 * 2), idesc);
      }
      if (kMmas == 4) commit(&slot);
    };
    const long long t0 = clock64();
    if (kLane) {
      if ((threadIdx.x & 31) == 0)
        for (int s = 0; s < kStages; ++s) group(s);
      __syncwarp();
    } else {
      for (int s = 0; s < kStages; ++s) {
        if (elect_one()) group(s);
        __syncwarp();
      }
    }
    const long long t1 = clock64();
    if (kLane ? (threadIdx.x & 31) == 0 : elect_one()) commit(&done);
    __syncwarp();
    bool ok = false;
    for (int i = 0; i < 1000000 && !ok; ++i) ok = try_wait(&done, 0);
    const long long t2 = clock64();
    if (blockIdx.x == 0 && (threadIdx.x & 31) == 0) out->total = t2 - t0, out->issue = t1 - t0, out->gave_up = !ok;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

template <bool kTensor, bool kLane, int kMmas> void run(int n, Result* out) {
  auto kernel = issue_kernel<kTensor, kLane, kMmas>;
  Result r = {};
  bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) == cudaSuccess;
  for (int i = 0; i < 2 && ok; ++i) {
    kernel<<<148, 128, kSmem>>>(n, out);
    ok = cudaMemcpy(&r, out, sizeof(r), cudaMemcpyDeviceToHost) == cudaSuccess;
  }
  if (!ok) {
    printf("CUDA error: %s\n", cudaGetErrorString(cudaGetLastError()));
    exit(1);
  }
  printf("N %3d  A in %s memory  %2d MMAs%s, %-22s  %5.1f cycles per MMA  %6.1f cycles to issue a group  gave_up %d\n", n,
         kTensor ? "tensor" : "shared", kMmas, kMmas == 4 ? " and a commit" : "", kLane ? "loop run by one lane" : "elected lane of a warp",
         (double)r.total / kStages / kMmas, (double)r.issue / kStages, r.gave_up);
}

int main() {
  Result* out;
  if (cudaMalloc(&out, sizeof(Result)) != cudaSuccess) return 1;
  for (int n : {16, 32, 64, 128, 256}) {
    run<false, false, 16>(n, out);
    run<true, false, 16>(n, out);
  }
  for (int n : {16, 32, 64, 128, 256}) {
    run<true, false, 4>(n, out);
    run<true, true, 4>(n, out);
  }
  return 0;
}
