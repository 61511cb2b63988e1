// SPConvMM on the 5th-generation tensor cores: output-stationary implicit GEMM.
//
// For a tile of 128 consecutive output voxels and every kernel offset k that feeds at least one of them:
//   A = the input rows named by the neighbour table, gathered into registers and stored into tensor memory, from where
//       tcgen05.mma takes its A operand; rows without an input are zeros (the table carries a 128-bit row mask per
//       (tile, offset), and nothing is loaded for them),
//   B = W[k]^T, K-major in shared memory, by TMA (once per kernel when all offsets fit into 112 KB, else window by window),
//   D (+)= A * B (M = 128, N = Cout, K = 16 per instruction), fp32 accumulator in tensor memory.
// All offsets of a tile accumulate into the same columns, in ascending order; the epilogue reads them once, adds bias
// (+ residual), applies ReLU, converts and stores the row.  No atomics, no bias-initialisation pass.
// (The reference: gather iterator + mma.sync tiles of 64 pairs of one offset, fp16 accumulate, half2 atomicAdd
// scatter, trt/spconv/mm/kernel.h:84-179, mm/output_iterator.h:189-206.)
//
// Why A goes through registers into tensor memory (B200).  From shared memory an M128 K16 MMA takes 41 / 42 / 48 / 64 cycles
// at N = 16 / 32 / 64 / 128: the tensor core fetches 4 KB of A each time.  From tensor memory it takes 15 / 20 / 32 / 64
// (microbench/mma_operand.cu).  Zeros for missing rows cost nothing in registers, so no MMA carries a lane mask.  Plain loads go
// through L1, which the operand ring in shared memory had taken: neighbouring offsets and rows of a tile read the same voxels.
// And up to 128 output channels a weight block is fetched once for the two or three tiles a CTA works on together, not once per
// tile (with more there are too few accumulators for that, see open_round: one MMA warp and its two teams do the work).
// 27 offsets, us per launch, before (rows copied by cp.async into a shared-memory ring, MMAs under lane masks) and now:
// 16 -> 16 at 281 k voxels 33 / 31, 32 -> 32 at 463 k 81 / 67, 32 -> 64 at 463 k 96 / 75, 64 -> 64 at 238 k 80 / 65,
// 64 -> 128 101 / 87, 128 -> 128 at 66 k 59 / 51, 256 -> 128 at 50 k 82 / 73, 256 -> 256 115 / 115.
//
// Where a weight is not finite, 0 * W is not zero.  Such a layer takes the kernels without kWide: their products then leave the
// accumulator rows without an input alone (tcgen05.mma with a lane mask), and the accumulators start as zeros.
//
// What bounds it now: the instruction streams of the roles, again.  An SM needs 720 to 770 warp instructions for a unit (128 rows
// x 128 bytes) and issues 1.7 to 2.4 a cycle; a lone warp executes a dependent one every four to six cycles, and a trip through a
// full memory pipe (a barrier test, a shared-memory load) takes 70 cycles and more.  Hence:
//   * two or three MMA warps, each with a tile of the round (or its windows of the one tile a CTA has) and two producer teams of
//     its own: one warp needs about 470 cycles from one product to the next, whatever the tensor core could do -- four or six
//     teams to one warp are no faster;
//   * an MMA warp waits and issues in one elected lane, two units at a time, from values that the whole warp has computed
//     by counters: fed from memory or by a loop of one lane, the compiler cannot keep the descriptors in uniform registers, and
//     four MMAs with a commit take 223 cycles to issue instead of 143 (microbench/mma_operand.cu);
//   * the control warp lists the units of a round, so that a producer finds its next one with a single load;
//   * a lane of a producer holds two or four rows (rows_per_lane): 16-byte pieces dealt out lane by lane cost four times
//     the address arithmetic;
//   * ids, row masks, input and residual rows of the next round are prefetched into L2: the loads run one unit ahead, which
//     covers L2 but not DRAM (128 -> 128 at 66 k voxels behind other layers: 66.0 us without, 61.4 with).
// For 128 output channels the tensor pipe is busy half of the launch, and 128-row tiles round up (520 tiles on 148 SMs are 3.5,
// so 4).
//
// Roles of a CTA (persistent, one per SM) with T = 2 or 3 MMA warps: 8 T producer warps, 4 epilogue warps (8 for T = 2), T MMA
// warps, 1 control warp (lists, weights by TMA -- those that are held are fetched by
// the last MMA warp --, prefetches).  Units pass through a ring of 2 T slots in tensor memory, one per team
// of four producer warps (a warp can only write its quarter of the lanes).  Everything is handed over through mbarriers; every
// wait is bounded (about one second) and on expiry raises an error word, lets the CTA drain and return instead of spinning.
// A barrier is always waited for by the side that has seen its phase before (same team, same MMA warp, same epilogue warps):
// a waiter two phases ahead would take the phase before last for the one it waits for.
//
// A tile row need not stand for output tile * 128 + row: the table carries the output row of every tile row, and a
// table rebuilt by d3d_spconv_mm_regroup lists its outputs sorted by offset mask, so that a tile keeps only the few
// offsets its like outputs share; windows no tile of a round has are left out of it.
#include <cuda.h>

#include <mutex>
#include <new>
#include <type_traits>

#include "common.cuh"
#include "spconv_mm_internal.h"

namespace d3d {
namespace {

constexpr int kTileRows = 128;
constexpr int kUnitCols = 32;    // tensor-memory columns of one unit of A: 128 rows x 128 bytes
constexpr int kMaxAcc = 8;       // accumulators in tensor memory
constexpr int kMaxBSlots = 8;    // weight blocks in flight
constexpr int kTmemCols = 512;
constexpr int kMaxMmaWarps = 3;  // MMA warps, each with a tile of the round and two producer teams
constexpr int kListUnits = 128;  // units of a tile: 32 offsets of four parts
// Warp roles for T MMA warps: 8 T producer warps (2 T teams of four), four epilogue warps (whose index mod 4 covers the four
// TMEM lane quarters), the MMA warps and the control warp.
__host__ __device__ constexpr int epilogue_sets(int mma_warps) { return mma_warps == 2 ? 2 : 1; }
__host__ __device__ constexpr int threads_of(int mma_warps) { return (9 * mma_warps + 4 * epilogue_sets(mma_warps) + 1) * 32; }
constexpr uint32_t kWaitLimitCycles = 2000u * 1000u * 1000u;  // about a second; differences of the 32-bit clock hold twice that

__device__ int g_tc_error;  // 0 ok; otherwise the code of the first wait that gave up

// How the lanes of a producer warp share its 32 rows of a unit.  Rows of 128 bytes: four lanes to a row, 32 bytes of four
// rows each -- a load then takes 64 bytes of a line at a time instead of 32, and the L1 data pipe is what these layers run
// into.  Shorter rows: two lanes to a row, 64 bytes of two rows each (over all offsets of the unit): half the addresses,
// and the loaded registers are stored as they lie.
__host__ __device__ constexpr int rows_per_lane(int offs) { return offs == 1 ? 4 : 2; }

// The row of a tile's quarter (32 rows) that the producers put into TMEM lane `lane` of it.
__host__ __device__ constexpr int row_of_lane(int offs, int lane) {
  return 4 * (lane & 7) + (rows_per_lane(offs) == 4 ? lane >> 3 : 2 * (lane >> 3 & 1) + (lane >> 4));
}

// Short launches: the MMA warps share a tile, every window going to the next one.  Bit k: offset k lies in a window of warp i.
__host__ __device__ constexpr uint32_t every(int period, int width) {
  uint32_t bits = 0;
  for (int k = 0; k < 32; ++k) bits |= (k % period < width ? 1u : 0u) << k;
  return bits;
}
template <int kOffs, int kMma> __device__ __forceinline__ uint32_t offsets_of(int i) {
  constexpr uint32_t bits = every(kOffs * kMma, kOffs);
  return bits << (i * kOffs);
}
// Bit w: window w is warp i's.
template <int kMma> __device__ __forceinline__ uint32_t windows_of(int i) { return offsets_of<1, kMma>(i); }

struct TcParams {
  const int32_t* table;        // [tiles][kvol][128]
  const uint32_t* tile_mask;   // [tiles] bit k set: offset k feeds the tile
  const uint32_t* row_masks;   // [tiles][kvol][4] bit r of word q set: row 32 q + r has an input under the offset
  const int32_t* perm;         // [tiles][128] output row of every tile row, -1 = none
  const void* in_feats;        // [n_in_rows][cin]
  int64_t m_max;
  int32_t n_in_rows;  // rows of the gathered tensor
  int kvol, cin, cout;
  int num_tiles;
  int parts;          // units per kernel offset: cin / 64, at least 1
  int num_acc;        // accumulators
  int ring_col;       // first tensor-memory column of the ring
  int spread;         // the tiles of a CTA lie a grid apart, instead of side by side
  int regrouped;      // tiles in ascending order of their offset masks: dealt out costly ones first
  uint32_t b_bytes;   // one weight block: cout rows of row_bytes, per (offset, part)
  int b_slots;        // ring of weight windows; 0: all kvol blocks stay in shared memory
  int row_bytes;      // bytes of one weight row of a block = min(cin, 64) * 2
  uint32_t idesc;
  uint32_t layout_type;  // UMMA smem layout code: 6 = 32B, 4 = 64B, 2 = 128B swizzle
  const void* weights;  // all of them, in the layout of the tensor map
  const float* bias;
  void* out;
  const void* residual;
  int relu;
  int is_bf16;
  uint32_t wait_limit;  // cycles after which a wait gives up
  int table_wide;       // the table starts on 16 bytes
  int masked;           // a weight is not finite: products leave the accumulator rows without an input alone
};

// ---- PTX wrappers ------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Whether the phase is over, without waiting for it.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait.  Returns false (and leaves `code` in the flag) when the barrier did not flip within the limit or another role
// already gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code,
                                          uint32_t limit) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint32_t t0 = (uint32_t)clock();
  while (!mbar_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if ((uint32_t)clock() - t0 > limit) {
      *abort_flag = code;
      return false;
    }
  }
  return true;
}
// Waits for something the warp has set in motion itself and that needs no other role to end, whoever has given up meanwhile: a
// CTA must not end, nor return its tensor memory, while copies or MMAs of its own are on their way.
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {
  const uint32_t t0 = (uint32_t)clock();
  while (!mbar_try_wait(bar, parity) && (uint32_t)clock() - t0 <= kWaitLimitCycles) {
  }
}
__device__ __forceinline__ void tma_load_2d(const CUtensorMap* map, uint64_t* bar, void* dst, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      :
      : "r"(smem_u32(dst)), "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
// Programmatic dependent launch.  `pdl_release` lets the next kernel of the stream start its prologue once every CTA
// of this grid has called it (the CTAs of the next grid become resident as this grid's CTAs leave their SMs);
// `pdl_wait` blocks until the preceding grid has completed and its memory is visible.  Both are no-ops when the
// kernels were launched without the programmatic attribute.
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// True in exactly one lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred P;\n\t.reg .b32 r;\n\t"
      "elect.sync r|P, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// Waits for this thread's tensor-memory loads; `r` is what they have loaded.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

// D (+)= A * B, A in tensor memory.
__device__ __forceinline__ void umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D += A * B for the rows (lanes of D) whose bit in `rows` is set.
__device__ __forceinline__ void umma_f16_ta_rows(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                                 const uint32_t (&rows)[4]) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.eq.b32 p, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%4, %5, %6, %7}, p;\n\t}"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(~rows[0]), "r"(~rows[1]), "r"(~rows[2]), "r"(~rows[3])
      : "memory");
}
// Zeros in 16 columns of the warp's 32 TMEM lanes.
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};"
      ::"r"(taddr), "r"(0u) : "memory");
}
// Lane t of the warp writes registers 4c, 4c + 1 to columns 8c + 2 (t % 4) and the next of TMEM lane t / 4, registers
// 4c + 2, 4c + 3 to the same columns of lane t / 4 + 8, for c = 0..3.
__device__ __forceinline__ void tmem_st_16x256b_x4(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// Lane t of the warp writes register k to column 2k + t / 2 % 2 of TMEM lane t / 4 + 8 * (t % 2), for k = 0..15.
__device__ __forceinline__ void tmem_st_16x64b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x64b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// Loads 16 (kWords = 4) or 32 bytes (8) where `has`, else leaves v as it is; kWide: 32 bytes in one go, from an address
// that is a multiple of them.
template <int kWords, bool kWide> __device__ __forceinline__ void load_words(uint32_t* v, const unsigned char* src, bool has) {
  if (kWords == 4) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t@q ld.global.v4.b32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3])
        : "l"(src), "r"((int)has));
  } else if (kWide) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %9, 0;\n\t"
        "@q ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t}"
        : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])
        : "l"(src), "r"((int)has));
  } else {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %9, 0;\n\t"
        "@q ld.global.v4.b32 {%0, %1, %2, %3}, [%8];\n\t"
        "@q ld.global.v4.b32 {%4, %5, %6, %7}, [%8 + 16];\n\t}"
        : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])
        : "l"(src), "r"((int)has));
  }
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// A unit of work is 128 rows of a tile under the kOffs offsets of a window (one 64-channel part of them).  The producers'
// list of a round names for every unit the first (tile, offset) block of the table (x) and, in y, the part (bits 0-1) and
// the number of offsets (at most kOffs, bits 4-6).
struct __align__(16) Shared {
  uint2 units[2][kMaxMmaWarps][kListUnits];
  int4 round[2];              // tiles (none: the end), windows, units of a tile
  uint64_t list_full[2];      // control -> producers, MMA
  uint64_t list_empty[2];     // producers, MMA -> control
  uint64_t full[2 * kMaxMmaWarps];   // producers -> MMA
  uint64_t empty[2 * kMaxMmaWarps];  // MMA (tcgen05.commit) -> producers
  uint64_t acc_full[kMaxAcc];
  uint64_t acc_empty[kMaxAcc];
  uint64_t b_full[kMaxBSlots];
  uint64_t b_empty[kMaxBSlots];
  uint64_t drained[kMaxMmaWarps];  // the MMAs of a warp that gave up are over
  uint64_t b_ready;     // resident weights have landed
  uint64_t live_ready;  // `live` is known
  int live;             // where the tiles without an offset begin, found once for all roles
  uint32_t tmem_base;
  int abort_flag;
};

// Carved dynamic shared memory: weights (resident blocks or the ring of windows) aligned to 1024, bias, control block.
struct Smem {
  unsigned char* weights;
  float* bias;
  Shared* sh;
};
template <int kOffs> __device__ __forceinline__ Smem carve_smem(unsigned char* raw, const TcParams& p) {
  Smem s;
  s.weights = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
  const size_t blocks = p.b_slots ? (size_t)p.b_slots * 2 * kOffs : (size_t)((p.kvol + kOffs - 1) / kOffs * kOffs);
  s.bias = reinterpret_cast<float*>(s.weights + blocks * p.b_bytes);
  s.sh = reinterpret_cast<Shared*>(s.bias + ((p.cout + 3) & ~3));
  return s;
}

// ---- the order of the work -----------------------------------------------------------------------------------------
// A CTA takes its tiles in rounds, one for each of its MMA warps; a round walks the windows of kOffs kernel offsets that any of
// its tiles has, in ascending order (each window in `parts` units of 64 input channels), two (window, part)s at a time: one unit
// per (window, part, tile).  A weight block is thus used by all tiles of the round while it is in shared memory.  The control
// warp lists the units of a round for the producers; the MMA warps and the epilogue count along.
//
// Rounds cover the live tiles first, in whole rounds and one of the remaining tiles shared out evenly (157 tiles of 64 -> 64: one
// each and nine CTAs with two 14.7 us, 78 CTAs with two 16.0), then whatever lies behind them (tiles no offset feeds).  Launches
// of at most two tiles to a CTA are one round (p.spread).
//
// Launches of at most one tile to a CTA (kSplit): both MMA warps work on it, each window going to the next warp -- by its number,
// not by its place among those the tile has, so that a regrouped table gives the same sums --, with an accumulator, a list and
// weight slots each; the epilogue adds the two sums.  27 offsets and 6 k voxels, us with one warp / both: 16 -> 16 7.3 / 6.5,
// 32 -> 64 9.3 / 7.9, 64 -> 64 12.3 / 10.1, 128 -> 128 19.3 / 15.8 (7.1 and 5.8 at 32 -> 64 and 16 -> 16 since weights that are
// held are not asked for by the control warp).  A kernel of its own: the same by a flag costs 0.3 to 0.9 us,
// since a short launch fetches most of its code for the first time.
struct Round {
  int start;      // index of the round's first tile over all CTAs
  int next;       // of the next round's
  int first;      // of this CTA's (tiles in the order of the table)
  int limit;      // this CTA's tiles lie below this index
  int tiles;      // tiles of a CTA, at most
  uint32_t mask;  // lane i (mod 4): offset mask of the CTA's tile i, 0 = no such tile
};
// Where the tiles behind which no tile has an offset begin, found by the whole warp from the offset masks alone: up to a
// 128th of them late (that many are looked at, in one trip to L2; eight to a lane instead of four made the kernel large enough
// to cost 64 -> 128 at 238 k voxels 88 -> 93 us).  Where empty tiles lie between others the answer may be smaller; every CTA comes
// to the same one, which is what dealing the tiles out asks for.
__device__ __forceinline__ int live_tiles(const TcParams& p) {
  // (at most one tile to a CTA: nothing to deal out)
  if (p.spread || p.num_tiles <= (int)gridDim.x) return p.num_tiles;
  constexpr int kProbes = 4;
  const int step = (p.num_tiles + 32 * kProbes - 1) / (32 * kProbes);
  uint32_t mask[kProbes];
#pragma unroll
  for (int i = 0; i < kProbes; ++i) {
    const int64_t tile = (int64_t)(i * 32 + (threadIdx.x & 31)) * step;
    mask[i] = tile < p.num_tiles ? __ldg(p.tile_mask + tile) : 0u;
  }
  int parts = 0;  // up to the last probe with an offset
#pragma unroll
  for (int i = 0; i < kProbes; ++i) {
    const uint32_t has = __ballot_sync(0xffffffffu, mask[i] != 0u);
    if (has) parts = i * 32 + 32 - __clz(has);
  }
  const int64_t live = (int64_t)parts * step;
  return live < p.num_tiles ? (int)live : p.num_tiles;
}
// Index of the CTA's tile i in a round, and the tile it stands for.
__device__ __forceinline__ int tile_index(const TcParams& p, const Round& r, int i) {
  const int g = (int)gridDim.x, c = (int)blockIdx.x;
  if (!p.spread) return r.first + i;
  return r.start + i * g + (p.regrouped && (i & 1) ? g - 1 - c : c);
}
__device__ __forceinline__ int tile_of(const TcParams& p, int index) {
  return p.regrouped ? p.num_tiles - 1 - index : index;
}
template <int kMma, bool kSplit> __device__ __forceinline__ void open_round(const TcParams& p, int live, int start, Round& r) {
  const int g = (int)gridDim.x;
  const int end = start < live ? live : p.num_tiles;
  // With few accumulators one tile at a time: an MMA warp that had no tile in the round before must not be able to wait for
  // an accumulator whose use before last has not been read yet -- the phase would be taken for the one it waits for.  It is
  // at most 2 kMma - 2 tiles ahead of the first tile that another warp may still be at.
  const int rest = end - start, most = !kSplit && p.num_acc >= 2 * kMma - 1 ? kMma : 1;
  r.tiles = rest >= most * g ? most : rest <= 0 ? 0 : (rest + g - 1) / g;
  // the first `more` CTAs take all of them, the others one less
  const int c = (int)blockIdx.x, less = r.tiles - 1, more = rest - less * g < g ? rest - less * g : g;
  r.start = start, r.next = start + less * g + more;
  r.first = start + c * less + (c < more ? c : more);
  r.limit = p.spread ? r.next : r.first + less + (c < more ? 1 : 0);
  const int i = threadIdx.x & 3;
  const int index = tile_index(p, r, i);
  r.mask = (i < r.tiles && index < r.limit) ? __ldg(p.tile_mask + tile_of(p, index)) : 0u;
}
// 16 accumulator columns of this thread's row: bias (+ residual), ReLU, convert, 32 bytes stored.  Two columns to an
// instruction where there is one for it: this runs on four warps that share the SM's issue slots with all producers.
template <bool kBf16, bool kAdd>
__device__ __forceinline__ void store_chunk(const uint32_t (&acc)[16], const float* bias_s, unsigned short* o,
                                            const uint4 (&res)[2], int relu, bool wide) {
  uint32_t w[8];
  const uint4* b4 = reinterpret_cast<const uint4*>(bias_s);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint4 b = b4[q];
    const uint32_t bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float x, y;
      asm("{\n\t.reg .b64 s, t;\n\tmov.b64 s, {%2, %3};\n\tmov.b64 t, {%4, %5};\n\tadd.rn.f32x2 s, s, t;\n\t"
          "mov.b64 {%0, %1}, s;\n\t}"
          : "=f"(x), "=f"(y)
          : "r"(acc[4 * q + 2 * h]), "r"(acc[4 * q + 2 * h + 1]), "r"(bb[2 * h]), "r"(bb[2 * h + 1]));
      if (kAdd) {
        const uint4& r4 = res[q / 2];
        const uint32_t r = q % 2 == 0 ? (h == 0 ? r4.x : r4.y) : (h == 0 ? r4.z : r4.w);
        if (relu == 2) x = fmaxf(x, 0.f), y = fmaxf(y, 0.f);  // activation before the residual is added
        if (kBf16) {
          x += __uint_as_float(r << 16), y += __uint_as_float(r & 0xFFFF0000u);
        } else {
          const __half2 hh = *reinterpret_cast<const __half2*>(&r);
          x += __low2float(hh), y += __high2float(hh);
        }
      }
      // the activation after the rounding: the same values (the maximum of a NaN and zero is zero either way)
      const bool clamp = relu == 1 || (relu == 2 && !kAdd);
      if (kBf16) {
        __nv_bfloat162 t = __floats2bfloat162_rn(x, y);
        if (clamp) t = __hmax2(t, __float2bfloat162_rn(0.f));
        w[2 * q + h] = *reinterpret_cast<uint32_t*>(&t);
      } else {
        __half2 t = __floats2half2_rn(x, y);
        if (clamp) t = __hmax2(t, __float2half2_rn(0.f));
        w[2 * q + h] = *reinterpret_cast<uint32_t*>(&t);
      }
    }
  }
  if (wide) {  // a whole sector
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                 "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
  } else {
    uint4* o4 = reinterpret_cast<uint4*>(o);
    o4[0] = make_uint4(w[0], w[1], w[2], w[3]);
    o4[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// Barrier initialisation and the TMEM allocation (by the first MMA warp); returns the TMEM base address.
template <bool kWide, int kMma, bool kSplit>
__device__ __forceinline__ uint32_t cta_setup(const TcParams& p, const Smem& s) {
  Shared* sh = s.sh;
  // all of this stands in front of a short launch: a barrier of every kind to a lane
  const int i = threadIdx.x;
  if (i < 32) {
    if (i < 2 * kMma) mbar_init(&sh->full[i], 4), mbar_init(&sh->empty[i], 1);
    if (i < kMma) mbar_init(&sh->drained[i], 1);
    if (i < p.num_acc) mbar_init(&sh->acc_full[i], 1), mbar_init(&sh->acc_empty[i], 4 * epilogue_sets(kMma));
    if (i < p.b_slots) mbar_init(&sh->b_full[i], 1), mbar_init(&sh->b_empty[i], kSplit ? 1 : kMma);
    if (i < 2) mbar_init(&sh->list_full[i], 1), mbar_init(&sh->list_empty[i], 9 * kMma);
    if (i == 0) {
      mbar_init(&sh->b_ready, 1), mbar_init(&sh->live_ready, 1);
      sh->abort_flag = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if ((int)(threadIdx.x >> 5) == 8 * kMma + 4 * epilogue_sets(kMma)) tmem_alloc(&sh->tmem_base, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (!kWide && p.masked) {  // accumulators start as zeros, and the epilogue leaves them so
    const int warp = (int)(threadIdx.x >> 5);
    if (warp >= 8 * kMma && warp < 8 * kMma + 4) {
      for (int c = 0; c < p.num_acc * p.cout; c += 16) tmem_zero16(sh->tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + c);
      tmem_st_wait();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }
  return sh->tmem_base;
}

// All roles meet, then the allocating warp returns the tensor memory and reports a wait that gave up.
template <int kMma>
__device__ __forceinline__ void cta_teardown(const Smem& s, uint32_t tmem_base) {
  tc_fence_before();
  __syncthreads();
  if ((int)(threadIdx.x >> 5) == 8 * kMma + 4 * epilogue_sets(kMma)) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
    if (s.sh->abort_flag && elect_one()) atomicCAS(&g_tc_error, 0, s.sh->abort_flag);
  }
}

// ---- producers -------------------------------------------------------------------------------------------------------
template <int kOffs, bool kWide, int kMma, bool kSplit>
__device__ __forceinline__ void producer_role(const TcParams& p, const Smem& s, uint32_t tmem_base, int warp, int lane) {
  constexpr int kRows = rows_per_lane(kOffs);
  constexpr int kWords = kOffs == 4 ? 4 : 8;               // 32-bit words a lane loads at a time
  constexpr int kLoads = 32 / (kRows * kOffs * kWords);    // loads per row and offset
  Shared* sh = s.sh;
  volatile int* abort_flag = &sh->abort_flag;
  const int team = warp / 4, quarter = warp % 4;
  // this lane reads piece `piece` of tile rows 32 * quarter + row0 and the next (kRows of them)
  const int row0 = kRows == 4 ? lane >> 2 << 2 : 4 * (lane >> 2) + 2 * (lane & 1);
  const int piece = kRows == 4 ? lane & 3 : lane >> 1 & 1;
  const unsigned char* src_lane = reinterpret_cast<const unsigned char*>(p.in_feats) + piece * (kWords * 4);
  const int32_t* ids_lane = p.table + quarter * 32 + row0;
  const uint32_t* rows_lane = p.row_masks + quarter;
  const uint32_t row_bytes = (uint32_t)p.cin * 2;
  const uint32_t last_in_row = (uint32_t)p.n_in_rows - 1u;
  const uint32_t dst = tmem_base + (uint32_t)(p.ring_col + team * kUnitCols) + ((uint32_t)(quarter * 32) << 16);

  const int owner = team % kMma;  // the MMA warp this team works for
  int buf = 0, n = team / kMma, len = 0;  // the unit's place in that warp's list
  uint32_t list_phase = 0;
  bool open = false;  // list `buf` is out
  enum { kUnit, kLater, kEnd };
  // Makes list[n] a unit, going to the next rounds if need be.  Does not wait for a list unless `block`: with a unit in
  // hand that would be a deadlock, for the next list comes after the last weights of this one.
  auto settle = [&](bool block) -> int {
    while (!open || n >= len) {
      if (open) {  // done with this one
        n -= len;
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->list_empty[buf]);
        if (buf) list_phase ^= 1;
        buf ^= 1;
        open = false;
      }
      if (!block && !__all_sync(0xffffffffu, mbar_test(&sh->list_full[buf], list_phase))) return kLater;
      if (!__all_sync(0xffffffffu, mbar_wait(&sh->list_full[buf], list_phase, abort_flag, 13, p.wait_limit))) return kEnd;
      const int4 round = sh->round[buf];
      if (round.x == 0) return kEnd;
      len = kSplit ? __popc((uint32_t)round.y & windows_of<kMma>(owner)) * p.parts : owner < round.x ? round.z : 0;
      open = true;
    }
    return kUnit;
  };
  struct Unit {
    int32_t id[kOffs][kRows];
    uint32_t rows[kOffs];  // bit i: row i of the quarter has an input under the offset
    int part;
  } cur;
  auto load_unit = [&]() {
    const uint2 e = sh->units[buf][owner][n];
    cur.part = e.y & 3u;
    const int offs = (int)(e.y >> 4);
    const int32_t* ids = ids_lane + (int64_t)e.x * kTileRows;
    const uint32_t* rows = rows_lane + (int64_t)e.x * 4;
#pragma unroll
    for (int o = 0; o < kOffs; ++o) {
      const bool in = o == 0 || o < offs;
      if (!kWide && !p.table_wide) {
#pragma unroll
        for (int i = 0; i < kRows; ++i) cur.id[o][i] = in ? __ldg(ids + o * kTileRows + i) : 0;
      } else if (kRows == 4) {
        const int4 q = in ? __ldg(reinterpret_cast<const int4*>(ids + o * kTileRows)) : make_int4(0, 0, 0, 0);
        cur.id[o][0] = q.x, cur.id[o][1] = q.y, cur.id[o][kRows - 2] = q.z, cur.id[o][kRows - 1] = q.w;
      } else {
        const int2 q = in ? __ldg(reinterpret_cast<const int2*>(ids + o * kTileRows)) : make_int2(0, 0);
        cur.id[o][0] = q.x, cur.id[o][1] = q.y;
      }
      cur.rows[o] = in ? __ldg(rows + o * 4) : 0u;
    }
  };
  pdl_wait();  // masks, ids and features may come from the preceding kernels
  uint32_t phase = 1;
  int next = settle(true);
  if (next == kUnit) load_unit();
  while (next == kUnit) {
    uint32_t v[kRows][32 / kRows];  // the words of the lane's rows
    const unsigned char* src = src_lane + cur.part * 128;
#pragma unroll
    for (int i = 0; i < kRows; ++i)
#pragma unroll
      for (int q = 0; q < 32 / kRows; ++q) v[i][q] = 0u;
#pragma unroll
    for (int o = 0; o < kOffs; ++o) {
      const uint32_t rows = cur.rows[o] >> row0;
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        const bool has = (rows >> i) & 1u;
#ifdef DEPLOY3D_BOUNDS_CHECK
        if (has) (void)D3D_BOUNDS_OK(cur.id[o][i], 0, (long long)last_in_row + 1, kSiteMmTcId);
#endif
        // an id beyond the tensor is clamped to its last row
        const unsigned char* row = src + (uint64_t)min((uint32_t)cur.id[o][i], last_in_row) * row_bytes;
#pragma unroll
        for (int c = 0; c < kLoads; ++c)
          load_words<kWords, kWide>(&v[i][(o * kLoads + c) * kWords], row + c * 64, has);
      }
    }
    n += 2;
    next = settle(false);
    if (next == kUnit) load_unit();  // in flight while this unit's rows arrive
    if (!__all_sync(0xffffffffu, mbar_wait(&sh->empty[team], phase, abort_flag, 12, p.wait_limit))) return;
    tc_fence_after();
    if constexpr (kRows == 4) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // rows 0, 1 and 2, 3, interleaved by two words
        uint32_t w[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) w[q] = v[2 * h + (q >> 1 & 1)][(q >> 2) * 2 + (q & 1)];
        tmem_st_16x256b_x4(dst + ((uint32_t)(16 * h) << 16), w);
      }
    } else {
      tmem_st_16x64b_x16(dst, v[0]);
      tmem_st_16x64b_x16(dst + (16u << 16), v[kRows - 1]);
    }
    tmem_st_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh->full[team]);
    phase ^= 1;
    if (next == kLater && (next = settle(true)) == kUnit) load_unit();
  }
}

// ---- control warp ----------------------------------------------------------------------------------------------------
// Low word of a K-major operand descriptor: start address in 16-byte units, leading byte offset 1 (unused for the
// swizzled K-major layouts).  Advancing the operand by `d` bytes adds d / 16 to this word.
__device__ __forceinline__ uint32_t desc_lo(uint32_t smem_addr) { return ((smem_addr & 0x3FFFFu) >> 4) | (1u << 16); }

__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  if (bytes) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
// Brings what a round reads towards the SM: ids and row masks of its tiles, the rows of the input that lie where the outputs
// do (a submanifold layer gathers each of them, here or in a tile nearby), the rows of the residual.  The producers are only
// one unit ahead with their loads, which covers L2 but not DRAM (64 -> 64 at 238 k voxels behind other layers: 77.8 us without).
template <bool kWide> __device__ __forceinline__ void prefetch_round(const TcParams& p, int live, const Round& r) {
  const int i = threadIdx.x & 31, index = tile_index(p, r, i);
  if (i >= r.tiles || index >= r.limit || index >= live) return;
  const int64_t tile = tile_of(p, index), row = tile * kTileRows;
  if (kWide || p.table_wide) {
    prefetch_l2(p.table + tile * p.kvol * kTileRows, (uint32_t)(p.kvol * kTileRows * 4));
    prefetch_l2(p.row_masks + tile * p.kvol * 4, (uint32_t)(p.kvol * 16));
  }
  if (p.regrouped) return;
  const int64_t in = p.n_in_rows == p.m_max && row < p.n_in_rows ? p.n_in_rows - row : 0, out = p.m_max - row;
  prefetch_l2(reinterpret_cast<const unsigned char*>(p.in_feats) + row * p.cin * 2,
              (uint32_t)(in < kTileRows ? in : kTileRows) * p.cin * 2);
  if (p.residual)
    prefetch_l2(reinterpret_cast<const unsigned char*>(p.residual) + row * p.cout * 2,
                (uint32_t)(out < kTileRows ? out : kTileRows) * p.cout * 2);
}

// Lists the units of every round and brings in weights that are not held, the block of every (window, part) as soon as a slot
// is free.
template <int kOffs, bool kWide, int kMma, bool kSplit>
__device__ __forceinline__ void control_role(const TcParams& p, const Smem& s, const CUtensorMap* map_b) {
  constexpr uint32_t kWindow = kOffs == 1 ? 1u : kOffs == 2 ? 3u : 15u;
  constexpr int kWindows = 32 / kOffs;
  Shared* sh = s.sh;
  volatile int* abort_flag = &sh->abort_flag;
  const int lane = threadIdx.x & 31;
  const uint32_t b_tx = (uint32_t)p.cout * p.row_bytes;
  const bool resident = p.b_slots == 0;
  const int parts = p.parts, ring_slots = kSplit ? p.b_slots / kMma : p.b_slots;
  if (!resident && lane == 0) {  // (constants of the layer) a slice of the weights for every CTA, towards L2
    const uint32_t bytes = (uint32_t)p.kvol * (uint32_t)p.cout * (uint32_t)p.cin * 2u;
    const uint32_t slice = (bytes / gridDim.x + 127u) & ~127u, from = blockIdx.x * slice;
    if (from < bytes)
      prefetch_l2(reinterpret_cast<const unsigned char*>(p.weights) + from, bytes - from < slice ? bytes - from : slice);
  }
  __syncwarp();
  pdl_wait();  // the offset masks come from the preceding kernels
  Round r;
  open_round<kMma, kSplit>(p, p.num_tiles, 0, r);  // as if all were live, so that the masks are on their way
  const int live = kSplit ? p.num_tiles : live_tiles(p);
  if (!kSplit && lane == 0) {
    sh->live = live;
    mbar_arrive(&sh->live_ready);
  }
  if (!kSplit && live < r.tiles * (int)gridDim.x && live < p.num_tiles) open_round<kMma, kSplit>(p, live, 0, r);  // not a whole round
  int buf = 0, b_slot = 0;
  uint32_t list_phase = 0, b_phase = 0;
  bool ok = true;  // no wait for a weight slot has given up
  for (;;) {
    const bool end = r.tiles == 0;
    uint32_t masks[kMma], all = 0;
    int count = 0;
#pragma unroll
    for (int i = 0; i < kMma; ++i) {
      masks[i] = __shfl_sync(0xffffffffu, r.mask, i);
      all |= masks[i], count += masks[i] != 0u;
    }
    const Round done = r;
    if (all == 0u && !end) {
      open_round<kMma, kSplit>(p, live, done.next, r);
      continue;
    }
    if (!__all_sync(0xffffffffu, mbar_wait(&sh->list_empty[buf], list_phase ^ 1, abort_flag, 14, p.wait_limit))) break;
    // lane w lists window w
    const uint32_t bits = lane < kWindows ? kWindow << (lane * kOffs) : 0u;
    const bool present = (all & bits) != 0u;
    const uint32_t windows = __ballot_sync(0xffffffffu, present);
    const int rank = __popc(windows & lanemask_lt());  // of the window in the round
    const int steps = __popc(windows) * parts;
    const int offs = p.kvol - lane * kOffs < kOffs ? p.kvol - lane * kOffs : kOffs;
    if (kSplit && present) {
      const uint32_t blk = (uint32_t)tile_of(p, tile_index(p, done, 0)) * (uint32_t)p.kvol + (uint32_t)(lane * kOffs);
      const int own = __popc(windows & windows_of<kMma>(lane % kMma) & lanemask_lt());
      for (int part = 0; part < parts; ++part)
        sh->units[buf][lane % kMma][own * parts + part] = make_uint2(blk, (uint32_t)part | (uint32_t)offs << 4);
    } else if (present) {
      int place = 0;  // of the tile among the round's tiles that have an offset
#pragma unroll
      for (int i = 0; i < kMma; ++i) {
        if (masks[i] == 0u) continue;
        const uint32_t blk = (uint32_t)tile_of(p, tile_index(p, done, i)) * (uint32_t)p.kvol + (uint32_t)(lane * kOffs);
        for (int part = 0; part < parts; ++part)
          sh->units[buf][place][rank * parts + part] = make_uint2(blk, (uint32_t)part | (uint32_t)offs << 4);
        ++place;
      }
    }
    if (lane == 0) sh->round[buf] = make_int4(count, (int)windows, steps, 0);
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh->list_full[buf]);
    if (buf) list_phase ^= 1;
    buf ^= 1;
    if (end) break;
    open_round<kMma, kSplit>(p, live, done.next, r);  // the next round's masks are on their way
    prefetch_round<kWide>(p, live, r);
    if (!resident) {
      // two (window, part)s to a slot; the MMA warps that share a tile have slots of their own, lane i counts those of warp i
      constexpr int kRings = kSplit ? kMma : 1;
      uint32_t rest = kSplit ? windows & windows_of<kMma>(lane % kMma) : windows;
      int part = 0, todo = __popc(rest) * parts;
      while (ok && __any_sync(0xffffffffu, lane < kRings && todo > 0)) {
#pragma unroll 1
        for (int ring = 0; ring < kRings; ++ring) {
          const int left = kSplit ? __shfl_sync(0xffffffffu, todo, ring) : todo;
          if (left <= 0) continue;
          const int slot = kSplit ? __shfl_sync(0xffffffffu, b_slot, ring) + ring * ring_slots : b_slot;
          const uint32_t phase = kSplit ? __shfl_sync(0xffffffffu, b_phase, ring) : b_phase;
          ok = __all_sync(0xffffffffu, mbar_wait(&sh->b_empty[slot], phase ^ 1, abort_flag, 11, p.wait_limit));
          if (!ok) break;
          if (lane == (kSplit ? ring : 0)) {
            const int both = left > 1 ? 2 : 1;
            mbar_arrive_expect_tx(&sh->b_full[slot], (uint32_t)(both * kOffs) * b_tx);
            for (int h = 0; h < both; ++h) {
              const int k = (__ffs(rest) - 1) * kOffs;
#pragma unroll
              for (int o = 0; o < kOffs; ++o)  // behind the last offset: zeros, as above
                tma_load_2d(map_b, &sh->b_full[slot], s.weights + (size_t)((slot * 2 + h) * kOffs + o) * p.b_bytes, part * 64,
                            (k + o) * p.cout);
              if (++part == parts) part = 0, rest &= rest - 1u;
            }
          }
          if (!kSplit || lane == ring) {
            todo -= 2;
            if (++b_slot == ring_slots) b_slot = 0, b_phase ^= 1;
          }
          __syncwarp();
        }
      }
      if (!ok) break;
    }
  }
  // the last weights of every slot have landed
  if (resident) mbar_drain(&sh->b_ready, 0);
  for (int b = 0; b < ring_slots; ++b)
    if (lane < (kSplit ? kMma : 1)) mbar_drain(&sh->b_full[lane * ring_slots + b], b < b_slot ? b_phase : b_phase ^ 1);
  __syncwarp();
}

// ---- MMA warps -------------------------------------------------------------------------------------------------------
// One tile of a round (kSplit: its windows of the tile).  The warp walks the round together and by counters: what feeds an MMA
// has to be the same for the whole warp in a way the compiler can see.
template <int kOffs, bool kWide, int kMma, bool kSplit>
__device__ __forceinline__ void mma_role(const TcParams& p, const Smem& s, const CUtensorMap* map_b, uint32_t tmem_base, int me) {
  constexpr int kSteps = 4 / kOffs;  // MMAs (K = 16) per offset of a unit
  Shared* sh = s.sh;
  volatile int* abort_flag = &sh->abort_flag;
  // descriptor high word: stride between 8-row groups, version, swizzle mode
  const uint64_t desc_hi = (uint64_t)(((8u * (uint32_t)p.row_bytes) >> 4) | (1u << 14) | (p.layout_type << 29)) << 32;
  const uint32_t b_step = p.b_bytes >> 4, b_lo0 = desc_lo(smem_u32(s.weights));
  const uint32_t idesc = p.idesc;
  const uint32_t ring = tmem_base + (uint32_t)p.ring_col;
  const bool resident = p.b_slots == 0;
  const int parts = p.parts, num_acc = p.num_acc;
  const int b_first = kSplit ? me * (p.b_slots / kMma) : 0, b_end = kSplit ? b_first + p.b_slots / kMma : p.b_slots;
  const uint32_t cout = (uint32_t)p.cout;
  // Weights that are held: constants of the layer, whose load does not wait for the preceding kernel.  The last MMA warp asks for
  // them: 28 loads take a lane 1.1 us, which the control warp would spend in front of the first list.
  if (resident && me == kMma - 1 && elect_one()) {
    // blocks behind the last offset, up to a whole window: rows beyond the tensor, which TMA fills with zeros
    const int blocks = (p.kvol + kOffs - 1) / kOffs * kOffs;
    mbar_arrive_expect_tx(&sh->b_ready, (uint32_t)blocks * (cout * p.row_bytes));
    for (int k = 0; k < blocks; ++k) tma_load_2d(map_b, &sh->b_ready, s.weights + (size_t)k * p.b_bytes, 0, k * p.cout);
  }
  __syncwarp();
  if (resident && !__all_sync(0xffffffffu, mbar_wait(&sh->b_ready, 0, abort_flag, 23, p.wait_limit))) return;
  pdl_wait();  // the first list comes after the preceding kernels, which may take longer than a wait is allowed to
  // the slots of this warp's two teams, taken in turn
  const uint32_t a_of[2] = {ring + (uint32_t)(me * kUnitCols), ring + (uint32_t)((me + kMma) * kUnitCols)};
  uint64_t* const full_of[2] = {&sh->full[me], &sh->full[me + kMma]};
  uint64_t* const empty_of[2] = {&sh->empty[me], &sh->empty[me + kMma]};
  int buf = 0, b_slot = b_first, acc0 = 0;
  uint32_t list_phase = 0, b_phase = 0, turn = 0, acc_phase = 0;  // turn: bit 0 the slot, bit 1 its phase
  bool ok = true;  // no wait has given up
  for (;;) {
    ok = __all_sync(0xffffffffu, mbar_wait(&sh->list_full[buf], list_phase, abort_flag, 15, p.wait_limit));
    if (!ok) break;
    const int4 round = sh->round[buf];
    const int count = (int)__reduce_or_sync(0xffffffffu, (unsigned)round.x);
    const uint32_t windows = __reduce_or_sync(0xffffffffu, kSplit ? (unsigned)round.y & windows_of<kMma>(me) : (unsigned)round.y);
    if (count == 0) break;
    // this warp's tile of the round, if there is one, and its accumulator (of a shared tile even where it has no window)
    const bool mine = kSplit || me < count;
    const bool wrap = !kSplit && acc0 + me >= num_acc;
    const int acc = wrap ? acc0 + me - num_acc : acc0 + me;
    const uint32_t d_addr = tmem_base + (uint32_t)acc * cout;
    ok = !mine || __all_sync(0xffffffffu, mbar_wait(&sh->acc_empty[acc], acc_phase ^ (wrap ? 0u : 1u), abort_flag, 22, p.wait_limit));
    if (!ok) break;
    tc_fence_after();
    uint32_t add = 0u;  // the first products of a round start the sums
    uint32_t rest = windows;
    const int steps = __popc(windows) * parts;
    for (int seq = 0; seq < steps; seq += 2) {  // two (window, part)s at a time
      const bool both = seq + 1 < steps;
      uint32_t b_lo[2];
      if (resident) {
        b_lo[0] = b_lo0 + (uint32_t)((__ffs(rest) - 1) * kOffs) * b_step;
        rest &= rest - 1u;
        b_lo[1] = b_lo0 + (uint32_t)((__ffs(rest) - 1) * kOffs) * b_step;
        rest &= rest - 1u;
      } else {
        b_lo[0] = b_lo0 + (uint32_t)(b_slot * 2 * kOffs) * b_step;
        b_lo[1] = b_lo[0] + (uint32_t)kOffs * b_step;
      }
      uint64_t desc[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int m = 0; m < 4; ++m)
          desc[h][m] = desc_hi | (b_lo[h] + (uint32_t)(m / kSteps) * b_step + 2u * (m % kSteps));
      const bool odd = turn & 1u;
      const uint32_t a_addr[2] = {odd ? a_of[1] : a_of[0], odd ? a_of[0] : a_of[1]};
      uint64_t* const full[2] = {odd ? full_of[1] : full_of[0], odd ? full_of[0] : full_of[1]};
      uint64_t* const empty[2] = {odd ? empty_of[1] : empty_of[0], odd ? empty_of[0] : empty_of[1]};
      if (!kWide && p.masked) {
        // Under the row masks of every offset, one unit after the other; the masks come from L2 (64 -> 64 at 238 k voxels: 94 us,
        // without them 76).
        for (int h = 0; h < (both ? 2 : 1); ++h) {
          uint32_t rows[kOffs][4];
          if (mine) {
            const uint2 e = sh->units[buf][me][seq + h];
#pragma unroll
            for (int o = 0; o < kOffs; ++o)
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint32_t word = o < (int)(e.y >> 4) ? __ldg(p.row_masks + ((int64_t)e.x + o) * 4 + q) : 0u;
                rows[o][q] = __ballot_sync(0xffffffffu, (word >> row_of_lane(kOffs, threadIdx.x & 31)) & 1u);
              }
          }
          if (elect_one() && ok) {
            if (!resident && h == 0) ok = mbar_wait(&sh->b_full[b_slot], b_phase, abort_flag, 24, p.wait_limit);
            ok = ok && (!mine || mbar_wait(full[h], ((turn + (uint32_t)h) >> 1) & 1u, abort_flag, 21, p.wait_limit));
            if (ok && mine) {
              tc_fence_after();
#pragma unroll
              for (int m = 0; m < 4; ++m) {
                const uint32_t(&r)[4] = rows[m / kSteps];
                if (r[0] | r[1] | r[2] | r[3]) umma_f16_ta_rows(d_addr, a_addr[h] + 8 * m, desc[h][m], idesc, r);
              }
              umma_commit(empty[h]);
            }
            if (!resident && ok && h == (both ? 1 : 0)) umma_commit(&sh->b_empty[b_slot]);
          }
          __syncwarp();
        }
      } else
      // One lane waits and issues, for both windows at once: every instruction of this warp between two products is one too
      // many.  After a wait that gave up it issues nothing.
      if (elect_one() && ok) {
        if (!resident) ok = mbar_wait(&sh->b_full[b_slot], b_phase, abort_flag, 24, p.wait_limit);
        auto unit = [&](int h) {
          ok = ok && mbar_wait(full[h], ((turn + (uint32_t)h) >> 1) & 1u, abort_flag, 21, p.wait_limit);
          if (!ok) return;
          tc_fence_after();
          umma_f16_ta(d_addr, a_addr[h], desc[h][0], idesc, h ? 1u : add);
#pragma unroll
          for (int m = 1; m < 4; ++m) umma_f16_ta(d_addr, a_addr[h] + 8 * m, desc[h][m], idesc, 1u);
          umma_commit(empty[h]);  // the slot may be refilled once these MMAs have read it
        };
        if (mine) {
          unit(0);
          if (both) unit(1);
        }
        if (!resident && ok) umma_commit(&sh->b_empty[b_slot]);
      }
      __syncwarp();
      add = 1u;
      if (mine) turn = (turn + (both ? 2u : 1u)) & 3u;
      if (!resident && ++b_slot == b_end) b_slot = b_first, b_phase ^= 1;
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) break;
    if (elect_one()) {
      if (mine) umma_commit(&sh->acc_full[acc]);
      mbar_arrive(&sh->list_empty[buf]);
    }
    __syncwarp();
    if (buf) list_phase ^= 1;
    buf ^= 1;
    acc0 += kSplit ? kMma : count;
    if (acc0 >= num_acc) acc0 -= num_acc, acc_phase ^= 1;
  }
  if (!ok) {  // nobody reads these accumulators: see the MMAs out here
    if (elect_one()) umma_commit(&sh->drained[me]);
    __syncwarp();
    mbar_drain(&sh->drained[me], 0);
  }
}

// ---- epilogue --------------------------------------------------------------------------------------------------------
// Epilogue warp `quad` (= warp index mod 4: it may touch TMEM lanes [32*quad, 32*quad + 32)) of set `set`: the sets share
// the columns of every tile, so that an accumulator is free again soon (of 256 output channels there is only one).
template <int kOffs, bool kWide, int kMma, bool kSplit>
__device__ __forceinline__ void epilogue_role(const TcParams& p, const Smem& s, uint32_t tmem_base, int quad, int set) {
  Shared* sh = s.sh;
  volatile int* abort_flag = &sh->abort_flag;
  const int lane = threadIdx.x & 31;
  const int row_in_tile = quad * 32 + row_of_lane(kOffs, lane);
  const bool wide = reinterpret_cast<uintptr_t>(p.out) % 32 == 0;
  const int half = epilogue_sets(kMma) == 2 ? (p.cout + 31) / 32 * 16 : p.cout;
  const int from = set ? half : 0, to = set ? p.cout : half;
  int acc = 0;
  uint32_t acc_phase = 0;
  const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
  {
    constexpr int kThreads = 128 * epilogue_sets(kMma);
    for (int c = set * 128 + quad * 32 + lane; c < p.cout; c += kThreads) s.bias[c] = __ldg(p.bias + c);
    asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");  // the epilogue warps
  }
  pdl_wait();  // residual rows come from an earlier layer; output rows may still be read by the preceding kernel
  if (!kSplit && !__all_sync(0xffffffffu, mbar_wait(&sh->live_ready, 0, abort_flag, 32, p.wait_limit))) return;
  const int live = kSplit ? p.num_tiles : sh->live;
  Round r;
  open_round<kMma, kSplit>(p, live, 0, r);
  if (quad == 0 && set == 0) prefetch_round<kWide>(p, live, r);  // of the first round; the control warp sees to the others
  for (; r.tiles; open_round<kMma, kSplit>(p, live, r.next, r)) {
    for (int i = 0; i < r.tiles; ++i) {
      const uint32_t mask = __shfl_sync(0xffffffffu, r.mask, i);
      const int index = tile_index(p, r, i);
      if (index >= r.limit) continue;
      const int64_t row = __ldg(p.perm + (int64_t)tile_of(p, index) * kTileRows + row_in_tile);
      const bool empty_tile = mask == 0;  // bias (+ residual) only, no accumulator involved
      const bool row_ok = row >= 0 && row < p.m_max;
      unsigned short* out_row = reinterpret_cast<unsigned short*>(p.out) + row * p.cout;
      const uint4* res_row = reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(p.residual) + row * p.cout);
      const uint32_t taddr = lane_base + (uint32_t)(acc * p.cout);
      constexpr int kAccs = kSplit ? kMma : 1;  // accumulators of a tile
      int first = 0;                            // the first of them that has a product
      while (kSplit && first + 1 < kAccs && (mask & offsets_of<kOffs, kMma>(first)) == 0u) ++first;
      auto columns = [&](auto with_residual) {
        constexpr bool kAdd = decltype(with_residual)::value;
        uint4 res[2];  // of the next 16 columns, on their way
        if (kAdd && row_ok && from < to) res[0] = __ldg(res_row + from / 8), res[1] = __ldg(res_row + from / 8 + 1);
        if (!empty_tile) {
#pragma unroll
          for (int m = 0; m < kAccs; ++m)
            if (!__all_sync(0xffffffffu, mbar_wait(&sh->acc_full[acc + m], acc_phase, abort_flag, 31, p.wait_limit))) return false;
          tc_fence_after();
        }
        for (int c0 = from; c0 < to; c0 += 16) {
          uint32_t v[16];
          if (empty_tile) {
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] = 0u;
          } else {
            tmem_ld16(taddr + first * p.cout + c0, v);
          }
          const uint4 now[2] = {res[0], res[1]};
          if (kAdd && row_ok && c0 + 16 < to) res[0] = __ldg(res_row + c0 / 8 + 2), res[1] = __ldg(res_row + c0 / 8 + 3);
          if (!empty_tile) tmem_ld_wait(v);
          if (kSplit) {  // the other warps' sums, in the order of the warps
#pragma unroll
            for (int m = 1; m < kAccs; ++m) {
              if (m <= first || (mask & offsets_of<kOffs, kMma>(m)) == 0u) continue;
              uint32_t w[16];
              tmem_ld16(taddr + m * p.cout + c0, w);
              tmem_ld_wait(w);
#pragma unroll
              for (int q = 0; q < 16; ++q) v[q] = __float_as_uint(__uint_as_float(v[q]) + __uint_as_float(w[q]));
            }
          }
          if (row_ok) {
            if (p.is_bf16) store_chunk<true, kAdd>(v, s.bias + c0, out_row + c0, now, p.relu, wide);
            else store_chunk<false, kAdd>(v, s.bias + c0, out_row + c0, now, p.relu, wide);
          }
        }
        return true;
      };
      if (!(p.residual ? columns(std::true_type{}) : columns(std::false_type{}))) return;
      if (!empty_tile) {
        if (!kWide && p.masked) {
          for (int m = 0; m < kAccs; ++m)
            for (int c0 = from; c0 < to; c0 += 16) tmem_zero16(taddr + m * p.cout + c0);
          tmem_st_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane < kAccs) mbar_arrive(&sh->acc_empty[acc + lane]);
        if ((acc += kAccs) == p.num_acc) acc = 0, acc_phase ^= 1;
      }
    }
  }
}

template <int kOffs, bool kWide, int kMma, bool kSplit>
__global__ void __launch_bounds__(threads_of(kMma), 1)
spconv_mm_tc_kernel(const __grid_constant__ CUtensorMap map_b, const TcParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  constexpr int kEpilogue = 4 * epilogue_sets(kMma);
  const Smem s = carve_smem<kOffs>(smem_raw, p);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tmem_base = cta_setup<kWide, kMma, kSplit>(p, s);
  pdl_release();
  if (warp < 8 * kMma) {
    producer_role<kOffs, kWide, kMma, kSplit>(p, s, tmem_base, warp, lane);
  } else if (warp < 8 * kMma + kEpilogue) {
    epilogue_role<kOffs, kWide, kMma, kSplit>(p, s, tmem_base, warp & 3, (warp - 8 * kMma) / 4);
  } else if (warp < 9 * kMma + kEpilogue) {
    mma_role<kOffs, kWide, kMma, kSplit>(p, s, &map_b, tmem_base, warp - 8 * kMma - kEpilogue);
  } else {
    control_role<kOffs, kWide, kMma, kSplit>(p, s, &map_b);
  }
  __syncwarp();
  cta_teardown<kMma>(s, tmem_base);
}

// ---- host ------------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<EncodeTiledFn>(ptr);
    return static_cast<EncodeTiledFn>(nullptr);
  }();  // initialised once, thread-safe
  return fn;
}

// 2-D map over a row-major 16-bit matrix [rows][cols]; the box is box_rows x box_cols, swizzled by its width.
bool make_map(CUtensorMap* map, int dtype, const void* base, uint64_t cols, uint64_t rows, uint32_t box_cols,
              uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * 2};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t elem[2] = {1, 1};
  const CUtensorMapSwizzle swz = box_cols * 2 == 32   ? CU_TENSOR_MAP_SWIZZLE_32B
                                 : box_cols * 2 == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                      : CU_TENSOR_MAP_SWIZZLE_128B;
  return fn(map, dtype == D3D_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
            const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct TcState {
  CUtensorMap map_b;
  bool map_b_ok = false;
};

// Tuning override for experiments (0 = automatic).
int g_plan_mma_warps = 0;
uint32_t g_wait_limit = kWaitLimitCycles;  // d3d_debug_set_wait_limit

typedef void (*KernelFn)(const CUtensorMap, const TcParams);
struct KernelEntry {
  int offs, wide, mma_warps, split;
  KernelFn fn;
};
#define D3D_TC_K(O, V, M, S) {O, V, M, S, spconv_mm_tc_kernel<O, V, M, S>}
const KernelEntry kKernels[] = {
    D3D_TC_K(4, true, 2, false), D3D_TC_K(4, false, 2, false), D3D_TC_K(2, true, 2, false), D3D_TC_K(2, false, 2, false),
    D3D_TC_K(1, true, 2, false), D3D_TC_K(1, false, 2, false), D3D_TC_K(2, true, 3, false), D3D_TC_K(2, false, 3, false),
    D3D_TC_K(1, true, 3, false), D3D_TC_K(1, false, 3, false), D3D_TC_K(4, true, 2, true), D3D_TC_K(4, false, 2, true),
    D3D_TC_K(2, true, 2, true), D3D_TC_K(2, false, 2, true), D3D_TC_K(1, true, 2, true), D3D_TC_K(1, false, 2, true),
};
#undef D3D_TC_K
constexpr int kNumKernels = sizeof(kKernels) / sizeof(kKernels[0]);

const KernelEntry* find_kernel(int offs, int wide, int mma_warps, int split) {
  for (int i = 0; i < kNumKernels; ++i)
    if (kKernels[i].offs == offs && kKernels[i].wide == wide && kKernels[i].mma_warps == mma_warps && kKernels[i].split == split)
      return &kKernels[i];
  return nullptr;
}

}  // namespace

bool spconv_mm_tc_eligible(const d3d_spconv_mm_s* h, int dtype) {
  if (dtype != D3D_HALF && dtype != D3D_BF16) return false;
  const int cin = h->p.in_channels, cout = h->p.out_channels, kvol = h->p.kernel_vol;
  if (!(cin == 16 || cin == 32 || cin == 64 || cin == 128 || cin == 256)) return false;
  if (cout % 16 != 0 || cout < 16 || cout > 256) return false;
  if (kvol > 32) return false;
  return encode_fn() != nullptr;
}

// The channel at position `pos` of a weight row in the order the kernel multiplies in.
int spconv_mm_tc_channel(int cin, int pos) {
  const int width = cin < 64 ? cin : 64;  // channels of a unit's row
  const int in = pos % width;
  if (rows_per_lane(64 / width) == 4)  // four lanes of 16 channels each; a store puts two words of each side by side
    return pos - in + in / 4 % 4 * 16 + in / 16 * 4 + in % 4;
  const int run = width / 2, word = in / 4, half = in / 2 % 2;  // two lanes of half the channels each, word by word
  return pos - in + half * run + word * 2 + in % 2;
}

void spconv_mm_tc_release(d3d_spconv_mm_s* h) {
  delete reinterpret_cast<TcState*>(h->tc_state);
  h->tc_state = nullptr;
}

// Creates the per-handle state of the tensor-core path (the tensor map over the transposed weights).  Called from
// d3d_spconv_mm_configure, so that an enqueue neither allocates nor encodes.
int spconv_mm_tc_prepare(d3d_spconv_mm_s* h, int dtype) {
  if (!spconv_mm_tc_eligible(h, dtype)) return D3D_OK;
  const int cin = h->p.in_channels, cout = h->p.out_channels, kvol = h->p.kernel_vol;
  TcState* st = new (std::nothrow) TcState();
  D3D_REQUIRE(st, D3D_ERR_INVALID_ARGUMENT);
  const uint32_t box_cols = cin < 64 ? cin : 64;
  st->map_b_ok = make_map(&st->map_b, dtype, h->wt_dev, cin, (uint64_t)kvol * cout, box_cols, cout);
  h->tc_state = st;
  return st->map_b_ok ? D3D_OK : D3D_ERR_CUDA;
}

int launch_spconv_mm_tc(const MmLaunch& a) {
  d3d_spconv_mm_s* h = const_cast<d3d_spconv_mm_s*>(a.h);
  const int cin = h->p.in_channels, cout = h->p.out_channels, kvol = h->p.kernel_vol;
  const int64_t m_max = h->p.max_num_act_out;
  if (m_max == 0) return D3D_OK;
  D3D_REQUIRE(a.max_num_act_in >= 1 && a.max_num_act_in < (1ll << 31), D3D_ERR_INVALID_ARGUMENT);
  D3D_REQUIRE(reinterpret_cast<uintptr_t>(a.in_feats) % 16 == 0 && reinterpret_cast<uintptr_t>(a.out_feats) % 16 == 0,
              D3D_ERR_INVALID_ARGUMENT);
  D3D_REQUIRE(!a.residual || reinterpret_cast<uintptr_t>(a.residual) % 16 == 0, D3D_ERR_INVALID_ARGUMENT);
  TcState* st = reinterpret_cast<TcState*>(h->tc_state);
  D3D_REQUIRE(st && st->map_b_ok, D3D_ERR_INVALID_ARGUMENT);  // configure() creates it

  TcParams p;
  const TableParts t = table_parts(const_cast<int32_t*>(a.table), kvol, m_max);
  p.table = t.ids, p.tile_mask = t.tile_mask, p.row_masks = t.row_masks, p.perm = t.perm;
  p.in_feats = a.in_feats;
  p.m_max = m_max;
  p.n_in_rows = (int32_t)a.max_num_act_in;
  p.kvol = kvol, p.cin = cin, p.cout = cout;
  p.num_tiles = (int)t.tiles;
  const int width = cin < 64 ? cin : 64, offs = 64 / width;
  p.parts = cin / width;
  p.row_bytes = width * 2;
  p.layout_type = p.row_bytes == 32 ? 6u : p.row_bytes == 64 ? 4u : 2u;
  const uint32_t fmt = a.dtype == D3D_BF16 ? 1u : 0u;
  p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(cout >> 3) << 17) | ((uint32_t)(kTileRows >> 4) << 24);
  p.regrouped = a.regrouped ? 1 : 0;
  // the other kernels: features that only start on 16 bytes (rows of 32 bytes are loaded 16 at a time anyway), a table that
  // only starts on four, weights that are not finite (a row without an input is zeros here, and 0 * W has to be 0)
  p.table_wide = reinterpret_cast<uintptr_t>(a.table) % 16 == 0;
  p.masked = !h->finite;
  const bool wide = (offs == 4 || reinterpret_cast<uintptr_t>(a.in_feats) % 32 == 0) && p.table_wide && !p.masked;
  p.weights = h->wt_dev;
  p.bias = h->b_dev;
  p.out = a.out_feats;
  p.residual = a.residual;
  p.relu = a.relu;
  p.is_bf16 = a.dtype == D3D_BF16;
  p.wait_limit = g_wait_limit;

  // Three MMA warps where a unit's products are short (up to 64 columns: 24 producer warps then feed them) and a CTA has more than
  // two tiles, two where the tensor pipe is the longer part, where few offsets make the epilogue it (it has eight warps then) and for 16 input channels, whose
  // units take the most instructions.  us with two / three: 27 offsets 32 -> 32 83 / 72, 64 -> 64 77 / 69, 128 -> 64 61 / 58,
  // 64 -> 128 94 / 113, 128 -> 128 50 / 55, 256 -> 256 116 / 120, 16 -> 32 31 / 34; nine offsets 32 -> 32 15.8 / 17.2; three
  // offsets 64 -> 64 15.3 / 18.2.
  // One tile to a CTA: two MMA warps share it, since a chain of products is what such a launch lasts (an MMA warp takes 470 cycles
  // from one unit to the next, whatever feeds it).  From the second tile on a tile each is faster: they share their weights (157
  // tiles of 64 -> 64: 14.7 us, shared one after the other 17.8).
  //   Two tiles of a CTA lie a grid apart: that is balanced wherever the live tiles end, so that these need not be looked for, which
  // costs two trips to L2 in front of the first list (219 live of 256 tiles, 16 -> 32 9.7 / 8.6 us; the CTAs that start first have
  // two: the other way round 64 -> 64 behind another launch 13.1 / 13.8).
  const bool is_short = p.num_tiles <= 2 * kNumSMs, split = p.num_tiles <= kNumSMs && cout <= 192 && kvol > offs;
  const int mma_warps = cin < 32 || split        ? 2
                        : g_plan_mma_warps       ? g_plan_mma_warps
                        : cout <= 64 && kvol > 9 ? (is_short ? 2 : 3)
                                                 : 2;
  p.spread = p.regrouped || is_short;
  const KernelEntry* k = find_kernel(offs, wide, mma_warps, split);
  D3D_REQUIRE(k, D3D_ERR_INVALID_ARGUMENT);
  // tensor memory: a slot for every producer team, the rest accumulators
  p.ring_col = kTmemCols - 2 * mma_warps * kUnitCols;
  p.num_acc = p.ring_col / cout;
  if (p.num_acc > kMaxAcc) p.num_acc = kMaxAcc;
  if (split) p.num_acc -= p.num_acc % mma_warps;
  // shared memory: weights
  p.b_bytes = (uint32_t)align_up((size_t)cout * p.row_bytes, (size_t)8 * p.row_bytes);
  const size_t ctrl = 1024 + align_up((size_t)cout * 4 + 16, 16) + sizeof(Shared);
  size_t weights = align_up(kvol, offs) * p.b_bytes;
  p.b_slots = 0;
  // in shared memory for good up to 112 KB, which leaves L1 as much (16 -> 16 to 32 -> 64, held or streamed: the same to 1 %)
  // but not where a CTA has two tiles: the first products need not wait for all (219 tiles of 32 -> 64: 13.1 us held, 12.7 streamed;
  // with one tile the load in front of a chained launch is worth more: 6.0 held, 6.9 streamed)
  if (p.parts > 1 || weights > (is_short && !split ? 56 : 112) * 1024) {
    const size_t window = (size_t)2 * offs * p.b_bytes;  // two of them to a slot
    p.b_slots = (int)(128 * 1024 / window);
    if (p.b_slots < 3) p.b_slots = 3;
    if (p.b_slots > kMaxBSlots) p.b_slots = kMaxBSlots;
    if (split) p.b_slots = p.b_slots < 2 * mma_warps ? 2 * mma_warps : p.b_slots - p.b_slots % mma_warps;
    weights = p.b_slots * window;
  }
  const size_t smem = ctrl + weights;
  D3D_REQUIRE(smem <= 227 * 1024, D3D_ERR_TOO_LARGE);
  {
    // raising the dynamic shared memory limit is per function and per device; once each, under a lock
    static std::mutex attr_lock;
    static bool attr_set[64][kNumKernels] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return D3D_ERR_CUDA;
    const int ki = (int)(k - kKernels);
    std::lock_guard<std::mutex> guard(attr_lock);
    if (!attr_set[dev][ki]) {
      if (cudaFuncSetAttribute(k->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess)
        return D3D_ERR_CUDA;
      attr_set[dev][ki] = true;
    }
  }
  const int grid = p.num_tiles < kNumSMs ? p.num_tiles : kNumSMs;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid), cfg.blockDim = dim3(threads_of(mma_warps));
  cfg.dynamicSmemBytes = smem, cfg.stream = reinterpret_cast<cudaStream_t>(a.stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = a.chained ? 1 : 0;
  if (cudaLaunchKernelEx(&cfg, k->fn, st->map_b, p) != cudaSuccess) return D3D_ERR_CUDA;
  D3D_CHECK_LAUNCH();
  return D3D_OK;
}

}  // namespace d3d

// Debug aid without a reference counterpart (the reference prints CUDA errors, trt/include/common/macros.h:14-34):
// synchronises the device and returns the error word the tensor-core kernel raises when one of its bounded waits
// expires (0 = none), clearing it.
extern "C" int d3d_debug_take_kernel_error(int* code) {
  if (!code) return D3D_ERR_INVALID_ARGUMENT;
  int zero = 0;
  if (cudaDeviceSynchronize() != cudaSuccess) return D3D_ERR_CUDA;
  if (cudaMemcpyFromSymbol(code, d3d::g_tc_error, sizeof(int)) != cudaSuccess) return D3D_ERR_CUDA;
  if (cudaMemcpyToSymbol(d3d::g_tc_error, &zero, sizeof(int)) != cudaSuccess) return D3D_ERR_CUDA;
  return D3D_OK;
}

// Debug aid without a reference counterpart: after how many cycles a bounded wait of the tensor-core kernel gives up, for every
// later launch of this process (0 = the usual second).  Not thread-safe.
extern "C" int d3d_debug_set_wait_limit(int cycles) {
  D3D_REQUIRE(cycles >= 0, D3D_ERR_INVALID_ARGUMENT);
  d3d::g_wait_limit = cycles ? (uint32_t)cycles : d3d::kWaitLimitCycles;
  return D3D_OK;
}

// Tuning aid without a reference counterpart: overrides the plan of the tensor-core kernel for every later launch of
// this process.  16 or 24 producer warps (two or three MMA warps), 0 = automatic; offsets per stage and stages belong to an
// earlier kernel and have no effect.  Not thread-safe.
extern "C" int d3d_debug_set_tc_plan(int group, int max_stages, int prod_warps) {
  if (group < 0 || group > 8 || max_stages < 0 || max_stages > 8 ||
      !(prod_warps == 0 || prod_warps == 4 || prod_warps == 8 || prod_warps == 16 || prod_warps == 24))
    return D3D_ERR_INVALID_ARGUMENT;
  d3d::g_plan_mma_warps = prod_warps >= 16 ? prod_warps / 8 : 0;
  return D3D_OK;
}
