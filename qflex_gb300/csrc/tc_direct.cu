// The split-precision products that split A themselves (sm_103a, tcgen05 +
// TMEM + TMA).
//
// C = A * B, A complex64 in global memory, B as planes of Bt (n x k, K-major,
// see split.cu). A is brought in as it lies -- row-major, or through the index
// permutation that would have laid it out so (AGather) -- and split into its
// planes inside the kernel. Against a split kernel (or a plane-writing
// permutation) before the product that saves one pass over A: 8 B read and 8
// (3xFP16), 12 (BF16x3) or 16 (3xTF32) written per element.
//
// Structure: persistent, one CTA per SM over tiles of 128 rows x BN (128, 64
// or 32) columns, 512 threads in four warpgroups whose registers setmaxnreg
// divides (56, 176, 176, 104 per thread: 128 on average, the launch's own
// share). Work goes by blocks of A, 128 rows x two k-steps: 32 values, or in
// 3xTF32, whose k-steps are of 8, 16, half a place of A's ring.
//   warp 0       B producer: four 8 KB TMA boxes a block (re and im rows of
//                64 bytes, hi and lo, of each k-step)
//   warp 1       TMEM allocation; issues every MMA
//   warp 2       A loader: TMA boxes into a ring of blocks (with warp 3,
//                16- or 8-byte cp.async copies where no box fits)
//   warps 4..11  epilogue: drains TMEM sums, scales and stores the tile
//   warps 12..15 A converter: thread r reads row r of the block, finds the
//                largest component, scales by the power of two that brings it
//                into [2^14, 2^15), splits into hi + lo and writes the planes
//                to its TMEM lane, where the MMAs read A
// TMEM holds two blocks of planes (128 columns) and three sums of BN columns:
// a block's real part is summed from zero into one, its imaginary part into
// the next, and the epilogue, which applies the block's exponent as it adds a
// sum to the tile, drains one while the others fill.
//
// PAIR (clusters of two CTAs, cta_group::2): CTA r has rows 128 r .. + 127 of a
// tile of 256, their planes in its own tensor memory, and half of B's columns
// in its shared memory; CTA 0 issues MMAs of M = 256 for both. B's stages and
// the MMAs' reads of them halve. CTA 0's barriers take both CTAs' arrivals
// (planes written, sums drained) and B's bytes; commits go to both CTAs.
//
// What bounds it: a block's 24 MMAs take 1536 cycles of the tensor pipe, and
// one warp issues them, one converts per SM partition, so what these do
// between MMAs counts as much; next shared memory, of which the MMAs read 64
// bytes a cycle (a pair's 32). Measured at k = 4096 (1024 x 1024, 64 CTAs: no
// power limit), cycles a block: A's planes in shared memory, A by cp.async
// and five waits and commits a block 2360; planes in TMEM the same; two waits
// and commits 2030; A by TMA boxes 1950; pairs 1640. At (4096, 4096, 4096),
// 901 us, the card's power limit is reached. (65536, 256, 256) x 4 went from
// 341 to 286 us, of which each tile's store, 5600 cycles, leaves the tensor
// pipe idle for 3300; (4096, 1024, 4096) from 319 to 240; (65536, 256, 16) x
// 4 takes 96, of which writing C alone is 80.
//
// The other kinds scale nothing. 3xTF32: (2048, 2048, 2048) 18 + 256 + 22 us
// with both operands split before the product, 216 + 17; (65536, 256, 256) x 4
// 228 + 495 and 436. BF16x3, six planes of A (192 TMEM columns and two sums),
// 48 MMAs a block: (4096, 1024, 2048) 28 + 279 and 217 us, (65536, 256, 256) x
// 4 193 + 485 and 427.
//
// B holds no negated copy: the real part takes -Ai Bi by the descriptor's
// negate-A bit, and a k-step loads 16 KB of B, not 24. MMAs of N = 128 run at
// the rate of N = 256 when A lies in TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "half_split.cuh"
#include "per_device.h"
#include "tc_common.cuh"
#include "tc_gemm.h"

namespace qfx {
namespace {

constexpr int BM = 128;
constexpr int A_BLOCK = 128 * 32 * 8;  // bytes of A as it lies, 32 values of a row
constexpr int A_BUFS = 2;              // blocks of planes in TMEM
constexpr int EXP_RING = 4;            // block exponents, see the converter
constexpr int SLOT = 4096;             // output box: 32 rows x 16 complex
template <int KIND>
__host__ __device__ constexpr int block_values() {  // values of a row in two k-steps
  return KIND == KIND_TF32 ? 16 : 32;
}
constexpr int THREADS = 512;
constexpr int LOADERS = 64, CONVERTERS = 128;

// Shared memory and TMEM for tiles of 128 rows and BN columns; of a PAIR, with
// half of B's columns.
template <int KIND, int BN, bool PAIR>
struct Layout {
  static constexpr int PLANES = KIND == KIND_BF16 ? 6 : 4;   // of A
  static constexpr int HALVES = KIND == KIND_BF16 ? 2 : 3;  // sums, the real or imaginary part of a block
  static constexpr int TMEM_A_BLOCK = 2 * PLANES * 8;       // 2 k-steps x planes x 8 words
  static constexpr int A_RING = BN == 128 ? 3 : BN == 64 ? 4 : 5;  // blocks of 128 rows x 32 values
  static constexpr int B_COLS = PAIR ? BN / 2 : BN;
  static constexpr int B_PART = B_COLS * 64;               // re or im rows of a k-step (hi, lo)
  static constexpr int B_STEP = B_COLS * PLANES * 32;      // re, im rows, BF16x3: re, im rows of the third pieces
  static constexpr int B_STAGES = PAIR && KIND != KIND_BF16 ? 4 : 2;  // two k-steps each
  static constexpr int DONE = PAIR ? 4 : 3;      // barriers of finished blocks in turn
  static_assert(DONE >= B_STAGES && DONE > A_BUFS, "a barrier's phase is read before the next but one");
  static constexpr int B_STAGE = 2 * B_STEP;
  static constexpr int SLOTS = BN == 32 ? 1 : 2;  // of each epilogue warp
  static constexpr int COLS = BN / 2;             // columns of an epilogue warp
  static constexpr int OFF_B = A_RING * A_BLOCK;
  static constexpr int OFF_STAGING = OFF_B + B_STAGES * B_STAGE;
  static constexpr int OFF_SCALE = OFF_STAGING + 8 * SLOTS * SLOT;
  static constexpr int OFF_EXP = OFF_SCALE + 8 * COLS * 4;  // after each epilogue warp's column exponents
  static constexpr int OFF_BAR = OFF_EXP + EXP_RING * BM;
  static constexpr int EXP_BARS = KIND == KIND_FP16 ? EXP_RING : 0;
  static constexpr int N_BARS = 2 * A_RING + A_BUFS + B_STAGES + 2 * DONE + HALVES + 1 + 2 * EXP_BARS;
  static constexpr int SMEM = OFF_BAR + N_BARS * 8 + 24;  // and tmem_slot .. peer_abort
  static_assert(SMEM <= 227 * 1024, "one CTA's shared memory");
  static constexpr int TMEM_A = HALVES * BN;  // the planes, after the sums
  static constexpr int TMEM_COLS = BN == 32 ? 256 : 512;
  static_assert(TMEM_A + A_BUFS * TMEM_A_BLOCK <= TMEM_COLS, "TMEM");
};

// The real (IM = 0) or imaginary part of a block: two k-steps of A's planes in
// TMEM (re hi, lo, im hi, lo, 8 columns each from `a`) against B's re rows
// (`blo`, hi and lo 32 bytes apart) and im rows (B_PART further), small terms
// first.
template <int KIND, int BN, bool PAIR, int IM>
__device__ __forceinline__ void mma_block(std::uint32_t d, std::uint32_t a, std::uint32_t blo, std::uint32_t bhi) {
  constexpr int rows = PAIR ? 2 * BM : BM;
  constexpr std::uint32_t pos = KIND == KIND_TF32 ? idesc_tf32(rows, BN, false) : idesc_f16(rows, BN, false);
  constexpr std::uint32_t neg = KIND == KIND_TF32 ? idesc_tf32(rows, BN, true) : idesc_f16(rows, BN, true);
  constexpr std::uint32_t part = Layout<KIND, BN, PAIR>::B_PART / 16;
  // Ar multiplies B's part of the same name, Ai the other one (negated for
  // the real part).
  const std::uint32_t x = IM ? blo + part : blo, y = IM ? blo : blo + part;
#define QFX_MMA(g, a_, b_, id, p) " tcgen05.mma.cta_group::" g " [%0], [" a_ "], " b_ ", " id ", " p ";\n"
#define QFX_KSTEP(g, rh, rl, ih, il, p)                                                                  \
  QFX_MMA(g, rh, "xl", "%5", p)                                                                          \
  QFX_MMA(g, rl, "xh", "%5", "p1")                                                                       \
  QFX_MMA(g, ih, "yl", "%6", "p1")                                                                       \
  QFX_MMA(g, il, "yh", "%6", "p1") QFX_MMA(g, rh, "xh", "%5", "p1") QFX_MMA(g, ih, "yh", "%6", "p1")
#define QFX_BDESC " mov.b64 xh, {x0, %4};\n mov.b64 xl, {x1, %4};\n mov.b64 yh, {y0, %4};\n mov.b64 yl, {y1, %4};\n"
#define QFX_BLOCK(g) \
    asm volatile( \
        "{\n .reg .pred p0, p1;\n .reg .b32 a1, a2, a3, a4, a5, a6, a7, x0, x1, y0, y1;\n" \
        " .reg .b64 xh, xl, yh, yl;\n" \
        " setp.ne.b32 p0, %1, %1;\n setp.eq.b32 p1, %1, %1;\n" \
        " add.u32 a1, %1, 8;\n add.u32 a2, %1, 16;\n add.u32 a3, %1, 24;\n add.u32 a4, %1, 32;\n" \
        " add.u32 a5, %1, 40;\n add.u32 a6, %1, 48;\n add.u32 a7, %1, 56;\n" \
        " mov.b32 x0, %2;\n mov.b32 y0, %3;\n add.u32 x1, %2, 2;\n add.u32 y1, %3, 2;\n" \
        QFX_BDESC QFX_KSTEP(g, "%1", "a1", "a2", "a3", "p0") \
        " add.u32 x0, %2, %7;\n add.u32 y0, %3, %7;\n add.u32 x1, x0, 2;\n add.u32 y1, y0, 2;\n" \
        QFX_BDESC QFX_KSTEP(g, "a4", "a5", "a6", "a7", "p1") "}\n" ::"r"(d), \
        "r"(a), "r"(x), "r"(y), "r"(bhi), "r"(pos), "r"(IM ? pos : neg), "n"(2 * part))
  if constexpr (PAIR && KIND == KIND_TF32)
    QFX_BLOCK("2.kind::tf32");
  else if constexpr (PAIR)
    QFX_BLOCK("2.kind::f16");
  else if constexpr (KIND == KIND_TF32)
    QFX_BLOCK("1.kind::tf32");
  else
    QFX_BLOCK("1.kind::f16");
#undef QFX_BLOCK
#undef QFX_BDESC
#undef QFX_KSTEP
#undef QFX_MMA
}

// The same of BF16x3, one k-step: planes re 0, 1, 2, im 0, 1, 2 in TMEM; B's re
// rows (`blo`) and im rows with pieces 0 and 1 32 bytes apart, then those of
// piece 2, 32 bytes each. Per real product x y the terms x2 y0, x1 y1, x0 y2
// (~2^-16), x1 y0, x0 y1 (~2^-8) and x0 y0, smallest first. Pairs only.
template <int B_COLS, int BN, int IM>
__device__ __forceinline__ void mma_bf16_step(std::uint32_t d, std::uint32_t a, std::uint32_t blo, std::uint32_t bhi,
                                              std::uint32_t bhi2, std::uint32_t acc) {
  constexpr std::uint32_t pos = idesc_bf16(2 * BM, BN, false), neg = idesc_bf16(2 * BM, BN, true);
  constexpr std::uint32_t part = B_COLS * 64 / 16, part2 = B_COLS * 32 / 16;
  const std::uint32_t x = IM ? blo + part : blo, y = IM ? blo : blo + part;
  const std::uint32_t t = blo + 2 * part, x2 = IM ? t + part2 : t, y2 = IM ? t : t + part2;
#define QFX_MMA(a_, b_, id, p) " tcgen05.mma.cta_group::2.kind::f16 [%0], [" a_ "], " b_ ", " id ", " p ";\n"
  asm volatile(
      "{\n .reg .pred p0, p1;\n .reg .b32 r1, r2, i0, i1, i2, x1, y1;\n .reg .b64 x0d, x1d, x2d, y0d, y1d, y2d;\n"
      " setp.ne.b32 p0, %8, 0;\n setp.eq.b32 p1, %8, %8;\n"
      " add.u32 r1, %1, 8;\n add.u32 r2, %1, 16;\n add.u32 i0, %1, 24;\n add.u32 i1, %1, 32;\n add.u32 i2, %1, 40;\n"
      " add.u32 x1, %2, 2;\n add.u32 y1, %3, 2;\n mov.b64 x0d, {%2, %6};\n mov.b64 x1d, {x1, %6};\n"
      " mov.b64 y0d, {%3, %6};\n mov.b64 y1d, {y1, %6};\n mov.b64 x2d, {%4, %7};\n mov.b64 y2d, {%5, %7};\n"  //
      QFX_MMA("r2", "x0d", "%9", "p0") QFX_MMA("r1", "x1d", "%9", "p1") QFX_MMA("%1", "x2d", "%9", "p1")
      QFX_MMA("i2", "y0d", "%10", "p1") QFX_MMA("i1", "y1d", "%10", "p1") QFX_MMA("i0", "y2d", "%10", "p1")
      QFX_MMA("r1", "x0d", "%9", "p1") QFX_MMA("%1", "x1d", "%9", "p1") QFX_MMA("i1", "y0d", "%10", "p1")
      QFX_MMA("i0", "y1d", "%10", "p1") QFX_MMA("%1", "x0d", "%9", "p1") QFX_MMA("i0", "y0d", "%10", "p1") "}\n" ::"r"(d),
      "r"(a), "r"(x), "r"(y), "r"(x2), "r"(y2), "r"(bhi), "r"(bhi2), "r"(acc), "r"(pos), "r"(IM ? pos : neg));
#undef QFX_MMA
}

// 32 words of the thread's TMEM lane.
__device__ __forceinline__ void tmem_st32(std::uint32_t at, const std::uint32_t* w) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(at),
      "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]),
      "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15]), "r"(w[16]), "r"(w[17]), "r"(w[18]),
      "r"(w[19]), "r"(w[20]), "r"(w[21]), "r"(w[22]), "r"(w[23]), "r"(w[24]), "r"(w[25]), "r"(w[26]), "r"(w[27]),
      "r"(w[28]), "r"(w[29]), "r"(w[30]), "r"(w[31])
      : "memory");
}

// 16 words.
__device__ __forceinline__ void tmem_st16(std::uint32_t at, const std::uint32_t* w) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16};" ::"r"(at),
      "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]),
      "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15])
      : "memory");
}

// Two-lane FP32 arithmetic (round to nearest, each lane as the scalar form).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n .reg .b64 x, y, z, w;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n mov.b64 z, {%6, %7};\n"
      " fma.rn.f32x2 w, x, y, z;\n mov.b64 {%0, %1}, w;\n}\n"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n .reg .b64 x, y, w;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n"
      " mul.rn.f32x2 w, x, y;\n mov.b64 {%0, %1}, w;\n}\n"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
// 2^e as a float, 0 below the normal range (e <= 127).
__device__ __forceinline__ float pow2(int e) {
  return __uint_as_float(e >= -126 ? std::uint32_t(e + 127) << 23 : 0u);
}

__device__ __forceinline__ void cp_async16(std::uint32_t dst, const void* src, std::uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async8(std::uint32_t dst, const void* src, std::uint32_t bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(std::uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

#define QFX_SETMAXNREG_DEC(n) asm volatile("setmaxnreg.dec.sync.aligned.u32 " #n ";")
#define QFX_SETMAXNREG_INC(n) asm volatile("setmaxnreg.inc.sync.aligned.u32 " #n ";")

template <int KIND, int BN, bool PAIR>
__global__ void __launch_bounds__(THREADS, 1)
    cgemm_direct_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                               const __grid_constant__ CUtensorMap map_b2,
                               const __grid_constant__ CUtensorMap map_c, const __grid_constant__ AGather g,
                               const float2* __restrict__ A, float2* __restrict__ C, int tma_c, int m, int n, int k,
                               int batches, std::uint64_t ac_stride, int* __restrict__ err,
                               const int* __restrict__ exp_b, int watch) {
  using L = Layout<KIND, BN, PAIR>;
  constexpr int B_STAGES = L::B_STAGES, DONE = L::DONE, HALVES = L::HALVES, TMEM_A_BLOCK = L::TMEM_A_BLOCK;
  constexpr int A_RING = L::A_RING, B_PART = L::B_PART, B_STAGE = L::B_STAGE, TMEM_A = L::TMEM_A, COLS = L::COLS;
  extern __shared__ __align__(1024) std::uint8_t smem[];
  std::uint64_t* raw_full = reinterpret_cast<std::uint64_t*>(smem + L::OFF_BAR);  // a block of A has landed
  std::uint64_t* raw_empty = raw_full + A_RING;                                // and is in registers
  std::uint64_t* a_full = raw_empty + A_RING;                                  // its planes are in TMEM
  std::uint64_t* b_full = a_full + A_BUFS;
  std::uint64_t* re_full = b_full + B_STAGES;   // a block's real part is summed
  std::uint64_t* done = re_full + DONE;         // all MMAs of a block are done
  std::uint64_t* acc_empty = done + DONE;       // an accumulator was drained
  std::uint64_t* mma_done = acc_empty + HALVES;
  std::uint64_t* exp_full = mma_done + 1;             // a block's exponents are written
  std::uint64_t* exp_empty = exp_full + L::EXP_BARS;  // and read by the epilogue
  std::uint32_t* tmem_slot = reinterpret_cast<std::uint32_t*>(exp_empty + L::EXP_BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // What lands if the pipeline is abandoned: blocks of A by boxes and stages of
  // B asked for, in a pair those of B by CTA 1; whether the other CTA gave up.
  volatile int* issued_a = abort_flag + 1;
  volatile int* issued_b = issued_a + 1;
  volatile int* peer_b = issued_b + 1;
  volatile int* peer_abort = peer_b + 1;
  if (smem_u32(smem) & 1023) {  // the swizzles need it; the layout leaves no room to round up
    if (threadIdx.x == 0) atomicExch(err, 9);
    return;
  }

  // Uniform for the compiler: see the MMA issuer.
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x / 32, 0), lane = threadIdx.x % 32;
  const std::uint32_t rank = PAIR ? cluster_rank() : 0;
  const int first = PAIR ? blockIdx.x / 2 : blockIdx.x, stride = PAIR ? gridDim.x / 2 : gridDim.x;
  constexpr int TILE_M = PAIR ? 2 * BM : BM, GROUP = PAIR ? 4 : 8;
  const int tiles_m = (m + TILE_M - 1) / TILE_M;
  const int tiles_n = (n + BN - 1) / BN;
  const int per_batch = tiles_m * tiles_n;
  const int total = per_batch * batches;
  // Tiles run in groups of 1024 rows so that the CTAs working at one time
  // share A rows and B columns in L2.
  auto tile_of = [&](int t, int& mt, int& nt, int& batch) {
    batch = t / per_batch;
    const int r = t % per_batch;
    const int per_group = GROUP * tiles_n;
    const int group = r / per_group, in_group = r % per_group;
    const int group_m = min(GROUP, tiles_m - group * GROUP);
    mt = group * GROUP + in_group % group_m;
    if (PAIR) mt = 2 * mt + int(rank);
    nt = in_group / group_m;
  };
  // Waits and arrivals keep CTA scope in a pair as well: what the barriers
  // between its CTAs order are tensor-memory accesses (with the tcgen05
  // fences) and TMA writes. At cluster scope a block took 3200 cycles. The
  // blocks' exponents, ordinary shared memory, have barriers of their own
  // inside the CTA (exp_full, exp_empty): neither an arrival at the other
  // CTA nor a commit orders them.
  auto wait = [&](std::uint64_t* bar, std::uint32_t parity, int code) {
    return mbar_wait(bar, parity, abort_flag, err, code);
  };
  // Arrival at, and MMA completion on, barriers that a pair's CTA 0 waits on
  // or that both wait on.
  auto arrive = [&](std::uint64_t* bar) {
    if constexpr (PAIR)
      asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(peer_addr(bar, 0)) : "memory");
    else
      mbar_arrive(bar);
  };
  auto commit = [&](std::uint64_t* bar) {
    if constexpr (PAIR)
      umma_commit_pair(bar);
    else
      umma_commit(bar);
  };
  constexpr int VALUES = block_values<KIND>();
  const int blocks = (k + VALUES - 1) / VALUES, loads = (k + 31) / 32;  // of a tile
  // Blocks of all the CTA's tiles.
  const int work = first < total ? ((total - 1 - first) / stride + 1) * blocks : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < A_RING; ++s) {
      mbar_init(&raw_full[s], g.boxes ? 1 : LOADERS);
      mbar_init(&raw_empty[s], CONVERTERS / 32);
    }
    for (int s = 0; s < A_BUFS; ++s) mbar_init(&a_full[s], (PAIR ? 2 : 1) * CONVERTERS / 32);
    for (int s = 0; s < B_STAGES; ++s) mbar_init(&b_full[s], 1);
    for (int s = 0; s < DONE; ++s) {
      mbar_init(&re_full[s], 1);
      mbar_init(&done[s], 1);
    }
    for (int s = 0; s < HALVES; ++s) mbar_init(&acc_empty[s], PAIR ? 16 : 8);
    mbar_init(mma_done, 1);
    for (int s = 0; s < L::EXP_BARS; ++s) {
      mbar_init(&exp_full[s], CONVERTERS / 32);
      mbar_init(&exp_empty[s], 8);
    }
    *abort_flag = 0;
    *issued_a = *issued_b = *peer_b = *peer_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // The second half of a block that a k of 16 does not have.
  if (g.boxes && !g.plain && g.copies_real < 32)
    for (int i = threadIdx.x; i < A_RING * A_BLOCK / 32; i += THREADS)
      *reinterpret_cast<float4*>(smem + i / (A_BLOCK / 32) * A_BLOCK + A_BLOCK / 2 + i % (A_BLOCK / 32) * 16) =
          make_float4(0.f, 0.f, 0.f, 0.f);
  if (warp == 1) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                   "r"(L::TMEM_COLS));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                   "r"(L::TMEM_COLS));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if constexpr (PAIR) cluster_sync();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const std::uint32_t tmem = *tmem_slot;

  if (warp < 4) {
    QFX_SETMAXNREG_DEC(56);
    if (warp == 0 && lane == 0) {
      // B producer.
      constexpr int X_IM = KIND == KIND_TF32 ? 16 : 32;  // im rows in the map
      int q = 0, s = 0;
      for (int t = first; t < total && !*abort_flag; t += stride) {
        int mt, nt, batch;
        tile_of(t, mt, nt, batch);
        for (int b = 0; b < blocks; ++b) {
          if (q >= B_STAGES) {
            const int free = q - B_STAGES;
            if (!wait(&done[free % DONE], (free / DONE) & 1, 1)) break;
          }
          // A k of an odd number of k-steps: the last one's rows lie outside
          // the map and arrive as zeros.
          std::uint8_t* st = smem + L::OFF_B + s * B_STAGE;
          const int col = nt * BN + int(rank) * L::B_COLS;
          if (rank == 0) mbar_expect_tx(&b_full[s], (PAIR ? 2 : 1) * B_STAGE);  // both CTAs' halves
          for (int h = 0; h < 2; ++h, st += L::B_STEP) {
            if constexpr (PAIR) {
              const std::uint32_t bar = peer_addr(&b_full[s], 0);
              tma_load_4d_pair(&map_b, bar, st, 0, col, 2 * b + h, batch);
              tma_load_4d_pair(&map_b, bar, st + B_PART, X_IM, col, 2 * b + h, batch);
              if constexpr (KIND == KIND_BF16) {
                tma_load_4d_pair(&map_b2, bar, st + 2 * B_PART, 0, col, 2 * b + h, batch);
                tma_load_4d_pair(&map_b2, bar, st + 2 * B_PART + B_PART / 2, 16, col, 2 * b + h, batch);
              }
            } else {
              tma_load_4d(&map_b, &b_full[s], st, 0, col, 2 * b + h, batch);
              tma_load_4d(&map_b, &b_full[s], st + B_PART, X_IM, col, 2 * b + h, batch);
            }
          }
          ++q;
          if (++s == B_STAGES) s = 0;
        }
      }
      *issued_b = q;
    } else if (warp == 1 && rank == 0) {
      // MMA issuer (of a pair: CTA 0). The whole warp runs the loop in step and one elected lane
      // issues: the descriptors then live in uniform registers. Run by one
      // lane alone, every descriptor word moved there before each MMA, and
      // beside the other warps' work a k-step took 980 cycles instead of 775
      // (768 at the tensor pipe's rate; measured with this k-step, its
      // commits and barrier tests, a TMEM drain and shared-memory traffic).
      // What the warp does between two MMAs counts as well: a block's MMAs
      // take 1536 cycles, and a loop with five waits, each by the whole warp,
      // and five commits a block took 2370. So a block waits twice, its lanes
      // testing different barriers, and commits twice.
      //
      // A block is summed from zero, first its real, then its imaginary part,
      // each into the next of the three TMEM buffers. Lane kinds: 0 and 3
      // wait for the buffers of the real and the imaginary part, 1 for A's
      // planes, 2 for B's.
      const bool leader = elect_one();
      const std::uint64_t db = smem_desc_sw64(smem_u32(smem + L::OFF_B));
      const std::uint32_t b_hi = std::uint32_t(db >> 32), b_lo0 = std::uint32_t(db);
      const std::uint32_t b_hi2 = std::uint32_t(smem_desc_sw32(0) >> 32);
      auto issue = [&](auto im, std::uint32_t d, std::uint32_t a, std::uint32_t b) {
        constexpr int IM = decltype(im)::value;
        if constexpr (KIND == KIND_BF16) {
          mma_bf16_step<L::B_COLS, BN, IM>(d, a, b, b_hi, b_hi2, 0);
          mma_bf16_step<L::B_COLS, BN, IM>(d, a + 48, b + (L::B_STEP >> 4), b_hi, b_hi2, 1);
        } else {
          mma_block<KIND, BN, PAIR, IM>(d, a, b, b_hi);
        }
      };
      const int kind = lane & 3;
      std::uint64_t* const bars = kind == 1 ? a_full : kind == 2 ? b_full : acc_empty;
      const int ring = kind == 1 ? A_BUFS : kind == 2 ? B_STAGES : HALVES;
      const int step = kind == 1 || kind == 2 ? 1 : 2;
      int at = kind == 3 ? 1 : 0;
      std::uint32_t parity = kind == 1 || kind == 2 ? 0u : 1u;  // a fresh buffer is empty
      int xa = 0, sb = 0, h = 0, r = 0;
      for (int w = 0; w < work; ++w) {
        if (!__all_sync(0xffffffffu, kind == 3 || wait(bars + at, parity, 2))) break;
        __syncwarp();  // what one lane's wait orders, it orders for the leader
        asm volatile("tcgen05.fence::after_thread_sync;");
        const std::uint32_t a = tmem + TMEM_A + xa * TMEM_A_BLOCK, b = b_lo0 + sb * (B_STAGE >> 4);
        if (leader) {
          issue(std::integral_constant<int, 0>{}, tmem + h * BN, a, b);
          commit(&re_full[r]);
        }
        h = h == HALVES - 1 ? 0 : h + 1;
        // The epilogue's TMEM reads of a buffer precede the MMAs that
        // overwrite it.
        if (!__all_sync(0xffffffffu, kind != 3 || wait(bars + at, parity, 4))) break;
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (leader) {
          issue(std::integral_constant<int, 1>{}, tmem + h * BN, a, b);
          commit(&done[r]);
        }
        h = h == HALVES - 1 ? 0 : h + 1;
        xa ^= 1;
        sb = sb == B_STAGES - 1 ? 0 : sb + 1;
        r = r == DONE - 1 ? 0 : r + 1;
        at += step;
        if (at >= ring) {
          at -= ring;
          parity ^= 1u;
        }
      }
      __syncwarp();
      if (leader) commit(mma_done);
      __syncwarp();
    } else if (warp >= 2 && g.boxes) {
      // A loader, by TMA boxes.
      if (warp == 2 && lane == 0) {
        const std::uint32_t ring = smem_u32(smem);
        const std::uint32_t bytes = g.copies_real == 32 ? A_BLOCK : A_BLOCK / 2;
        int q = 0, s = 0;
        std::uint32_t ph = 0;
        for (int t = first; t < total && !*abort_flag; t += stride) {
          int mt, nt, batch;
          tile_of(t, mt, nt, batch);
          std::uint64_t tile_src = std::uint64_t(batch) * ac_stride;
          if (!g.plain)
            for (int x = 0; x < AGather::kBits && (mt >> x); ++x)
              if ((mt >> x) & 1) tile_src += g.tile_src[x];
          for (int b = 0; b < loads; ++b) {
            if (q >= A_RING && !wait(&raw_empty[s], ph ^ 1u, 5)) break;
            const std::uint32_t dst = ring + s * A_BLOCK;
            mbar_expect_tx(&raw_full[s], bytes);
            if (g.plain) {
              tma_load_3d(&map_a, &raw_full[s], dst, b * 32, mt * BM, batch);
              tma_load_3d(&map_a, &raw_full[s], dst + A_BLOCK / 2, b * 32 + 16, mt * BM, batch);
            } else {
              std::uint64_t src = tile_src;
              for (int x = 0; x < AGather::kBits && (b >> x); ++x)
                if ((b >> x) & 1) src += g.block_src[x];
              tma_load_5d(&map_a, &raw_full[s], dst, int(src / 16));
            }
            ++q;
            if (++s == A_RING) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
        *issued_a = q;
      }
    } else if (warp >= 2) {
      // A loader. A block is 2048 copies of 16 bytes (a pair of elements
      // adjacent in the source); thread lt takes copies lt + 64 i, whose
      // source and shared-memory offsets are lt's part plus copy i's part.
      const int lt = threadIdx.x - 64;
      const float2* lane_src = A;
      std::uint32_t lane_dst = 0;
      for (int b = 0; b < 6; ++b)
        if ((lt >> b) & 1) {
          lane_src += g.lane_src[b];
          lane_dst ^= g.lane_dst[b];
        }
      const std::uint32_t ring = smem_u32(smem);
      int q = 0, s = 0;
      std::uint32_t ph = 0;
      bool ok = true;
      for (int t = first; t < total && ok; t += stride) {
        int mt, nt, batch;
        tile_of(t, mt, nt, batch);
        const float2* tile_src = lane_src + std::uint64_t(batch) * ac_stride;
        if (g.plain)
          tile_src += std::uint64_t(mt) * BM * std::uint64_t(k);
        else
          for (int b = 0; b < AGather::kBits && (mt >> b); ++b)
            if ((mt >> b) & 1) tile_src += g.tile_src[b];
        for (int b = 0; b < loads; ++b) {
          if (q >= A_RING && !wait(&raw_empty[s], ph ^ 1u, 5)) {
            ok = false;
            break;
          }
          const float2* src = tile_src;
          if (g.plain)
            src += b * 32;
          else
            for (int x = 0; x < AGather::kBits && (b >> x); ++x)
              if ((b >> x) & 1) src += g.block_src[x];
          const std::uint32_t dst = ring + s * A_BLOCK;
          if (!g.plain) {
            // Copies from copies_real on belong to the half of a block that a
            // k of 16 does not have: zeros.
#pragma unroll
            for (int i = 0; i < 32; ++i)
              cp_async16(dst + (lane_dst ^ g.copy_dst[i]), i < g.copies_real ? src + g.copy_src[i] : A,
                         i < g.copies_real ? 16u : 0u);
          } else {
            // Rows that are not 16-byte aligned (copy u covers row u / 16,
            // values 2 (u % 16) and the next).
            const int have = k - (b * 32 + 2 * (lt & 15));  // values from the pair on
            const int rows = have > 0 ? m - (mt * BM + (lt >> 4)) : 0;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const bool in = 4 * i < rows, in2 = in && have > 1;
              const float2* from = src + g.copy_src[i];
              const std::uint32_t to = dst + (lane_dst ^ g.copy_dst[i]);
              cp_async8(to, in ? from : A, in ? 8u : 0u);
              cp_async8(to + 8, in2 ? from + 1 : A, in2 ? 8u : 0u);
            }
          }
          cp_async_arrive(&raw_full[s]);
          ++q;
          if (++s == A_RING) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  } else if (warp >= 12) {
    // A converter: thread r, row r of the tile.
    QFX_SETMAXNREG_DEC(104);
    const int row = threadIdx.x - 384;
    std::uint32_t row_at = 0;
    for (int b = 0; b < 7; ++b)
      if ((row >> b) & 1) row_at ^= g.row_at[b];
    std::int8_t* exps = reinterpret_cast<std::int8_t*>(smem + L::OFF_EXP);
    const std::uint32_t ring = smem_u32(smem);
    const std::uint32_t lanes = tmem + TMEM_A + (std::uint32_t((warp - 12) * 32) << 16);
    int s = 0, x = 0, xa = 0, r = DONE - A_BUFS;
    std::uint32_t ph = 0, pd = 1, pe = 1;  // block w - A_BUFS: barrier r
    const bool odd = KIND == KIND_FP16 && (lane & 1);
    // Values of the thread's row from the first (h = 0) or second 16 of place s
    // of the ring on.
    auto read = [&](auto& v, int s, int h) {
      const std::uint32_t block = ring + s * A_BLOCK, at = h ? row_at ^ g.value_at[16] : row_at;
      constexpr int N = sizeof(v) / sizeof(v[0]);
      if (g.pairs) {
#pragma unroll
        for (int i = 0; i < N; i += 2)
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(v[i].x), "=f"(v[i].y), "=f"(v[i + 1].x), "=f"(v[i + 1].y)
                       : "r"(block + (at ^ g.value_at[i]))
                       : "memory");
      } else {
#pragma unroll
        for (int i = 0; i < N; ++i)
          asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];"
                       : "=f"(v[i].x), "=f"(v[i].y)
                       : "r"(block + (at ^ g.value_at[i]))
                       : "memory");
      }
    };
    // The values read are in registers: their place in the ring is free.
    auto release = [&] {
      __syncwarp();
      if (lane == 0) mbar_arrive(&raw_empty[s]);
    };
    // Waits for the MMAs of the block two back, whose place in TMEM comes
    // next, and (the odd lanes meanwhile) for the epilogue's reads of the
    // exponents EXP_RING blocks back.
    auto place = [&] {
      if (!__all_sync(0xffffffffu, wait(odd ? &exp_empty[x] : &done[r], odd ? pe : pd, 10))) return false;
      __syncwarp();
      if (++r == DONE) {
        r = 0;
        pd ^= 1u;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      return true;
    };
    // Block w: its values lie in one place of the ring, or (3xTF32) in half of
    // one, b counting the tile's blocks.
    for (int w = 0, b = 0; w < work; ++w) {
      const int half = VALUES == 16 ? b & 1 : 0;
      b = b == blocks - 1 ? 0 : b + 1;
      const bool last = VALUES == 32 || half || b == 0;
      if (!half && !__all_sync(0xffffffffu, wait(&raw_full[s], ph, 6))) break;
      const std::uint32_t to = lanes + xa * TMEM_A_BLOCK;
      if constexpr (KIND == KIND_BF16) {
        bool ok = true;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float2 v[16];
          read(v, s, h);
          if (h == 1) release();
          std::uint32_t p[48];  // 8 words of every plane
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            split_bf16(v[2 * j].x, v[2 * j + 1].x, p[j], p[8 + j], p[16 + j]);
            split_bf16(v[2 * j].y, v[2 * j + 1].y, p[24 + j], p[32 + j], p[40 + j]);
          }
          if (h == 0) ok = place();
          if (!ok) break;
          tmem_st32(to + 48 * h, p);
          tmem_st16(to + 48 * h + 32, p + 32);
        }
        if (!ok) break;
      } else {
        float2 v[VALUES];
        read(v, s, half);
        std::uint32_t p[2][32];  // of each k-step: 8 words of every plane
        int e = 0;
        if constexpr (KIND == KIND_FP16) {
          // Bit patterns of non-negative floats order like their values.
          std::uint32_t mx[4] = {0u, 0u, 0u, 0u};
#pragma unroll
          for (int i = 0; i < VALUES; ++i)
            mx[i & 3] =
                max(mx[i & 3], max(__float_as_uint(v[i].x) & 0x7fffffffu, __float_as_uint(v[i].y) & 0x7fffffffu));
          // e with max * 2^e in [2^14, 2^15), at most 126 (2^e and 2^-e stay
          // normal floats; smaller blocks keep all their bits: below 2^-112 the
          // lo planes reach further down than FP32 itself). A block of zeros
          // takes 126 so that it never sets the scale of the sum; infinities
          // and NaN keep 0.
          const int be = int(max(max(mx[0], mx[1]), max(mx[2], mx[3])) >> 23);
          e = be == 255 ? 0 : min(141 - be, 126);
          const float sc = __uint_as_float(std::uint32_t(e + 127) << 23);
          const float2 sc2 = make_float2(sc, sc);
#pragma unroll
          for (int i = 0; i < VALUES; i += 16)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float2 a = v[i + 2 * j], b2 = v[i + 2 * j + 1];
              const float2 re = mul2(make_float2(a.x, b2.x), sc2), im = mul2(make_float2(a.y, b2.y), sc2);
              split_pair(re.x, re.y, p[i / 16][j], p[i / 16][8 + j]);
              split_pair(im.x, im.y, p[i / 16][16 + j], p[i / 16][24 + j]);
            }
        } else {
#pragma unroll
          for (int i = 0; i < VALUES; ++i) {
            std::uint32_t* o = p[i / 8] + i % 8;
            const float rh = tf32_rn(v[i].x), ih = tf32_rn(v[i].y);
            o[0] = __float_as_uint(rh);
            o[8] = __float_as_uint(tf32_rn(v[i].x - rh));
            o[16] = __float_as_uint(ih);
            o[24] = __float_as_uint(tf32_rn(v[i].y - ih));
          }
        }
        if (last) release();
        if (!place()) break;
        tmem_st32(to, p[0]);
        tmem_st32(to + 32, p[1]);
        if constexpr (KIND == KIND_FP16) exps[x * BM + row] = std::int8_t(e);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) {
        if constexpr (KIND == KIND_FP16) mbar_arrive(&exp_full[x]);
        arrive(&a_full[xa]);
      }
      xa ^= 1;
      if (++x == EXP_RING) {
        x = 0;
        pe ^= 1u;
      }
      if (last && ++s == A_RING) {
        s = 0;
        ph ^= 1u;
      }
    }
  } else {
    // Epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 and one half of
    // the tile's columns. The tensor core's FP32 accumulation rounds toward
    // zero; keeping each chunk short and adding the chunks here with
    // round-to-nearest keeps the product as accurate as FP32 arithmetic.
    QFX_SETMAXNREG_INC(176);
    const int q = warp % 4;
    const int part = (warp - 4) / 4;
    const int row = q * 32 + lane;
    const std::int8_t* exps = reinterpret_cast<const std::int8_t*>(smem + L::OFF_EXP);
    std::uint8_t* staging = smem + L::OFF_STAGING + (warp - 4) * L::SLOTS * SLOT;
    int* sc_row = reinterpret_cast<int*>(smem + L::OFF_SCALE) + (warp - 4) * COLS;
    const float beta = debias_beta<KIND>(err, 2, (k + VALUES / 2 - 1) / (VALUES / 2));
    const float2 beta2 = make_float2(beta, beta);
    int h = 0, x = 0, r = 0;
    std::uint32_t pr = 0, px = 0;
    const bool odd = KIND == KIND_FP16 && (lane & 1);
    bool ok = true;
    const std::uint32_t base0 = tmem + (std::uint32_t(q * 32) << 16) + part * COLS;
    // Adds the next TMEM buffer, times `f`, to `sum`.
    auto drain = [&](float2(&sum)[COLS / 2], float2 f) {
      const std::uint32_t base = base0 + h * BN;
      constexpr int STEP = COLS < 32 ? COLS : 32;  // columns of one wait
#pragma unroll
      for (int j0 = 0; j0 < COLS; j0 += STEP) {
        std::uint32_t v[2][16];
#pragma unroll
        for (int i = 0; i < STEP / 16; ++i) TMEM_LD16(base + j0 + 16 * i, v[i]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < STEP / 2; ++j) {
          const std::uint32_t* w = v[j / 8] + 2 * (j % 8);
          float2& a = sum[j0 / 2 + j];
          a = fma2(make_float2(__uint_as_float(w[0]), __uint_as_float(w[1])), f, a);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) arrive(&acc_empty[h]);
      h = h == HALVES - 1 ? 0 : h + 1;
    };
    for (int t = first; t < total && ok; t += stride) {
      int mt, nt, batch;
      tile_of(t, mt, nt, batch);
      const int m0 = mt * BM, n0 = nt * BN + part * COLS;
      const int ncols = n - n0;
      // Exponents of the lane's columns, fetched before the drain.
      const int* eb = exp_b + std::uint64_t(batch) * n + n0;
      const int eb0 = KIND == KIND_FP16 && lane < min(ncols, COLS) ? eb[lane] : 0;
      const int eb1 = KIND == KIND_FP16 && COLS > 32 && 32 + lane < ncols ? eb[32 + lane] : eb0;
      float2 re[COLS / 2], im[COLS / 2];  // columns 2 j, 2 j + 1
#pragma unroll
      for (int j = 0; j < COLS / 2; ++j) re[j] = im[j] = make_float2(0.f, 0.f);
      // The sums are kept times 2^eref (and the column's 2^eb): a chunk of a
      // block with exponent e is added times 2^(eref - e) <= 1. eref starts
      // two below the first block's exponent and drops, rescaling the sums,
      // only when a later block is more than four times larger.
      int eref = 0;
      for (int b = 0; b < blocks; ++b) {
        // The odd lanes wait for the block's exponents.
        if (!__all_sync(0xffffffffu, wait(odd ? &exp_full[x] : &re_full[r], odd ? px : pr, 3))) {
          ok = false;
          break;
        }
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;");
        int e = 0;
        if constexpr (KIND == KIND_FP16) {
          e = exps[x * BM + row];
          __syncwarp();
          if (lane == 0) mbar_arrive(&exp_empty[x]);
          if (++x == EXP_RING) {
            x = 0;
            px ^= 1u;
          }
        }
        if (b == 0) {
          eref = KIND == KIND_FP16 ? e - 2 : 0;
        } else if (KIND == KIND_FP16 && __any_sync(0xffffffffu, e < eref)) {
          const int next = e < eref ? e - 2 : eref;
          const float f = pow2(next - eref);
          const float2 f2 = make_float2(f, f);
          eref = next;
#pragma unroll
          for (int j = 0; j < COLS / 2; ++j) {
            re[j] = mul2(re[j], f2);
            im[j] = mul2(im[j], f2);
          }
        }
        const float sa = pow2(eref - e);
        const float2 sa2 = make_float2(sa, sa);
        drain(re, sa2);
        if (!__all_sync(0xffffffffu, wait(&done[r], pr, 3))) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        drain(im, sa2);
        if (++r == DONE) {
          r = 0;
          pr ^= 1u;
        }
      }
      if (!ok) break;
      // The MMA issuer already works on the next tiles. The columns'
      // exponents go through 64 words of the warp's own shared memory, from
      // where four at a time are read as one broadcast.
      __syncwarp();
      if (lane < COLS) sc_row[lane] = eb0 << 23;
      if (COLS > 32) sc_row[32 + lane] = eb1 << 23;
      // When every scale 2^-(eref + eb) of the warp's block is a normal float
      // each element takes one multiply by it (exact unless the result leaves
      // the normal range). Otherwise the sums are scaled here, by two powers
      // of two each clamped to the normal range (the first is exact whenever
      // the result is normal), and the store multiplies by one: a branch per
      // element would keep the store's chains from overlapping (a tile's
      // store took 5500 cycles that way).
      const int lo = __reduce_min_sync(0xffffffffu, eref) + __reduce_min_sync(0xffffffffu, min(eb0, eb1));
      const int hi = __reduce_max_sync(0xffffffffu, eref) + __reduce_max_sync(0xffffffffu, max(eb0, eb1));
      __syncwarp();
      std::uint32_t c0 = std::uint32_t(127 - eref) << 23;
      if (hi > 126 || lo < -127) {
#pragma unroll
        for (int j = 0; j < COLS / 2; ++j) {
          const int t0 = -(eref + (sc_row[2 * j] >> 23)), t1 = -(eref + (sc_row[2 * j + 1] >> 23));
          const int a0 = min(max(t0 >> 1, -126), 127), b0 = min(max(t0 - a0, -126), 127);
          const int a1 = min(max(t1 >> 1, -126), 127), b1 = min(max(t1 - a1, -126), 127);
          const float2 fa = make_float2(pow2(a0), pow2(a1)), fb = make_float2(pow2(b0), pow2(b1));
          re[j] = mul2(mul2(re[j], fa), fb);
          im[j] = mul2(mul2(im[j], fa), fb);
        }
        c0 = 127u << 23;
        __syncwarp();
        if (lane < COLS) sc_row[lane] = 0;
        if (COLS > 32) sc_row[32 + lane] = 0;
        __syncwarp();
      }
#pragma unroll
      for (int j = 0; j < COLS / 2; ++j) {
        re[j] = fma2(re[j], beta2, re[j]);
        im[j] = fma2(im[j], beta2, im[j]);
      }
      if (watch) {
        float2 z[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};  // NaN once a sum is no number
#pragma unroll
        for (int j = 0; j < COLS / 2; ++j) {
          z[0] = fma2(re[j], make_float2(0.f, 0.f), z[0]);
          z[1] = fma2(im[j], make_float2(0.f, 0.f), z[1]);
        }
        const float zero = (z[0].x + z[0].y) + (z[1].x + z[1].y);
        if (__any_sync(0xffffffffu, zero != 0.f) && lane == 0) atomicExch(err + 4, watch);
      }
      float2* cb = C + std::uint64_t(batch) * ac_stride;
      // Boxes of 32 rows x 16 complex, the warp's slots in turn. (Boxes of 8
      // columns: twice the fences and barriers, a tile's store took 7200
      // cycles. A thread storing its own row piece in 32-byte sectors,
      // without shared memory, 9400.)
#pragma unroll
      for (int j0 = 0; j0 < COLS; j0 += 16) {
        std::uint8_t* slot = staging + (j0 / 16) % L::SLOTS * SLOT;
        if (tma_c) {
          if (lane == 0) {
            if (L::SLOTS == 2)
              bulk_wait_read1();
            else
              bulk_wait_read();
          }
          __syncwarp();
        }
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          const int4 es = *reinterpret_cast<const int4*>(sc_row + j0 + j);
          const float s0 = __uint_as_float(c0 - std::uint32_t(es.x)), s1 = __uint_as_float(c0 - std::uint32_t(es.y));
          const float s2 = __uint_as_float(c0 - std::uint32_t(es.z)), s3 = __uint_as_float(c0 - std::uint32_t(es.w));
          const int p = (j0 + j) / 2;
          // 128-byte swizzle: unit u of row r lies at u ^ (r % 8).
          const std::uint32_t u = j / 2, w = lane & 7;
          *reinterpret_cast<float4*>(slot + lane * 128 + ((u ^ w) << 4)) =
              make_float4(re[p].x * s0, im[p].x * s0, re[p].y * s1, im[p].y * s1);
          *reinterpret_cast<float4*>(slot + lane * 128 + (((u + 1) ^ w) << 4)) =
              make_float4(re[p + 1].x * s2, im[p + 1].x * s2, re[p + 1].y * s3, im[p + 1].y * s3);
        }
        if (tma_c) {
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            const int y = m0 + q * 32;
            if (y < m && j0 < ncols) tma_store_3d(&map_c, slot, 2 * (n0 + j0), y, batch);
            bulk_commit();
          }
        } else {
          // Odd n and unaligned outputs: two rows of 16 columns at a time.
          __syncwarp();
          for (int r0 = 0; r0 < 32; r0 += 2) {
            const int r = r0 + lane / 16, col = lane % 16;
            const float2 v = *reinterpret_cast<const float2*>(slot + r * 128 + (((col / 2) ^ (r & 7)) << 4) +
                                                              (col & 1) * 8);
            const int gr = m0 + q * 32 + r;
            if (gr < m && j0 + col < ncols) cb[std::uint64_t(gr) * n + n0 + j0 + col] = v;
          }
          __syncwarp();
        }
      }
    }
    // Every bulk store has written global memory before the CTA ends.
    if (tma_c && lane == 0) bulk_wait_all();
    __syncwarp();
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 1) {
    // Release TMEM only after every MMA this CTA issued (or, in a pair, that
    // read this CTA's memories) has completed; the wait is immediate unless
    // the pipeline was abandoned.
    const unsigned long long t0 = now_ns();
    while (!(PAIR ? mbar_test_cluster(mma_done, 0) : mbar_test(mma_done, 0)) && now_ns() - t0 < WAIT_NS) {
    }
  }
  if constexpr (PAIR) {
    if (threadIdx.x == 0) {
      auto tell = [&](volatile int* word, int v) {
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_addr(const_cast<int*>(word), rank ^ 1)), "r"(v)
                     : "memory");
      };
      tell(peer_abort, *abort_flag);
      if (rank == 1) tell(peer_b, *issued_b);
    }
    __syncthreads();
    cluster_sync();
  }
  if (*abort_flag || *peer_abort) {
    // Every copy asked for lands before shared memory is released (waits are
    // bounded here as well). A pair's stages of B complete on CTA 0's barriers:
    // where one CTA alone asked for its half of a stage, CTA 0 makes the
    // barrier expect that half only.
    if (threadIdx.x == 0) {
      auto land = [&](std::uint64_t* bar, std::uint32_t parity) {
        const unsigned long long t0 = now_ns();
        while (!mbar_test(bar, parity) && now_ns() - t0 < WAIT_NS) {
        }
      };
      const int qa = *issued_a, qb = *issued_b, qp = PAIR ? *peer_b : qb;
      for (int w = max(qa - A_RING, 0); w < qa; ++w) land(&raw_full[w % A_RING], (w / A_RING) & 1);
      const int last = max(qb, qp);
      for (int w = max(last - B_STAGES, 0); w < last && rank == 0; ++w) {
        std::uint64_t* bar = &b_full[w % B_STAGES];
        if (w >= qb)
          mbar_expect_tx(bar, B_STAGE);
        else if (w >= qp)
          asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(B_STAGE)
                       : "memory");
        land(bar, (w / B_STAGES) & 1);
      }
    }
    __syncthreads();
    if constexpr (PAIR) cluster_sync();
  }
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    if constexpr (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TMEM_COLS));
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TMEM_COLS));
  }
}

void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw std::string("ERROR (qflex_gb300: CUDA ") + what + ") --> " + cudaGetErrorString(e);
}

}  // namespace

AGather make_a_rows(std::size_t k, bool aligned) {
  AGather g;
  std::memset(&g, 0, sizeof(g));
  g.plain = 1;
  g.pairs = 1;
  g.copies_real = 32;
  g.boxes = aligned ? 1 : 0;
  // Boxes: rows of 16 values, 128 bytes, unit u of row r at u ^ (r % 8).
  // Copies: copy u = 16 row + pair; its unit of the block is u with the low
  // three bits XORed with the row's. Either way a quarter-warp of rows reading
  // the same values hits eight different units.
  auto at = [](std::uint32_t u) { return (u ^ ((u >> 4) & 7u)) << 4; };
  for (int b = 0; b < 6; ++b) {
    g.lane_src[b] = b < 4 ? std::uint64_t(2) << b : std::uint64_t(k) << (b - 4);
    g.lane_dst[b] = at(1u << b);
  }
  for (std::uint32_t i = 0; i < 32; ++i) {
    g.copy_src[i] = std::uint64_t(4) * i * k;
    g.copy_dst[i] = at(64u * i);
    g.value_at[i] = (aligned ? (i >> 4) * (A_BLOCK / 2) | ((i & 15) >> 1) << 4 : at(i >> 1)) | (i & 1u) << 3;
  }
  for (int b = 0; b < 7; ++b) g.row_at[b] = aligned ? 128u << b ^ (b < 3 ? 16u << b : 0u) : at(16u << b);
  return g;
}

bool make_a_gather(int nbits, const std::uint8_t* perm, std::size_t m, std::size_t k, AGather* g) {
  int kl = 0;
  while ((std::size_t(1) << kl) < k) ++kl;
  if ((std::size_t(1) << kl) != k || kl < 4 || nbits > 31 || m < std::size_t(BM) || (m << kl) >> nbits != 1)
    return false;
  int from[32] = {};  // source digit of every digit of the row-major operand
  for (int p = 0; p < nbits; ++p) from[perm[p]] = p;
  // A block's digits, 7 of the row and 5 of the value (4 when k = 16: then
  // the block's top digit is one that no value has), in source order.
  const int kb = kl < 5 ? kl : 5;
  int at_e[12], n_e = 0, row_e[7], val_e[5];
  for (int p = 0; p < nbits; ++p) {
    const int d = perm[p];
    if (d < kb)
      val_e[d] = n_e;
    else if (d >= kl && d < kl + 7)
      row_e[d - kl] = n_e;
    else
      continue;
    at_e[n_e++] = p;
  }
  if (kb < 5) val_e[4] = n_e;
  // The source's three lowest digits lie in the block: every copy of 16
  // bytes is a pair of neighbours and eight lanes read at least 64
  // consecutive bytes. (Tensors of the grid contractions keep their last
  // index, 3 or 4 digits, in one piece; anything else is permuted first.)
  if (at_e[0] != 0 || at_e[1] != 1 || at_e[2] != 2) return false;
  std::memset(g, 0, sizeof(*g));
  g->nbits = nbits;
  // Where element e of the block (source order) lies: unit e / 2 with its low
  // three bits XORed by one mask per higher bit, chosen so that the low row
  // digits, which the lanes of a reading warp differ in, reach different
  // units: lanes 0..7 read 16 bytes each (pairs) or lanes 0..15 8 bytes.
  std::uint32_t mask[11] = {};
  {
    std::uint32_t used = 0;
    int want[3], n_want = 0;
    for (int d = 0; d < 4 && n_want < 3; ++d)
      if (row_e[d] != 0) want[n_want++] = row_e[d] - 1;
    for (int w : want)
      if (w < 3) used |= 1u << w;
    for (int w : want)
      if (w >= 3) {
        const std::uint32_t free_bit = (used & 1) == 0 ? 1u : (used & 2) == 0 ? 2u : 4u;
        mask[w] = free_bit;
        used |= free_bit;
      }
  }
  auto at = [&](std::uint32_t e) {
    std::uint32_t u = e >> 1, x = u;
    for (int b = 3; b < 11; ++b)
      if ((u >> b) & 1) x ^= mask[b];
    return (x << 4) | ((e & 1u) << 3);
  };
  g->pairs = val_e[0] == 0 ? 1 : 0;
  g->copies_real = kb < 5 ? 16 : 32;
  for (int b = 0; b < 6; ++b) {
    g->lane_src[b] = std::uint64_t(1) << at_e[b + 1];
    g->lane_dst[b] = at(2u << b);
  }
  for (std::uint32_t i = 0; i < 32; ++i) {
    for (int b = 0; b < 5; ++b)
      if (((i >> b) & 1) && 7 + b < n_e) g->copy_src[i] += std::uint64_t(1) << at_e[7 + b];
    g->copy_dst[i] = at(i << 7);
    std::uint32_t e = 0;
    for (int q = 0; q < 5; ++q)
      if ((i >> q) & 1) e |= 1u << val_e[q];
    g->value_at[i] = at(e);
  }
  for (int d = 0; d < 7; ++d) g->row_at[d] = at(1u << row_e[d]);
  // As one TMA box when the block is 16 neighbours by at most three runs of
  // neighbouring digits: the run with the lowest row digit that is not among
  // the 16 comes next to them, where the 128-byte swizzle spreads the rows
  // that a reading warp's lanes differ in.
  if (at_e[3] == 3) {
    int start[4], len[4], runs = 0;
    for (int e = 4; e < n_e; ++e) {
      if (e == 4 || at_e[e] != at_e[e - 1] + 1) {
        if (runs == 3) {
          runs = 4;
          break;
        }
        start[runs] = e;
        len[runs++] = 0;
      }
      ++len[runs - 1];
    }
    if (runs <= 3) {
      int low = 0;
      while (low < 6 && row_e[low] < 4) ++low;
      for (int x = 1; x < runs; ++x)
        if (row_e[low] >= start[x] && row_e[low] < start[x] + len[x]) {
          std::swap(start[0], start[x]);
          std::swap(len[0], len[x]);
        }
      std::uint32_t box_at[12];  // where the block's digits lie in the box
      for (int e = 0; e < 4; ++e) box_at[e] = 8u << e;
      std::uint32_t next = 128;
      for (int x = 0; x < 3; ++x) {
        g->run_bits[x] = x < runs ? len[x] : 0;
        g->run_src[x] = x < runs ? std::uint64_t(1) << at_e[start[x]] : 16;
        for (int e = 0; e < g->run_bits[x]; ++e, next <<= 1)
          box_at[start[x] + e] = next < 1024 ? next | next >> 3 : next;
      }
      box_at[11] = n_e == 11 ? 1u << 14 : box_at[11];
      g->boxes = 1;
      for (std::uint32_t i = 0; i < 32; ++i) {
        g->value_at[i] = 0;
        for (int q = 0; q < 5; ++q)
          if ((i >> q) & 1) g->value_at[i] ^= box_at[val_e[q]];
      }
      for (int d = 0; d < 7; ++d) g->row_at[d] = box_at[row_e[d]];
    }
  }
  for (int b = 0; kl + 7 + b < nbits; ++b) g->tile_src[b] = std::uint64_t(1) << from[kl + 7 + b];
  for (int b = 0; 5 + b < kl; ++b) g->block_src[b] = std::uint64_t(1) << from[5 + b];
  return true;
}

void a_gather_on_host(const AGather& g, std::size_t m, std::size_t k, const float2* src, float2* dst) {
  std::vector<float2> block(A_BLOCK / sizeof(float2));
  for (std::size_t mt = 0; mt < m / BM; ++mt)
    for (std::size_t b = 0; b < (k + 31) / 32; ++b) {
      std::uint64_t base = 0;
      for (int x = 0; x < AGather::kBits; ++x) {
        if ((mt >> x) & 1) base += g.tile_src[x];
        if ((b >> x) & 1) base += g.block_src[x];
      }
      std::fill(block.begin(), block.end(), make_float2(NAN, NAN));
      if (g.boxes && g.copies_real < 32)
        std::fill(block.begin() + A_BLOCK / 16, block.end(), make_float2(0.f, 0.f));
      const std::uint32_t rows = 8u << (g.run_bits[0] + g.run_bits[1] + g.run_bits[2] + 4);
      if (g.boxes && rows != (g.copies_real == 32 ? A_BLOCK : A_BLOCK / 2))
        throw std::string("ERROR (qflex_gb300: product) --> box of a wrong size");
      for (std::uint32_t at = 0; g.boxes && at < rows; at += 8) {
        std::uint64_t from = base + ((at >> 3) & 15);
        std::uint32_t rest = at >> 7;
        for (int x = 0; x < 3; ++x) {
          from += (rest & ((1u << g.run_bits[x]) - 1)) * g.run_src[x];
          rest >>= g.run_bits[x];
        }
        if (base % 16 || from >= m * k) throw std::string("ERROR (qflex_gb300: product) --> box out of range");
        block[(at ^ ((at >> 3) & 0x70)) / 8] = src[from];
      }
      for (int u = 0; !g.boxes && u < 2048; ++u) {
        std::uint64_t from = base + g.copy_src[u / LOADERS];
        std::uint32_t to = g.copy_dst[u / LOADERS];
        for (int x = 0; x < 6; ++x)
          if ((u >> x) & 1) {
            from += g.lane_src[x];
            to ^= g.lane_dst[x];
          }
        const bool real = u / LOADERS < g.copies_real;
        if ((real && (from + 2 > m * k || from % 2)) || to + 16 > A_BLOCK || to % 16)
          throw std::string("ERROR (qflex_gb300: product) --> copy out of range");
        for (int h = 0; h < 2; ++h) block[to / 8 + h] = real ? src[from + h] : make_float2(0.f, 0.f);
      }
      for (int row = 0; row < BM; ++row) {
        std::uint32_t at = 0;
        for (int x = 0; x < 7; ++x)
          if ((row >> x) & 1) at ^= g.row_at[x];
        for (std::size_t v = 0; v < 32 && b * 32 + v < k; ++v) {
          const std::uint32_t slot = at ^ g.value_at[v];
          if (slot + 8 > A_BLOCK || (g.pairs && v % 2 && slot != ((at ^ g.value_at[v - 1]) | 8u)))
            throw std::string("ERROR (qflex_gb300: product) --> block read out of range");
          dst[(mt * BM + row) * k + b * 32 + v] = block[slot / 8];
        }
      }
    }
}

// Columns of a tile: the narrowest that holds n, for fewer MMAs and smaller
// B stages and so more blocks of A in flight. In tiles of 128, 64 and 32:
// (32768, 64, 64) x 16 112 and 86 us (reading A and writing C alone 80),
// (1048576, 16, 256) 498 and, in tiles of 32, 353 us (342).
static int direct_columns(std::size_t n) { return n <= 32 ? 32 : n <= 64 ? 64 : 128; }
// Pairs where a second row tile exists and the MMAs of a tile take longer than
// its store, which starts later in a pair. 3xFP16, single CTAs against pairs:
// (65536, 256, k) x 4 with k = 32 104 and 106 us, 64 143 and 149, 256 301 and
// 286; (8192, 128, 128) x 16 59 and 60.5; (4096, 1024, 4096) 272 and 240.
// 3xTF32 takes twice the MMAs; with k = 32 and 64 pairs cost a short launch 2 us
// and win from some 1000 tiles on: (16384, 256, 32) x 4 46 and 44, (16384, 8192,
// 32) 253 and 242, (65536, 256, 64) x 4 187 and 173, but (512, 512, 64) 19 and
// 21, and with half a tile of columns (65536, 64, 64) x 4 85 and 88. BF16x3 runs
// in pairs alone: split and product,
// and this, (65536, 256, k) x 4 with k = 16 122 and 98 us, 64 200 and 154;
// (32768, 64, 64) x 16 220 and 133; (256, 256, 64) 12 and 12.
bool tc_direct_pair(SplitKind kind, std::size_t m, std::size_t k) {
  return m > (std::size_t)BM && k > (kind == KIND_FP16 ? 128u : kind == KIND_TF32 ? 64u : 0u);
}

std::size_t tc_direct_workspace_elems(SplitKind kind, std::size_t n, std::size_t k) {
  if (kind == KIND_TF32) return 4 * n * ((k + 7) / 8 * 8);
  if (kind == KIND_BF16) return 3 * n * ((k + 15) / 16 * 16);
  return 2 * n * ((k + 15) / 16 * 16) + 2 * n;  // B's planes, exponents and largest components
}

void launch_cgemm_direct(SplitKind kind, const float2* A, const AGather& gather, const float2* B, BLayout b_layout,
                         float2* C, std::size_t m, std::size_t n, std::size_t k, std::uint64_t ac_stride,
                         std::uint64_t b_stride, int batch, float* workspace, int* err, const TcConfig& cfg,
                         cudaStream_t s, int watch) {
  if (!tc_runs(m, n, k)) throw std::string("ERROR (qflex_gb300: tensor cores) --> shape not eligible");
  if (cfg.chunk != 2)
    throw std::string("ERROR (qflex_gb300: tensor cores) --> the direct product takes chunks of 2 k-steps");
  if (gather.boxes && !gather.plain && batch > 1) {
    if (ac_stride % 16) throw std::string("ERROR (qflex_gb300: tensor cores) --> batch stride of a gathered operand");
    // The box's last coordinate counts 128 bytes in 31 bits.
    const std::uint64_t most = ((std::uint64_t(1) << 35) - (std::uint64_t(1) << gather.nbits)) / ac_stride + 1;
    if (most < (std::uint64_t)batch) {
      for (int at = 0; at < batch; at += (int)most)
        launch_cgemm_direct(kind, A + at * ac_stride, gather, B + at * b_stride, b_layout, C + at * ac_stride, m, n, k,
                            ac_stride, b_stride, (int)std::min<std::uint64_t>(most, batch - at), workspace, err, cfg,
                            s, watch);
      return;
    }
  }
  const int bn = kind == KIND_FP16 ? direct_columns(n) : 128;
  const std::size_t singles = ((m + BM - 1) / BM) * ((n + 127) / 128) * (std::size_t)batch;
  const bool pair = bn == 128 && (tc_direct_pair(kind, m, k) ||
                                  (kind == KIND_TF32 && m > (std::size_t)BM && n > 64 && k > 16 && singles >= 1000));
  if (kind == KIND_BF16 && !pair)
    throw std::string("ERROR (qflex_gb300: tensor cores) --> the direct BF16x3 product runs in pairs");
  const int b_cols = pair ? bn / 2 : bn;
  int* eb = nullptr;
  CUtensorMap mb, mb2;
  std::memset(&mb2, 0, sizeof(mb2));
  if (kind == KIND_FP16) {
    const std::size_t kpad = (k + 15) / 16 * 16;
    __half* pb = reinterpret_cast<__half*>(workspace);
    eb = reinterpret_cast<int*>(pb + 4 * n * kpad * (std::size_t)batch);
    std::uint32_t* top = reinterpret_cast<std::uint32_t*>(eb + n * (std::size_t)batch);
    launch_split(KIND_FP16, 4, {pb, nullptr, eb, top}, B, n, k, b_stride, batch, b_layout == BLayout::kn, s);
    mb = plane_map_f16(pb, n, kpad, batch, b_cols, 64);
  } else if (kind == KIND_BF16) {
    const std::size_t kpad = (k + 15) / 16 * 16;
    __nv_bfloat16* pb = reinterpret_cast<__nv_bfloat16*>(workspace);
    __nv_bfloat16* pt = pb + 4 * n * kpad * (std::size_t)batch;
    launch_split(KIND_BF16, 4, {pb, pt}, B, n, k, b_stride, batch, b_layout == BLayout::kn, s);
    mb = plane_map_bf16(pb, n, kpad, batch, b_cols, 64, 32);
    mb2 = plane_map_bf16(pt, n, kpad, batch, b_cols, 32, 16);
  } else {
    launch_split(KIND_TF32, 4, {workspace}, B, n, k, b_stride, batch, b_layout == BLayout::kn, s);
    mb = plane_map(workspace, n, (k + 7) / 8 * 8, batch, b_cols, 32, 16);
  }
  CUtensorMap ma;
  std::memset(&ma, 0, sizeof(ma));
  if (gather.boxes && gather.plain) {
    const std::uint64_t dims[3] = {k, m, (std::uint64_t)batch};
    const std::uint64_t strides[2] = {k * 8, (batch > 1 ? ac_stride : m * k + (m * k & 1)) * 8};
    const std::uint32_t box[3] = {16, BM, 1};
    ma = element_map(A, 3, dims, strides, box);
  } else if (gather.boxes) {
    const std::uint64_t units = ((batch - 1) * ac_stride + (std::uint64_t(1) << gather.nbits)) / 16;
    std::uint64_t dims[5] = {16, 1, 1, 1, units}, strides[4] = {0, 0, 0, 128};
    std::uint32_t box[5] = {16, 1, 1, 1, 1};
    for (int x = 0; x < 3; ++x) {
      dims[1 + x] = box[1 + x] = 1u << gather.run_bits[x];
      strides[x] = gather.run_src[x] * 8;
    }
    ma = element_map(A, 5, dims, strides, box);
  }
  CUtensorMap mc;
  const int tma_c = output_map(C, m, n, ac_stride, batch, &mc) ? 1 : 0;
  const std::size_t rows = pair ? 2 * BM : BM;
  const std::size_t tiles = ((m + rows - 1) / rows) * ((n + bn - 1) / bn) * (std::size_t)batch;
  auto run = [&](auto of_kind, auto columns, auto paired) {
    constexpr int BN = decltype(columns)::value;
    constexpr int KIND = decltype(of_kind)::value;
    constexpr bool PAIR = decltype(paired)::value;
    auto* kernel = cgemm_direct_kernel<KIND, BN, PAIR>;
    cudaLaunchConfig_t lc = {};
    lc.blockDim = dim3(THREADS, 1, 1);
    lc.dynamicSmemBytes = Layout<KIND, BN, PAIR>::SMEM;
    lc.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    lc.attrs = at;
    lc.numAttrs = PAIR ? 1 : 0;
    static PerDevice pairs;  // resident at once (SMs pair up within a GPC)
    const int resident = pairs([&] {
      raise_smem_limit(kernel, Layout<KIND, BN, PAIR>::SMEM);
      int v = 1;
      lc.gridDim = dim3(2, 1, 1);
      if (PAIR && (cudaOccupancyMaxActiveClusters(&v, kernel, &lc) != cudaSuccess || v < 1)) {
        cudaGetLastError();
        v = (int)persistent_grid(1u << 20) / 2;
      }
      return v;
    });
    lc.gridDim = dim3(PAIR ? 2 * (unsigned)std::min<std::size_t>(tiles, (std::size_t)resident) : persistent_grid(tiles),
                      1, 1);
    check(cudaLaunchKernelEx(&lc, kernel, ma, mb, mb2, mc, gather, A, C, tma_c, (int)m, (int)n, (int)k, batch, ac_stride, err,
                             (const int*)eb, watch),
          "cgemm_direct");
  };
  using std::integral_constant;
  const integral_constant<int, KIND_FP16> fp16;
  const integral_constant<int, KIND_TF32> tf32;
  const integral_constant<int, 128> c128;
  if (kind == KIND_BF16)
    run(integral_constant<int, KIND_BF16>{}, c128, std::true_type{});
  else if (kind == KIND_TF32)
    pair ? run(tf32, c128, std::true_type{}) : run(tf32, c128, std::false_type{});
  else if (bn == 128)
    pair ? run(fp16, c128, std::true_type{}) : run(fp16, c128, std::false_type{});
  else if (bn == 64)
    run(fp16, integral_constant<int, 64>{}, std::false_type{});
  else
    run(fp16, integral_constant<int, 32>{}, std::false_type{});
  check(cudaGetLastError(), "cgemm_direct");
}

}  // namespace qfx
