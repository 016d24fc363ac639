// The 3xFP16 product that splits A itself (sm_103a, tcgen05 + TMEM + TMA).
//
// C = A * B, A complex64 in global memory, B as FP16 planes of Bt (n x k,
// K-major, see split_fp16_kernel). A is brought in as it lies -- row-major,
// or through the index permutation that would have laid it out so (AGather)
// -- and split into its four FP16 planes inside the kernel. Against a split
// kernel (or a plane-writing permutation) before the product that saves one
// pass over A: 8 B read and 8 B written per element.
//
// Structure: persistent, one CTA per SM over 128 x 128 complex tiles, 512
// threads in four warpgroups whose registers setmaxnreg divides (56, 176,
// 176, 104 per thread: 128 on average, the launch's own share).
//   warp 0       B producer: two 8 KB TMA boxes per k-step (re and im rows of
//                64 bytes, hi and lo)
//   warp 1       TMEM allocation; issues every MMA
//   warps 2, 3   A loader: 16-byte cp.async copies of one 128 x 32 block of A
//                (32 KB) into a ring of three blocks
//   warps 4..11  epilogue: drains TMEM chunks, scales and stores the tile
//   warps 12..15 A converter: thread r reads row r of the block, finds the
//                largest component, scales by the power of two that brings it
//                into [2^14, 2^15), splits into hi + lo and writes the two
//                k-steps' 128-byte plane rows over the block it came from
// A block is two k-steps of 16, one TMEM chunk at the default chunk length,
// so the epilogue applies the block's exponent as it adds the chunk.
//
// What bounds it: a k-step's MMAs take 768 cycles of the tensor pipe and read
// 84 KB of operands; those reads (672 cycles at 128 bytes a cycle) share the
// way with the fills, 128 cycles of B's TMA boxes and 128 of A's copies: 928,
// and 938 measured at k = 4096. (The kernel that loads A's planes: 576 + 320 =
// 896, where the card's power limit is near.) At short k the converter comes
// next, about 1800 cycles a block of two k-steps, and a tile's store, 6100
// cycles of which two chunks of the next tile's MMAs overlap: (65536, 256,
// 256) x 4 takes 2930 cycles a block, 341 us; (65536, 256, 16) x 4 93 us.
//
// B holds no negated copy: Ar multiplies (Br; Bi) in one N = 256 MMA, and Ai
// takes two N = 128 MMAs, -Ai Bi (the descriptor's negate-A bit) and Ai Br.
// N = 128 MMAs run at the same rate, and a k-step loads 16 KB of B, not 24.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "half_split.cuh"
#include "tc_common.cuh"
#include "tc_gemm.h"

namespace qfx {
namespace {

constexpr int BM = 128, BN = 128;
constexpr int A_RING = 3;                   // blocks of 128 rows x 32 values
constexpr int A_BLOCK = 128 * 32 * 8;       // bytes, complex64 or two k-steps of planes
constexpr int B_STAGES = 4;                 // one k-step each
constexpr int B_PART = BN * 64;             // re or im rows of a k-step (hi, lo)
constexpr int B_STAGE = 2 * B_PART;
constexpr int EXP_RING = 6;                 // block exponents, see the converter
constexpr int OFF_B = A_RING * A_BLOCK;
constexpr int SLOT = 4096;                  // output box: 32 rows x 16 complex
constexpr int OFF_STAGING = OFF_B + B_STAGES * B_STAGE;
constexpr int OFF_SCALE = OFF_STAGING + 8 * 2 * SLOT;
constexpr int OFF_EXP = OFF_SCALE + 8 * (BN / 2) * 4;  // after each epilogue warp's column exponents
constexpr int OFF_BAR = OFF_EXP + EXP_RING * BM;
constexpr int N_BARS = 3 * A_RING + 2 * B_STAGES + 4 + 1;
constexpr int SMEM = OFF_BAR + N_BARS * 8 + 8;
static_assert(SMEM <= 227 * 1024, "one CTA's shared memory");
constexpr int TMEM_COLS = 512;  // two chunk buffers of (re, im) x 128 columns
constexpr int THREADS = 512;
constexpr int LOADERS = 64, CONVERTERS = 128;

// One k-step: A's planes (re hi, lo, im hi, lo 32 bytes apart in 128-byte
// rows) against B's re rows (`blo`, hi and lo 32 bytes apart) and im rows
// (B_PART further), small terms first.
__device__ __forceinline__ void mma_kstep(std::uint32_t d, std::uint32_t alo, std::uint32_t ahi, std::uint32_t blo,
                                          std::uint32_t bhi, std::uint32_t acc) {
  constexpr std::uint32_t wide = idesc_f16(BM, 2 * BN, false), pos = idesc_f16(BM, BN, false),
                          neg = idesc_f16(BM, BN, true);
  static_assert(B_PART / 16 == 512, "offset of the im rows below");
  asm volatile(
      "{\n .reg .pred p0, p1;\n .reg .b32 l1, l2, l3, m1, m2, m3, dm;\n"
      " .reg .b64 arh, arl, aih, ail, brh, brl, bih, bil;\n"
      " setp.ne.b32 p0, %5, 0;\n setp.eq.b32 p1, %5, %5;\n"
      " add.u32 l1, %1, 2;\n add.u32 l2, %1, 4;\n add.u32 l3, %1, 6;\n"
      " add.u32 m1, %3, 2;\n add.u32 m2, %3, 512;\n add.u32 m3, %3, 514;\n add.u32 dm, %0, 128;\n"
      " mov.b64 arh, {%1, %2};\n mov.b64 arl, {l1, %2};\n mov.b64 aih, {l2, %2};\n mov.b64 ail, {l3, %2};\n"
      " mov.b64 brh, {%3, %4};\n mov.b64 brl, {m1, %4};\n mov.b64 bih, {m2, %4};\n mov.b64 bil, {m3, %4};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], arh, brl, %6, p0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], arl, brh, %6, p1;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], aih, bil, %8, p1;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [dm], aih, brl, %7, p1;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], ail, bih, %8, p1;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [dm], ail, brh, %7, p1;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], arh, brh, %6, p1;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], aih, bih, %8, p1;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [dm], aih, brh, %7, p1;\n}\n" ::"r"(d),
      "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(acc), "r"(wide), "r"(pos), "r"(neg));
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
// Whether every converter thread says yes; also their barrier.
__device__ __forceinline__ bool converters_all(bool ok) {
  int r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 p, %1, 0;\n barrier.cta.red.and.pred q, 1, %2, p;\n"
      " selp.b32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"(int(ok)), "n"(CONVERTERS)
      : "memory");
  return r != 0;
}

#define QFX_SETMAXNREG_DEC(n) asm volatile("setmaxnreg.dec.sync.aligned.u32 " #n ";")
#define QFX_SETMAXNREG_INC(n) asm volatile("setmaxnreg.inc.sync.aligned.u32 " #n ";")

__global__ void __launch_bounds__(THREADS, 1)
    cgemm_fp16x3_direct_kernel(const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_c,
                               const __grid_constant__ AGather g, const float2* __restrict__ A,
                               float2* __restrict__ C, int tma_c, int m, int n, int k, int batches,
                               std::uint64_t ac_stride, int* __restrict__ err, int CHUNK,
                               const int* __restrict__ exp_b) {
  extern __shared__ __align__(1024) std::uint8_t smem[];
  std::uint64_t* raw_full = reinterpret_cast<std::uint64_t*>(smem + OFF_BAR);  // a block of A has landed
  std::uint64_t* a_full = raw_full + A_RING;                                   // its planes are written
  std::uint64_t* a_empty = a_full + A_RING;                                    // its MMAs are done
  std::uint64_t* b_full = a_empty + A_RING;
  std::uint64_t* b_empty = b_full + B_STAGES;
  std::uint64_t* acc_full = b_empty + B_STAGES;
  std::uint64_t* acc_empty = acc_full + 2;
  std::uint64_t* mma_done = acc_empty + 2;
  std::uint32_t* tmem_slot = reinterpret_cast<std::uint32_t*>(mma_done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  if (smem_u32(smem) & 1023) {  // the swizzles need it; the layout leaves no room to round up
    if (threadIdx.x == 0) atomicExch(err, 9);
    return;
  }

  // Uniform for the compiler: see the MMA issuer.
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x / 32, 0), lane = threadIdx.x % 32;
  const int first = blockIdx.x, stride = gridDim.x;
  const int tiles_m = (m + BM - 1) / BM;
  const int tiles_n = (n + BN - 1) / BN;
  const int per_batch = tiles_m * tiles_n;
  const int total = per_batch * batches;
  // Tiles run in groups of 8 row-tiles so that the CTAs working at one time
  // share A rows and B columns in L2.
  auto tile_of = [&](int t, int& mt, int& nt, int& batch) {
    batch = t / per_batch;
    const int r = t % per_batch;
    const int per_group = 8 * tiles_n;
    const int group = r / per_group, in_group = r % per_group;
    const int group_m = min(8, tiles_m - group * 8);
    mt = group * 8 + in_group % group_m;
    nt = in_group / group_m;
  };
  auto wait = [&](std::uint64_t* bar, std::uint32_t parity, int code) {
    return mbar_wait(bar, parity, abort_flag, err, code);
  };
  const int kblocks = (k + 15) / 16;       // k-steps
  const int blocks = (kblocks + 1) / 2;    // blocks of A

  if (threadIdx.x == 0) {
    for (int s = 0; s < A_RING; ++s) {
      mbar_init(&raw_full[s], LOADERS);
      mbar_init(&a_full[s], CONVERTERS / 32);
      mbar_init(&a_empty[s], 1);
    }
    for (int s = 0; s < B_STAGES; ++s) {
      mbar_init(&b_full[s], 1);
      mbar_init(&b_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 8);
    }
    mbar_init(mma_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const std::uint32_t tmem = *tmem_slot;

  if (warp < 4) {
    QFX_SETMAXNREG_DEC(56);
    if (warp == 0 && lane == 0) {
      // B producer.
      int q = 0, s = 0;
      std::uint32_t ph = 0;
      for (int t = first; t < total && !*abort_flag; t += stride) {
        int mt, nt, batch;
        tile_of(t, mt, nt, batch);
        for (int kb = 0; kb < kblocks; ++kb) {
          if (q >= B_STAGES && !wait(&b_empty[s], ph ^ 1u, 1)) break;
          std::uint8_t* st = smem + OFF_B + s * B_STAGE;
          mbar_expect_tx(&b_full[s], B_STAGE);
          tma_load_4d(&map_b, &b_full[s], st, 0, nt * BN, kb, batch);
          tma_load_4d(&map_b, &b_full[s], st + B_PART, 32, nt * BN, kb, batch);
          ++q;
          if (++s == B_STAGES) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      if (*abort_flag) {
        // The copies already issued land before the CTA's shared memory is
        // released (bounded as well).
        for (int w = q > B_STAGES ? q - B_STAGES : 0; w < q; ++w) {
          const unsigned long long t0 = now_ns();
          while (!mbar_test(&b_full[w % B_STAGES], (w / B_STAGES) & 1) && now_ns() - t0 < WAIT_NS) {
          }
        }
      }
    } else if (warp == 1) {
      // MMA issuer. The whole warp runs the loop in step and one elected lane
      // issues: the descriptors then live in uniform registers. Run by one
      // lane alone, every descriptor word moved there before each MMA, and
      // beside the other warps' work a k-step took 980 cycles instead of 775
      // (768 at the tensor pipe's rate; measured with this k-step, its
      // commits and barrier tests, a TMEM drain and shared-memory traffic).
      // Chunk c (CHUNK k-steps of one tile, c counts across tiles)
      // accumulates from zero into TMEM buffer c % 2.
      const bool leader = elect_one();
      const std::uint64_t da = smem_desc_sw128(smem_u32(smem)), db = smem_desc_sw64(smem_u32(smem + OFF_B));
      const std::uint32_t a_hi = std::uint32_t(da >> 32), b_hi = std::uint32_t(db >> 32);
      const std::uint32_t a_lo0 = std::uint32_t(da), b_lo0 = std::uint32_t(db);
      auto wait_all = [&](std::uint64_t* bar, std::uint32_t parity, int code) {
        return __all_sync(0xffffffffu, wait(bar, parity, code));
      };
      int sa = 0, sb = 0, c = 0, kc = 0;
      std::uint32_t pa = 0, pb = 0;
      bool go = true;
      for (int t = first; t < total && go; t += stride) {
        kc = 0;
        for (int kb = 0; kb < kblocks; ++kb) {
          const int buf = c & 1;
          const bool start = kc == 0;
          if (start && c >= 2) {
            // The epilogue's TMEM reads of this buffer precede the MMAs that
            // overwrite it.
            if (!wait_all(&acc_empty[buf], ((c >> 1) - 1) & 1, 4)) {
              go = false;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
          }
          if (!(kb & 1) && !wait_all(&a_full[sa], pa, 7)) {
            go = false;
            break;
          }
          if (!wait_all(&b_full[sb], pb, 2)) {
            go = false;
            break;
          }
          const bool block_end = (kb & 1) || kb == kblocks - 1;
          const bool chunk_end = ++kc == CHUNK || kb == kblocks - 1;
          if (leader) {
            mma_kstep(tmem + buf * 2 * BN, a_lo0 + ((sa * A_BLOCK + (kb & 1) * (A_BLOCK / 2)) >> 4), a_hi,
                      b_lo0 + ((sb * B_STAGE) >> 4), b_hi, start ? 0u : 1u);
            umma_commit(&b_empty[sb]);
            if (block_end) umma_commit(&a_empty[sa]);
            if (chunk_end) umma_commit(&acc_full[buf]);
          }
          __syncwarp();
          if (++sb == B_STAGES) {
            sb = 0;
            pb ^= 1u;
          }
          if (block_end && ++sa == A_RING) {
            sa = 0;
            pa ^= 1u;
          }
          if (chunk_end) {
            ++c;
            kc = 0;
          }
        }
      }
      if (leader) umma_commit(mma_done);
      __syncwarp();
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
        for (int b = 0; b < blocks; ++b) {
          if (q >= A_RING && !wait(&a_empty[s], ph ^ 1u, 5)) {
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
          if (!g.plain || (g.aligned && (mt + 1) * BM <= m && (b + 1) * 32 <= k)) {
            // Copies from copies_real on belong to the half of a block that a
            // k of 16 does not have: zeros.
#pragma unroll
            for (int i = 0; i < 32; ++i)
              cp_async16(dst + (lane_dst ^ g.copy_dst[i]), i < g.copies_real ? src + g.copy_src[i] : A,
                         i < g.copies_real ? 16u : 0u);
          } else {
            // Edge blocks and rows that are not 16-byte aligned (plain rows:
            // copy u covers row u / 16, values 2 (u % 16) and the next).
            const int have = min(2, k - (b * 32 + 2 * (lt & 15)));  // values of a pair that exist
            const int rows = have > 0 ? m - (mt * BM + (lt >> 4)) : 0;
            if (g.aligned) {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const bool in = 4 * i < rows;
                cp_async16(dst + (lane_dst ^ g.copy_dst[i]), in ? src + g.copy_src[i] : A, in ? 8u * have : 0u);
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const bool in = 4 * i < rows, in2 = in && have > 1;
                const float2* from = src + g.copy_src[i];
                const std::uint32_t to = dst + (lane_dst ^ g.copy_dst[i]);
                cp_async8(to, in ? from : A, in ? 8u : 0u);
                cp_async8(to + 8, in2 ? from + 1 : A, in2 ? 8u : 0u);
              }
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
    std::int8_t* exps = reinterpret_cast<std::int8_t*>(smem + OFF_EXP);
    const std::uint32_t ring = smem_u32(smem);
    int s = 0, x = 0;
    std::uint32_t ph = 0;
    bool ok = true;
    for (int t = first; t < total && ok; t += stride) {
      for (int b = 0; b < blocks; ++b) {
        const bool here = wait(&raw_full[s], ph, 6);
        const std::uint32_t block = ring + s * A_BLOCK;
        float2 v[32];
        if (here) {
          if (g.pairs) {
#pragma unroll
            for (int i = 0; i < 32; i += 2)
              asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                           : "=f"(v[i].x), "=f"(v[i].y), "=f"(v[i + 1].x), "=f"(v[i + 1].y)
                           : "r"(block + (row_at ^ g.value_at[i]))
                           : "memory");
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];"
                           : "=f"(v[i].x), "=f"(v[i].y)
                           : "r"(block + (row_at ^ g.value_at[i]))
                           : "memory");
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = make_float2(0.f, 0.f);
        }
        // Every row is in registers before any thread writes planes over the
        // block.
        if (!converters_all(here)) {
          ok = false;
          break;
        }
        // Bit patterns of non-negative floats order like their values.
        std::uint32_t mx[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int i = 0; i < 32; ++i)
          mx[i & 3] = max(mx[i & 3], max(__float_as_uint(v[i].x) & 0x7fffffffu, __float_as_uint(v[i].y) & 0x7fffffffu));
        // e with max * 2^e in [2^14, 2^15), at most 126 (2^e and 2^-e stay
        // normal floats; smaller blocks keep all their bits: below 2^-112 the
        // lo planes reach further down than FP32 itself). A block of zeros
        // takes 126 so that it never sets the scale of the sum; infinities
        // and NaN keep 0.
        const int be = int(max(max(mx[0], mx[1]), max(mx[2], mx[3])) >> 23);
        const int e = be == 255 ? 0 : min(141 - be, 126);
        const float sc = __uint_as_float(std::uint32_t(e + 127) << 23);
        const float2 sc2 = make_float2(sc, sc);
#pragma unroll
        for (int i = 0; i < 32; i += 8) {  // 8 values: one 16-byte unit of every plane
          std::uint32_t rh[4], rl[4], ih[4], il[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 a = v[i + 2 * j], b2 = v[i + 2 * j + 1];
            const float2 r = mul2(make_float2(a.x, b2.x), sc2), im = mul2(make_float2(a.y, b2.y), sc2);
            split_pair(r.x, r.y, rh[j], rl[j]);
            split_pair(im.x, im.y, ih[j], il[j]);
          }
          // k-step i / 16; unit u of the 128-byte row (two per plane) lies at
          // u ^ (row % 8).
          const std::uint32_t at = block + (i / 16) * (A_BLOCK / 2) + row * 128;
          const std::uint32_t h = (i / 8) & 1;
          auto put = [&](std::uint32_t u, const std::uint32_t* w) {
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + (((u + h) ^ (row & 7)) << 4)), "r"(w[0]),
                         "r"(w[1]), "r"(w[2]), "r"(w[3])
                         : "memory");
          };
          put(0, rh);
          put(2, rl);
          put(4, ih);
          put(6, il);
        }
        // Exponents live in a ring of their own: this block is at most four
        // ahead of the one the slowest epilogue warp drains (its MMAs are
        // done with the block three back, which needed all chunks up to five
        // back drained).
        exps[x * BM + row] = std::int8_t(e);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[s]);
        if (++x == EXP_RING) x = 0;
        if (++s == A_RING) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
  } else {
    // Epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 and one half of
    // the tile's columns. The tensor core's FP32 accumulation rounds toward
    // zero; keeping each chunk short and adding the chunks here with
    // round-to-nearest keeps the product as accurate as FP32 arithmetic.
    QFX_SETMAXNREG_INC(176);
    constexpr int COLS = BN / 2;
    const int q = warp % 4;
    const int part = (warp - 4) / 4;
    const int row = q * 32 + lane;
    const std::int8_t* exps = reinterpret_cast<const std::int8_t*>(smem + OFF_EXP);
    std::uint8_t* staging = smem + OFF_STAGING + (warp - 4) * 2 * SLOT;
    int* sc_row = reinterpret_cast<int*>(smem + OFF_SCALE) + (warp - 4) * COLS;
    const float beta = debias_beta<KIND_FP16>(err, CHUNK, kblocks);
    const float2 beta2 = make_float2(beta, beta);
    const int per_block = CHUNK == 1 ? 2 : 1;  // chunks of a whole block
    const int chunks = (kblocks + CHUNK - 1) / CHUNK;
    int c = 0, x = 0;
    bool ok = true;
    for (int t = first; t < total && ok; t += stride) {
      int mt, nt, batch;
      tile_of(t, mt, nt, batch);
      const int m0 = mt * BM, n0 = nt * BN + part * COLS;
      const int ncols = n - n0;
      // Exponents of the lane's columns, fetched before the drain.
      const int* eb = exp_b + std::uint64_t(batch) * n + n0;
      const int eb0 = lane < ncols ? eb[lane] : 0;
      const int eb1 = 32 + lane < ncols ? eb[32 + lane] : eb0;
      float2 re[COLS / 2], im[COLS / 2];  // columns 2 j, 2 j + 1
#pragma unroll
      for (int j = 0; j < COLS / 2; ++j) re[j] = im[j] = make_float2(0.f, 0.f);
      // The sums are kept times 2^eref (and the column's 2^eb): a chunk of a
      // block with exponent e is added times 2^(eref - e) <= 1. eref starts
      // two below the first block's exponent and drops, rescaling the sums,
      // only when a later block is more than four times larger.
      int eref = 0;
      for (int cc = 0; cc < chunks; ++cc, ++c) {
        const int buf = c & 1;
        if (!__all_sync(0xffffffffu, wait(&acc_full[buf], (c >> 1) & 1, 3))) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const int e = exps[x * BM + row];
        if (cc % per_block == per_block - 1 || cc == chunks - 1) {
          if (++x == EXP_RING) x = 0;
        }
        if (cc == 0) {
          eref = e - 2;
        } else if (__any_sync(0xffffffffu, e < eref)) {
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
        const std::uint32_t base = tmem + (std::uint32_t(q * 32) << 16) + buf * 2 * BN + part * COLS;
#pragma unroll
        for (int j0 = 0; j0 < COLS; j0 += 16) {
          std::uint32_t vr[16], vi[16];
          TMEM_LD16(base + j0, vr);
          TMEM_LD16(base + BN + j0, vi);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int p = j0 / 2 + j;
            re[p] = fma2(make_float2(__uint_as_float(vr[2 * j]), __uint_as_float(vr[2 * j + 1])), sa2, re[p]);
            im[p] = fma2(make_float2(__uint_as_float(vi[2 * j]), __uint_as_float(vi[2 * j + 1])), sa2, im[p]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);
      }
      if (!ok) break;
      // The MMA issuer already works on the next tiles. The columns'
      // exponents go through 64 words of the warp's own shared memory, from
      // where four at a time are read as one broadcast.
      __syncwarp();
      sc_row[lane] = eb0 << 23;
      sc_row[32 + lane] = eb1 << 23;
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
        sc_row[lane] = 0;
        sc_row[32 + lane] = 0;
        __syncwarp();
      }
#pragma unroll
      for (int j = 0; j < COLS / 2; ++j) {
        re[j] = fma2(re[j], beta2, re[j]);
        im[j] = fma2(im[j], beta2, im[j]);
      }
      float2* cb = C + std::uint64_t(batch) * ac_stride;
      // Four boxes of 32 rows x 16 complex, two slots in turn. (Boxes of 8
      // columns: twice the fences and barriers, a tile's store took 7200
      // cycles. A thread storing its own row piece in 32-byte sectors,
      // without shared memory, 9400.)
#pragma unroll
      for (int j0 = 0; j0 < COLS; j0 += 16) {
        std::uint8_t* slot = staging + ((j0 / 16) & 1) * SLOT;
        if (tma_c) {
          if (lane == 0) bulk_wait_read1();
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
    // Release TMEM only after every MMA this CTA issued has completed; the
    // wait is immediate unless the pipeline was abandoned.
    const unsigned long long t0 = now_ns();
    while (!mbar_test(mma_done, 0) && now_ns() - t0 < WAIT_NS) {
    }
    asm volatile("tcgen05.fence::after_thread_sync;");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
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
  g.aligned = aligned ? 1 : 0;
  g.pairs = 1;
  g.copies_real = 32;
  // Copy u = 16 row + pair; its unit of the block is u with the low three
  // bits XORed with the row's, so that a quarter-warp of rows reading the
  // same values hits eight different units.
  auto at = [](std::uint32_t u) { return (u ^ ((u >> 4) & 7u)) << 4; };
  for (int b = 0; b < 6; ++b) {
    g.lane_src[b] = b < 4 ? std::uint64_t(2) << b : std::uint64_t(k) << (b - 4);
    g.lane_dst[b] = at(1u << b);
  }
  for (std::uint32_t i = 0; i < 32; ++i) {
    g.copy_src[i] = std::uint64_t(4) * i * k;
    g.copy_dst[i] = at(64u * i);
    g.value_at[i] = at(i >> 1) | ((i & 1u) << 3);
  }
  for (int b = 0; b < 7; ++b) g.row_at[b] = at(16u << b);
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
  g->aligned = 1;
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
      for (int u = 0; u < 2048; ++u) {
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

std::size_t tc_direct_workspace_elems(std::size_t n, std::size_t k) {
  return 2 * n * ((k + 15) / 16 * 16) + 2 * n;  // B's planes, exponents and largest components
}

void launch_cgemm_fp16x3_direct(const float2* A, const AGather& gather, const float2* B, BLayout b_layout, float2* C,
                                std::size_t m, std::size_t n, std::size_t k, std::uint64_t ac_stride,
                                std::uint64_t b_stride, int batch, float* workspace, int* err, const TcConfig& cfg,
                                cudaStream_t s) {
  if (!tc_runs(m, n, k)) throw std::string("ERROR (qflex_gb300: tensor cores) --> shape not eligible");
  if (cfg.chunk < 1 || cfg.chunk > 2)
    throw std::string("ERROR (qflex_gb300: tensor cores) --> the direct product takes chunks of 1 or 2 k-steps");
  static std::once_flag attr;
  std::call_once(attr, [] {
    check(cudaFuncSetAttribute(cgemm_fp16x3_direct_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM),
          "cudaFuncSetAttribute");
  });
  const std::size_t kpad = (k + 15) / 16 * 16;
  __half* pb = reinterpret_cast<__half*>(workspace);
  int* eb = reinterpret_cast<int*>(pb + 4 * n * kpad * (std::size_t)batch);
  std::uint32_t* top = reinterpret_cast<std::uint32_t*>(eb + n * (std::size_t)batch);
  launch_split(KIND_FP16, 4, {pb, nullptr, eb, top}, B, n, k, b_stride, batch, b_layout == BLayout::kn, s);
  const CUtensorMap mb = plane_map_f16(pb, n, kpad, batch, BN, 64);
  CUtensorMap mc;
  const int tma_c = output_map(C, m, n, ac_stride, batch, &mc) ? 1 : 0;
  const std::size_t tiles = ((m + BM - 1) / BM) * ((n + BN - 1) / BN) * (std::size_t)batch;
  cgemm_fp16x3_direct_kernel<<<persistent_grid(tiles), THREADS, SMEM, s>>>(
      mb, mc, gather, A, C, tma_c, (int)m, (int)n, (int)k, batch, ac_stride, err, cfg.chunk, eb);
  check(cudaGetLastError(), "cgemm_fp16x3_direct");
}

}  // namespace qfx
