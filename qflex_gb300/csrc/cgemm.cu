// Complex64 products C = A * B (row-major) on the FP32 pipes of sm_103a.
//
// One kernel body for all tile shapes: BM x BN outputs per tile, TM x TN per
// thread, k in steps of BK. Blocks are persistent over the tiles (and the
// batch): the k-steps of a block's tiles form one sequence, whose operands
// cp.async brings into a ring of STAGES buffers, so a tile's products run
// while the next tile's operands are on their way. That matters most for the
// long, narrow products of the contractions (2^20 x 16 x 16), where a tile is
// two k-steps.
//
// Bound by the FP32 pipes where k is long (scalar FMAs reach about 61 TFLOP/s
// from registers alone at these clocks), by HBM at small k. Measured against
// one tile per block with operands staged through registers:
//   (2048, 2048, 2048)       1541 -> 1460 us (47 TFLOP/s)
//   (32768, 64, 64) x 16      462 ->  342 us (50 TFLOP/s)
//   (32768, 64, 8) x 16       221 ->   71 us
//   (32768, 8, 64) x 16       113 ->   72 us
//   (2^20, 16, 16)             75 ->   63 us (4.2 TB/s)
//   (2^20, 16, 256)           847 ->  747 us
// Copies of 16 bytes are worth 10 to 25 % of that against copies of 8; k-steps
// of 8 keep four blocks of the narrow tiles on an SM. Two-lane FMAs
// (fma.rn.f32x2) have the same rate from registers and lose more to packing
// their operands: 2049 us at 2048^3.
//
// Where the persistent blocks' rounds of tiles leave half of the chip idle, or
// rows do not start on 16 bytes, one tile per block is faster: those products
// run as they did before (cgemm_staged_kernel, staged_is_faster).
//
// Sums run over k in ascending order with four FMAs per complex term; products
// of few tiles may sum runs of k so and then add the runs in 64 bits.
//
// A is read as it lies or, for the tensors of a contraction, through the digit
// permutation that would have laid it out row-major (TileGather): then lanes
// follow the source's order and each copy goes to its place in the tile.
#include <algorithm>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "kernels.h"
#include "per_device.h"

namespace qfx {

namespace {

__device__ __forceinline__ void cfma(float2& c, float2 a, float2 b) {
  c.x = fmaf(a.x, b.x, c.x);
  c.x = fmaf(-a.y, b.y, c.x);
  c.y = fmaf(a.x, b.y, c.y);
  c.y = fmaf(a.y, b.x, c.y);
}
__device__ __forceinline__ void copy8(float2* dst, const float2* src, bool real) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                   static_cast<std::uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(real ? 8u : 0u)
               : "memory");
}

__device__ __forceinline__ void copy16(float2* dst, const float2* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   static_cast<std::uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy16(float2* dst, const float2* src, bool real) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   static_cast<std::uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(real ? 16u : 0u)
               : "memory");
}

// Row stride of a staged A tile in elements: 16 bytes more than its values,
// so that the rows a quarter-warp reads start in different banks.
constexpr int a_row(int BK) { return BK + 2; }

// What one variant of the kernel takes besides the matrices, no more, since a
// larger argument slows the launch: a gather, the split of k (`splits` runs of
// `terms`, whose sums go to `partial` as [entry][split][m][n]), or the
// condition under which it does anything.
struct SplitK {
  float2* partial;
  int splits, terms;
};
enum Variant { PLAIN, GATHERED, SPLIT };
template <int VARIANT>
using Extra = std::conditional_t<VARIANT == GATHERED, TileGather, std::conditional_t<VARIANT == SPLIT, SplitK, OnlyIf>>;

template <int BM, int BN, int BK, int TM, int TN, int STAGES, int VARIANT>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
    cgemm_kernel(const float2* __restrict__ A, const float2* __restrict__ B, float2* __restrict__ C, int m, int n,
                 int k, std::uint64_t batch_stride, int tiles_m, long long tiles, int pairs,
                 const __grid_constant__ Extra<VARIANT> g) {
  constexpr bool GATHER = VARIANT == GATHERED;
  constexpr int NT = (BM / TM) * (BN / TN);
  constexpr int TX = BN / TN, TY = BM / TM;
  constexpr int LA = BM * BK / NT, LB = (BK * BN + NT - 1) / NT;
  constexpr int AR = a_row(BK);
  constexpr int A_ELEMS = BM * AR, STAGE = A_ELEMS + BK * BN;
  static_assert(LA * NT == BM * BK && BK % 2 == 0 && TN % 2 == 0, "tile / threads mismatch");
  extern __shared__ __align__(16) float2 ring[];
  if constexpr (VARIANT == PLAIN)
    if (g.flag) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      if (*reinterpret_cast<const volatile int*>(g.flag) != g.value) return;
    }
  const int t = threadIdx.x;
  const int tx = t % TX, ty = t / TX;
  int ktiles = k > 0 ? (k + BK - 1) / BK : 1;  // no terms: one k-step of zeros
  if constexpr (VARIANT == SPLIT) ktiles = g.terms / BK;
  const int tiles_n = (n + BN - 1) / BN;
  const long long mine = (long long)blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  const long long steps = mine * ktiles;
  // Consecutive tiles share their rows of A. A split product counts the runs
  // of k like batch entries: `at` is the run's number.
  const std::uint64_t entry_stride = VARIANT == SPLIT ? 1 : batch_stride;
  auto place = [&](long long tile, unsigned& mt, unsigned& nt, std::uint64_t& at) {
    if (tiles <= 0xffffffffll) {  // 32-bit divisions are much the shorter
      const unsigned r = unsigned(tile) / unsigned(tiles_n);
      nt = unsigned(tile) % unsigned(tiles_n);
      mt = r % unsigned(tiles_m);
      at = std::uint64_t(r / unsigned(tiles_m)) * entry_stride;
    } else {
      const long long r = tile / tiles_n;
      nt = unsigned(tile % tiles_n);
      mt = unsigned(r % tiles_m);
      at = std::uint64_t(r / tiles_m) * entry_stride;
    }
  };

  const float2* lane_src = A;
  int lane_dst = 0;
  if constexpr (GATHER) {
    for (int b = 0; (1 << b) < NT; ++b)
      if ((t >> b) & 1) {
        lane_src += g.lane_src[b];
        lane_dst += g.lane_dst[b];
      }
  }

  // Loader position: k-step lk of the block's tile lt.
  long long lt = blockIdx.x;
  int lk = 0;
  auto load = [&](int slot) {
    float2* As = ring + slot * STAGE;
    float2* Bs = As + A_ELEMS;
    unsigned mt, nt;
    std::uint64_t at;
    place(lt, mt, nt, at);
    int k0 = lk * BK;
    if constexpr (VARIANT == SPLIT) {
      const unsigned run = unsigned(at);
      k0 += int(run % unsigned(g.splits)) * g.terms;
      at = std::uint64_t(run / unsigned(g.splits)) * batch_stride;
    }
    if constexpr (GATHER) {
      const float2* src = lane_src + at;
      for (int b = 0; b < TileGather::kBits && (mt >> b); ++b)
        if ((mt >> b) & 1) src += g.tile_src[b];
      for (int b = 0; b < TileGather::kBits && (lk >> b); ++b)
        if ((lk >> b) & 1) src += g.step_src[b];
#pragma unroll
      for (int i = 0; i < LA; ++i) copy8(As + lane_dst + g.copy_dst[i], src + g.copy_src[i], true);
    } else if ((pairs & 2) && (mt + 1) * BM <= unsigned(m) && k0 + BK <= k) {
      // Inside the matrix, rows on 16 bytes: pairs of values.
      constexpr int P = BK / 2, LP = (BM * P + NT - 1) / NT, ROWS = NT / P;
      static_assert(NT % P == 0, "pairs of a row of A / threads");
      const int r = t / P, c = 2 * (t % P);
      const float2* src = A + at + std::uint64_t(mt * BM + r) * k + k0 + c;
#pragma unroll
      for (int i = 0; i < LP; ++i) {
        if (BM * P % NT == 0 || r + i * ROWS < BM) copy16(As + (r + i * ROWS) * AR + c, src);
        src += std::uint64_t(ROWS) * k;
      }
    } else if ((pairs & 2) && k0 + BK <= k) {
      // Rows on 16 bytes, some of them past the last.
      constexpr int P = BK / 2, LP = (BM * P + NT - 1) / NT, ROWS = NT / P;
      const int r = t / P, c = 2 * (t % P), rows = m - int(mt * BM) - r;
      const float2* src = A + at + std::uint64_t(mt * BM + r) * k + k0 + c;
#pragma unroll
      for (int i = 0; i < LP; ++i) {
        if (BM * P % NT == 0 || r + i * ROWS < BM)
          copy16(As + (r + i * ROWS) * AR + c, i * ROWS < rows ? src : A, i * ROWS < rows);
        src += std::uint64_t(ROWS) * k;
      }
    } else if (k0 + BK <= k) {
      // Rows on 8 bytes.
      static_assert(NT % BK == 0, "values of a row of A / threads");
      const int r = t / BK, c = t % BK, rows = m - int(mt * BM) - r;
      const float2* src = A + at + std::uint64_t(mt * BM + r) * k + k0 + c;
#pragma unroll
      for (int i = 0; i < LA; ++i) {
        const bool real = i * (NT / BK) < rows;
        copy8(As + (r + i * (NT / BK)) * AR + c, real ? src : A, real);
        src += std::uint64_t(NT / BK) * k;
      }
    } else {
#pragma unroll
      for (int i = 0; i < LA; ++i) {
        const int idx = t + i * NT;
        const int r = idx / BK, c = idx % BK;
        const unsigned row = mt * BM + r;
        const bool real = row < unsigned(m) && k0 + c < k;
        copy8(As + r * AR + c, real ? A + at + std::uint64_t(row) * k + k0 + c : A, real);
      }
    }
    if ((pairs & 4) && (nt + 1) * BN <= unsigned(n) && k0 + BK <= k) {
      constexpr int P = BN / 2, LP = (BK * P + NT - 1) / NT, ROWS = NT / P;
      static_assert(NT % P == 0, "pairs of a row of B / threads");
      const int r = t / P, c = 2 * (t % P);
      const float2* src = B + at + std::uint64_t(k0 + r) * n + nt * BN + c;
#pragma unroll
      for (int i = 0; i < LP; ++i) {
        if (BK * P % NT == 0 || r + i * ROWS < BK) copy16(Bs + (r + i * ROWS) * BN + c, src);
        src += std::uint64_t(ROWS) * n;
      }
    } else {
#pragma unroll
      for (int i = 0; i < LB; ++i) {
        const int idx = t + i * NT;
        if (BK * BN % NT != 0 && idx >= BK * BN) break;
        const int r = idx / BN, c = idx % BN;
        const unsigned col = nt * BN + c;
        const bool real = k0 + r < k && col < unsigned(n);
        copy8(Bs + r * BN + c, real ? B + at + std::uint64_t(k0 + r) * n + col : B, real);
      }
    }
    if (++lk == ktiles) {
      lk = 0;
      lt += gridDim.x;
    }
  };

  float2 acc[TM][TN];
  long long loaded = 0, tile = blockIdx.x;
  int ks = 0, slot = 0, load_slot = 0;
  for (; loaded < STAGES - 1; ++loaded) {
    if (loaded < steps) load(load_slot);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (++load_slot == STAGES) load_slot = 0;
  }
  for (long long s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // step s has landed; everybody is done with the slot loaded next
    if (loaded < steps) load(load_slot);
    ++loaded;
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (++load_slot == STAGES) load_slot = 0;

    if (ks == 0) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
    }
    // Thread (tx, ty): rows ty + TY i, columns 2 tx, 2 tx + 1 of every 2 TX.
    const float2* As = ring + slot * STAGE + ty * AR;
    const float2* Bs = ring + slot * STAGE + A_ELEMS + 2 * tx;
#pragma unroll 4
    for (int kk = 0; kk < BK; kk += 2) {
      float4 a[TM];  // values kk and kk + 1
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(As + i * TY * AR + kk);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float2 b[TN];
#pragma unroll
        for (int j = 0; j < TN; j += 2) {
          const float4 v = *reinterpret_cast<const float4*>(Bs + (kk + h) * BN + j * TX);
          b[j] = make_float2(v.x, v.y);
          b[j + 1] = make_float2(v.z, v.w);
        }
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const float2 x = h ? make_float2(a[i].z, a[i].w) : make_float2(a[i].x, a[i].y);
#pragma unroll
          for (int j = 0; j < TN; ++j) cfma(acc[i][j], x, b[j]);
        }
      }
    }
    if (++slot == STAGES) slot = 0;
    if (++ks == ktiles) {
      ks = 0;
      unsigned mt, nt;
      std::uint64_t at;
      place(tile, mt, nt, at);
      tile += gridDim.x;
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const unsigned r = mt * BM + ty + i * TY;
        if (r >= unsigned(m)) continue;
        float2* c = C + at + std::uint64_t(r) * n;
        if constexpr (VARIANT == SPLIT) c = g.partial + (at * std::uint64_t(m) + r) * n;
#pragma unroll
        for (int j = 0; j < TN; j += 2) {
          const unsigned col = nt * BN + 2 * tx + j * TX;
          const float2 v0 = acc[i][j], v1 = acc[i][j + 1];
          if ((pairs & 1) && col + 1 < unsigned(n)) {
            *reinterpret_cast<float4*>(c + col) = make_float4(v0.x, v0.y, v1.x, v1.y);
          } else {
            if (col < unsigned(n)) c[col] = v0;
            if (col + 1 < unsigned(n)) c[col + 1] = v1;
          }
        }
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// One tile per block, operands staged through registers: the next k-step's
// are loaded while one is multiplied. A block of 128 x 64 has an SM to itself
// (164 registers), where it is as fast as two persistent ones, so its rounds
// of tiles are half as long; and rows that do not start on 16 bytes cost it
// nothing, where the persistent blocks' copies of 8 bytes cost them 3 to 10 %.
// The rule is staged_is_faster. The sums are the same.
template <int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
    cgemm_staged_kernel(const float2* __restrict__ A, const float2* __restrict__ B, float2* __restrict__ C, int m,
                        int n, int k, std::uint64_t batch_stride) {
  constexpr int NT = (BM / TM) * (BN / TN);
  constexpr int TX = BN / TN;
  constexpr int LA = BM * BK / NT, LB = BK * BN / NT;
  static_assert(LA * NT == BM * BK && LB * NT == BK * BN, "tile / threads mismatch");
  __shared__ __align__(16) float2 As[BK][BM + 2];
  __shared__ __align__(16) float2 Bs[BK][BN + 2];
  const std::uint64_t at = std::uint64_t(blockIdx.z) * batch_stride;
  A += at;
  B += at;
  C += at;
  const int tiles_m = (m + BM - 1) / BM;
  const int m0 = int(blockIdx.x % tiles_m) * BM, n0 = int(blockIdx.x / tiles_m) * BN;
  const int t = threadIdx.x, tx = t % TX, ty = t / TX;
  float2 acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
  float2 ra[LA], rb[LB];
  auto load = [&](int k0) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int r = m0 + (t + i * NT) / BK, c = k0 + (t + i * NT) % BK;
      ra[i] = r < m && c < k ? A[std::size_t(r) * k + c] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < LB; ++i) {
      const int r = k0 + (t + i * NT) / BN, c = n0 + (t + i * NT) % BN;
      rb[i] = r < k && c < n ? B[std::size_t(r) * n + c] : make_float2(0.f, 0.f);
    }
  };
  auto store = [&] {
#pragma unroll
    for (int i = 0; i < LA; ++i) As[(t + i * NT) % BK][(t + i * NT) / BK] = ra[i];
#pragma unroll
    for (int i = 0; i < LB; ++i) Bs[(t + i * NT) / BN][(t + i * NT) % BN] = rb[i];
  };
  const int ktiles = (k + BK - 1) / BK;
  load(0);
  store();
  __syncthreads();
  for (int kt = 0; kt < ktiles; ++kt) {
    const bool more = kt + 1 < ktiles;
    if (more) load((kt + 1) * BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float2 a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Bs[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) cfma(acc[i][j], a[i], b[j]);
    }
    __syncthreads();
    if (more) {
      store();
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = m0 + ty * TM + i;
    if (r >= m) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int c = n0 + tx * TN + j;
      if (c < n) C[std::size_t(r) * n + c] = acc[i][j];
    }
  }
}

// Adds the sums of a split product's runs: blocks of 32 elements of C, whose
// eight warps take every eighth run (one thread for all runs of an element
// took 15 us at 64).
__global__ void __launch_bounds__(256) split_finish_kernel(const float2* __restrict__ partial, float2* __restrict__ C,
                                                           std::uint64_t outputs, int splits,
                                                           std::uint64_t batch_stride) {
  __shared__ double2 part[8][32];
  const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
  const std::uint64_t at = std::uint64_t(blockIdx.x) * 32 + lane;
  double2 sum = make_double2(0, 0);
  if (at < outputs) {
    const float2* p = partial + blockIdx.y * outputs * splits + at;
#pragma unroll 8
    for (int q = w; q < splits; q += 8) {
      const float2 v = p[q * outputs];
      sum.x += double(v.x);
      sum.y += double(v.y);
    }
  }
  part[w][lane] = sum;
  __syncthreads();
  if (w || at >= outputs) return;
#pragma unroll
  for (int q = 1; q < 8; ++q) {
    sum.x += part[q][lane].x;
    sum.y += part[q][lane].y;
  }
  C[blockIdx.y * batch_stride + at] = make_float2(float(sum.x), float(sum.y));
}

// Sets *flag to `value` when an element of a product is no finite number.
__global__ void __launch_bounds__(256) flag_not_finite_kernel(const float2* __restrict__ C, std::uint64_t outputs,
                                                              std::uint64_t batch_stride, int* flag, int value) {
  C += blockIdx.y * batch_stride;
  float zero = 0.f;  // NaN once an infinity or NaN was met
  for (std::uint64_t i = std::uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < outputs;
       i += std::uint64_t(gridDim.x) * blockDim.x) {
    const float2 v = C[i];
    zero = fmaf(v.x, 0.f, fmaf(v.y, 0.f, zero));
  }
  if (zero != 0.f) atomicExch(flag, value);
}

bool is_conditional(const OnlyIf& c) { return c.flag != nullptr; }
template <typename T>
bool is_conditional(const T&) {
  return false;
}

struct Tile {
  int bm, bn, bk, threads;
};
template <int BM, int BN, int BK, int TM, int TN, int STAGES>
struct Shape {
  static constexpr int nt = (BM / TM) * (BN / TN);
  static constexpr Tile tile{BM, BN, BK, nt};
  static constexpr int smem = STAGES * (BM * a_row(BK) + BK * BN) * (int)sizeof(float2);

  template <int VARIANT>
  static void run(const float2* A, const float2* B, float2* C, std::size_t m, std::size_t n, std::size_t k,
                  std::uint64_t stride, int batch, const Extra<VARIANT>& g, cudaStream_t s) {
    auto* kernel = cgemm_kernel<BM, BN, BK, TM, TN, STAGES, VARIANT>;
    // Blocks that are resident at once on the current device.
    static PerDevice blocks;
    const int resident = blocks([&] {
      raise_smem_limit(kernel, smem);
      int dev = 0, sms = 152, per = 1;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, nt, smem);
      return sms * std::max(per, 1);
    });
    const long long tiles_m = (long long)((m + BM - 1) / BM);
    long long tiles = tiles_m * (long long)((n + BN - 1) / BN) * batch;
    if constexpr (VARIANT == SPLIT) tiles *= g.splits;
    // Which of C's, A's and B's rows start on 16 bytes (bits 0, 1, 2).
    const bool even = batch == 1 || stride % 2 == 0;
    auto rows16 = [&](const float2* p, std::size_t row) {
      return even && row % 2 == 0 && (reinterpret_cast<std::uintptr_t>(p) & 15) == 0;
    };
    const bool c16 = VARIANT == SPLIT ? n % 2 == 0 : rows16(C, n);
    const int pairs = (c16 ? 1 : 0) | (rows16(A, k) ? 2 : 0) | (rows16(B, n) ? 4 : 0);
    const unsigned grid = (unsigned)std::min<long long>(tiles, resident);
    cudaError_t e;
    if (VARIANT == PLAIN && is_conditional(g)) {
      // Launched while the kernel before it ends, for which it waits.
      cudaLaunchConfig_t lc = {};
      lc.gridDim = dim3(grid, 1, 1);
      lc.blockDim = dim3(nt, 1, 1);
      lc.dynamicSmemBytes = smem;
      lc.stream = s;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[0].val.programmaticStreamSerializationAllowed = 1;
      lc.attrs = at;
      lc.numAttrs = 1;
      e = cudaLaunchKernelEx(&lc, kernel, A, B, C, (int)m, (int)n, (int)k, stride, (int)tiles_m, tiles, pairs, g);
    } else {
      kernel<<<grid, nt, smem, s>>>(A, B, C, (int)m, (int)n, (int)k, stride, (int)tiles_m, tiles, pairs, g);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) throw std::string("ERROR (qflex_gb300: launch cgemm) --> ") + cudaGetErrorString(e);
  }
  static void launch(const float2* A, const float2* B, float2* C, std::size_t m, std::size_t n, std::size_t k,
                     std::uint64_t stride, int batch, const TileGather* g, OnlyIf only_if, cudaStream_t s) {
    if (g)
      run<GATHERED>(A, B, C, m, n, k, stride, batch, *g, s);
    else
      run<PLAIN>(A, B, C, m, n, k, stride, batch, only_if, s);
  }
};

// Calls f with the shape that a product takes: the narrowest that holds its
// columns (or rows), so that no more than half of a tile's outputs are padding
// from 5 columns on; k-steps of 16 where there are 16 terms and the tile is
// wide enough to keep two blocks on an SM.
template <typename F>
auto with_shape(std::size_t m, std::size_t n, std::size_t k, F&& f) {
  if (n <= 8) return f(Shape<256, 8, 8, 4, 4, 3>{});
  if (n <= 16) return f(Shape<256, 16, 8, 8, 4, 2>{});
  if (n <= 32) return f(Shape<128, 32, 8, 8, 4, 3>{});
  if (m <= 32) return f(Shape<16, 256, 8, 4, 8, 3>{});
  if (m <= 64 && n >= 128 && k > 8) return f(Shape<64, 128, 16, 8, 4, 3>{});  // (50, 1642, 1993) x 7 804 -> 438 us
  if (k <= 8) return f(Shape<128, 64, 8, 8, 4, 3>{});
  return f(Shape<128, 64, 16, 8, 4, 3>{});
}

// Few tiles: a product is then as long as one tile's chain of k-steps. Small
// tiles and six steps in flight shorten the chain, and where they are fewer
// than the SMs hold (two each), so does splitting k into runs of 64 or more.
// The shapes above against these: (16, 16, 32) 10 and 4 us, (256, 16, 64) 19
// and 5.5, (512, 512, 512) 104 and 42; with runs (256, 16, 512) 80 and 9,
// (16, 16, 4096) 500 and 12. Up to 101 tiles with 512 terms take runs too, in
// the shapes above: (1586, 161, 3221) 686 and 342, (1000, 512, 1000) 202 and
// 140. Calls f with the shape of such a product; false for other products.
template <typename F>
bool with_few_tiles(std::size_t m, std::size_t n, std::size_t k, int batch, bool scratch, F&& f) {
  const Tile tile = with_shape(m, n, k, [](auto shape) { return decltype(shape)::tile; });
  const std::size_t tiles = ((m + tile.bm - 1) / tile.bm) * ((n + tile.bn - 1) / tile.bn) * (std::size_t)batch;
  const bool runs = scratch && tiles <= 101 && k >= 512 && 3 * m * n * (std::size_t)batch <= kSkinnyScratchElems;
  if (!tiles || (tiles > 38 && !runs)) return false;
  if (tiles > 38)
    with_shape(m, n, k, [&](auto shape) {
      f(shape);
      return 0;
    });
  else
    n <= 8 ? f(Shape<64, 8, 16, 2, 2, 6>{}) : f(Shape<32, 32, 16, 2, 2, 6>{});
  return true;
}

// The runs of k (and their terms) in which the tiles of shape S sum a product
// that has scratch: 0 for none.
template <typename S>
int runs_of(std::size_t m, std::size_t n, std::size_t k, int batch, std::size_t* terms) {
  constexpr Tile t = S::tile;
  const std::size_t own = ((m + t.bm - 1) / t.bm) * ((n + t.bn - 1) / t.bn) * (std::size_t)batch;
  std::size_t splits = std::min<std::size_t>(304 / own, k / 64);
  splits = std::min<std::size_t>(splits, kSkinnyScratchElems / (m * n * (std::size_t)batch));
  if (splits < 3) return 0;
  *terms = ((k + splits - 1) / splits + t.bk - 1) / t.bk * t.bk;
  return (int)((k + *terms - 1) / *terms);
}

// Whether one tile per block is faster, for products of `tiles` tiles of the
// usual shape (and no gather).
// Tiles of 128 x 64, by estimates in us from the rounds of tiles, one on an SM
// (rounds) or two (pairs; a last round of up to 112 tiles finds an SM for each,
// from there on some SMs get two), and the padded terms, fitted to 1172 products
// of 39 to 3000 tiles (2 to 4 % standard deviation). 161 of those take over 2 %
// more in persistent blocks than in one tile per block, and 15 as chosen here;
// most is lost between 417 and 456 tiles: (5573, 290, 1392) x 2 838 us in one
// tile per block, 1049 in persistent ones.
// Tiles of 256 x 16 with rows on 8 bytes: up to 304 of them by how many 64-row
// tiles an SM gets, (74497, 11, 1713) 455 and 664, (10143, 11, 585) x 4 160 and
// 136; more where steps of 16 terms pad no more than those of 8, (157583, 13,
// 27) x 4 83 and 87, (157583, 13, 9) x 7 91 and 81, or terms are many.
bool staged_is_faster(const Tile& tile, std::size_t tiles, std::size_t m, std::size_t n, std::size_t k, int batch) {
  if (tile.bm == 256 && tile.bn == 16) {
    if (k % 2 == 0 || k < 25) return false;
    const std::size_t per_sm = ((m + 63) / 64 * (std::size_t)batch + 151) / 152;
    return tiles <= 152 ? per_sm >= 4 : tiles <= 304 ? per_sm >= 6 : k % 16 > 8 || k >= 150;
  }
  if (tile.bm != 128 || tile.bn != 64 || tile.bk != 16) return false;
  const double rounds = double((tiles + 151) / 152), terms = double((k + 15) / 16 * 16);
  const double staged = 6.9 + rounds * (4.1 + 0.1884 * terms);
  if (tiles <= 152) {
    const double q = m > 64 && k >= 128 ? double((k + 31) / 32 * 32) : terms;  // steps of 32, see below
    return staged < (k % 2 ? 7.9 + 0.2104 * q : n % 2 ? 9.4 + 0.1937 * q : 8.2 + 0.1884 * q);
  }
  const std::size_t last = tiles % 304;
  const bool spread = tiles > 304 && last > 0 && last <= 112;
  const double pairs = double(tiles / 304) + (last > 0 && !spread), alone = spread;
  return staged < (k % 2   ? 6.7 + pairs * (3.0 + 0.3847 * terms) + alone * (1.4 + 0.194 * terms)
                   : n % 2 ? 6.7 + pairs * (3.2 + 0.38 * terms) + alone * (1.6 + 0.195 * terms)
                           : 6.4 + pairs * (1.8 + 0.3702 * terms) + alone * (1.4 + 0.1951 * terms));
}

template <int BM, int BN, int BK, int TM, int TN>
void run_staged(const float2* A, const float2* B, float2* C, std::size_t m, std::size_t n, std::size_t k,
                std::uint64_t stride, int batch, cudaStream_t s) {
  dim3 grid((unsigned)(((m + BM - 1) / BM) * ((n + BN - 1) / BN)), 1, (unsigned)batch);
  cgemm_staged_kernel<BM, BN, BK, TM, TN><<<grid, (BM / TM) * (BN / TN), 0, s>>>(A, B, C, (int)m, (int)n, (int)k, stride);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::string("ERROR (qflex_gb300: launch cgemm_staged) --> ") + cudaGetErrorString(e);
}

}  // namespace

int tiled_splits(std::size_t m, std::size_t n, std::size_t k, int batch) {
  int splits = 0;
  with_few_tiles(m, n, k, batch, true, [&](auto shape) {
    std::size_t terms = 0;
    splits = runs_of<decltype(shape)>(m, n, k, batch, &terms);
  });
  return splits;
}

void launch_flag_not_finite(const float2* C, std::size_t outputs, std::uint64_t batch_stride, int batch, int* flag,
                            int value, cudaStream_t s) {
  dim3 grid((unsigned)std::min<std::size_t>((outputs + 1023) / 1024, 152 * 8), (unsigned)batch);
  flag_not_finite_kernel<<<grid, 256, 0, s>>>(C, outputs, batch_stride, flag, value);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::string("ERROR (qflex_gb300: launch flag_not_finite) --> ") + cudaGetErrorString(e);
}

bool make_tile_gather(int nbits, const std::uint8_t* perm, std::size_t m, std::size_t n, std::size_t k, TileGather* g) {
  const Tile tile = with_shape(m, n, k, [](auto shape) { return decltype(shape)::tile; });
  int kl = 0, ml = 0, bk = 0, bm = 0, lanes = 0;
  while ((std::size_t(1) << kl) < k) ++kl;
  while ((std::size_t(1) << ml) < m) ++ml;
  while ((1 << bk) < tile.bk) ++bk;
  while ((1 << bm) < tile.bm) ++bm;
  while ((1 << lanes) < tile.threads) ++lanes;
  if ((std::size_t(1) << kl) != k || (std::size_t(1) << ml) != m || kl + ml != nbits || nbits > 31 || kl < bk ||
      ml < bm)
    return false;
  std::memset(g, 0, sizeof(*g));
  int n_e = 0;
  for (int p = 0; p < nbits; ++p) {
    const int d = perm[p];
    const bool value = d < bk, row = d >= kl && d < kl + bm;
    if (!value && !row) {
      // The source's three lowest digits lie in the tile: eight lanes read 64
      // consecutive bytes.
      if (p < 3) return false;
      if (d < kl)
        g->step_src[d - bk] = std::uint64_t(1) << p;
      else
        g->tile_src[d - kl - bm] = std::uint64_t(1) << p;
      continue;
    }
    const std::uint32_t dst = value ? 1u << d : (std::uint32_t)a_row(tile.bk) << (d - kl);
    if (n_e < lanes) {
      g->lane_src[n_e] = std::uint64_t(1) << p;
      g->lane_dst[n_e] = dst;
    } else {
      const int b = n_e - lanes;
      for (int i = 0; i < TileGather::kCopies; ++i)
        if ((i >> b) & 1) {
          g->copy_src[i] += std::uint64_t(1) << p;
          g->copy_dst[i] += dst;
        }
    }
    ++n_e;
  }
  return true;
}

void tile_gather_on_host(const TileGather& g, std::size_t m, std::size_t n, std::size_t k, const float2* src,
                         float2* dst) {
  const Tile tile = with_shape(m, n, k, [](auto shape) { return decltype(shape)::tile; });
  const int ar = a_row(tile.bk), copies = tile.bm * tile.bk / tile.threads;
  std::vector<float2> staged(std::size_t(tile.bm) * ar);
  for (std::size_t mt = 0; mt < m / tile.bm; ++mt)
    for (std::size_t ks = 0; ks < k / tile.bk; ++ks) {
      std::uint64_t base = 0;
      for (int b = 0; b < TileGather::kBits; ++b) {
        if ((mt >> b) & 1) base += g.tile_src[b];
        if ((ks >> b) & 1) base += g.step_src[b];
      }
      for (int t = 0; t < tile.threads; ++t)
        for (int i = 0; i < copies; ++i) {
          std::uint64_t from = base + g.copy_src[i], to = g.copy_dst[i];
          for (int b = 0; (1 << b) < tile.threads; ++b)
            if ((t >> b) & 1) {
              from += g.lane_src[b];
              to += g.lane_dst[b];
            }
          if (copies > TileGather::kCopies || from >= m * k || to >= staged.size())
            throw std::string("ERROR (qflex_gb300: cgemm) --> copy out of range");
          staged[to] = src[from];
        }
      for (int r = 0; r < tile.bm; ++r)
        for (int v = 0; v < tile.bk; ++v)
          dst[(mt * tile.bm + r) * k + ks * tile.bk + v] = staged[std::size_t(r) * ar + v];
    }
}

void launch_cgemm_tiled(const float2* A, const TileGather* gather, const float2* B, float2* C, std::size_t m,
                        std::size_t n, std::size_t k, std::uint64_t batch_stride, int batch, float2* scratch,
                        cudaStream_t s, OnlyIf only_if) {
  if (m > 0x7fffffffull || n > 0x7fffffffull || k > 0x7fffffffull)
    throw std::string("ERROR (qflex_gb300: cgemm) --> dimension exceeds 2^31");
  // A gather is made for the usual shapes.
  if (!gather && with_few_tiles(m, n, k, batch, scratch != nullptr, [&](auto shape) {
        using S = decltype(shape);
        std::size_t terms = 0;
        const int splits = scratch ? runs_of<S>(m, n, k, batch, &terms) : 0;
        if (!splits) {
          S::template run<PLAIN>(A, B, C, m, n, k, batch_stride, batch, only_if, s);
          return;
        }
        S::template run<SPLIT>(A, B, C, m, n, k, batch_stride, batch, SplitK{scratch, splits, (int)terms}, s);
        dim3 grid((unsigned)((m * n + 31) / 32), (unsigned)batch);
        split_finish_kernel<<<grid, 256, 0, s>>>(scratch, C, m * n, splits, batch_stride);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) throw std::string("ERROR (qflex_gb300: launch split_finish) --> ") + cudaGetErrorString(e);
      }))
    return;
  const Tile tile = with_shape(m, n, k, [](auto shape) { return decltype(shape)::tile; });
  const std::size_t tiles = ((m + tile.bm - 1) / tile.bm) * ((n + tile.bn - 1) / tile.bn) * (std::size_t)batch;
  if (!gather && !only_if.flag && staged_is_faster(tile, tiles, m, n, k, batch)) {
    if (tile.bm == 256)
      run_staged<256, 16, 16, 8, 2>(A, B, C, m, n, k, batch_stride, batch, s);
    else
      run_staged<128, 64, 16, 8, 4>(A, B, C, m, n, k, batch_stride, batch, s);
    return;
  }
  // Where one or two blocks on an SM hold all tiles: up to 32 columns in tiles
  // of 64 rows, more of them with fewer outputs a thread ((16384, 16, 256) 40
  // and 20 us, (25646, 10, 112) x 2 34 and 23, (30000, 32, 64) 16.8 and 15.6);
  // more columns in k-steps of 32, half the barriers ((2000, 512, 256) 54.7 and
  // 51.2, (92, 717, 148) x 7 37.2 and 34.7).
  if (!gather && n > 8 && tiles <= (n <= 32 ? 304u : 152u)) {
    auto plain = [&](auto shape) {
      decltype(shape)::template run<PLAIN>(A, B, C, m, n, k, batch_stride, batch, only_if, s);
    };
    if (n <= 16) return plain(Shape<64, 16, 16, 4, 2, 4>{});
    if (n <= 32) return plain(Shape<64, 32, 16, 4, 4, 3>{});
    if (m > 64 && k >= 128) return plain(Shape<128, 64, 32, 8, 4, 2>{});
  }
  with_shape(m, n, k, [&](auto shape) {
    decltype(shape)::launch(A, B, C, m, n, k, batch_stride, batch, gather, only_if, s);
    return 0;
  });
}

}  // namespace qfx
