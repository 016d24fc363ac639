// A whole contraction in one kernel, for circuits whose tensors fit the shared
// memory of an SM: column flatten, every permutation and product of the
// program, and the FP64 amplitude sums. One block per output string, the
// string's arena in shared memory.
//
// The programs of such circuits are a few dozen operations of a few thousand
// multiply-adds; as separate launches (replayed as a graph) each costs about
// 3.3 us of device time, nearly all of it launch gaps and memory latency. Here
// an operation costs 0.4 to 3.7 us, bound by the one SM's issue slots and
// shared memory, and the grid tensors 8 us. A 4 x 5 grid of depth (1 + 16 + 1),
// 29 operations: 104 -> 53 us on the device for one string, 137 -> 56 us for
// 152, 548 -> 343 us for 1024.
//
// The arithmetic is that of the separate kernels: the same gate chains, sums
// over k in ascending order with four FMAs per complex term, and in products
// of vectors the same partial sums added in the same order.
#include <string>

#include "flatten.cuh"
#include "kernels.h"
#include "per_device.h"

namespace qfx {
namespace {

constexpr int NT = 512;

// Rows r0 + i * step and columns c0 .. c0 + TN - 1 of a product; A's element
// (r, kk) lies at row(r) + col[kk]. `even`: rows of B and C start on 16 bytes.
template <int TM, int TN, typename Row>
__device__ __forceinline__ void tile_product(const float2* A, const float2* B, float2* C, int m, int n, int k, int r0,
                                             int step, int c0, bool even, const std::uint32_t* col, Row row) {
  float2 acc[TM][TN];
  std::uint32_t at[TM];
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    at[i] = row(min(r0 + i * step, m - 1));
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
  }
  const bool whole = c0 + TN <= n, pairs = TN % 2 == 0 && whole && even;
#pragma unroll 4
  for (int kk = 0; kk < k; ++kk) {
    float2 b[TN];
    if (pairs) {
#pragma unroll
      for (int j = 0; j + 1 < TN; j += 2) {
        const float4 v = *reinterpret_cast<const float4*>(B + kk * n + c0 + j);
        b[j] = make_float2(v.x, v.y);
        b[j + 1] = make_float2(v.z, v.w);
      }
    } else {
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = B[kk * n + (whole ? c0 + j : min(c0 + j, n - 1))];
    }
    const std::uint32_t ck = col ? col[kk] : kk;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const float2 a = A[at[i] + ck];
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = cfma(a, b[j], acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = r0 + i * step;
    if (r >= m) continue;
    if (pairs) {
#pragma unroll
      for (int j = 0; j + 1 < TN; j += 2)
        *reinterpret_cast<float4*>(C + r * n + c0 + j) =
            make_float4(acc[i][j].x, acc[i][j].y, acc[i][j + 1].x, acc[i][j + 1].y);
    } else {
#pragma unroll
      for (int j = 0; j < TN; ++j)
        if (c0 + j < n) C[r * n + c0 + j] = acc[i][j];
    }
  }
}

__device__ __forceinline__ float2 warp_sum(float2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}

// Products with one column (m x k times a vector of more than 32) or one row
// (of up to 255 columns): a warp per output, as the separate kernels for
// vectors sum them (gemv_rows_warp, gemv_cols_block). One thread per output
// would add up to 1024 terms one after the other.
__device__ __noinline__ void column_product(const float2* A, const float2* B, float2* C, int m, int k) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int i = threadIdx.x >> 5; i < m; i += NT / 32) {
    float2 acc = make_float2(0.f, 0.f);
    for (int kk = lane; kk < k; kk += 32) acc = cfma(A[i * k + kk], B[kk], acc);
    acc = warp_sum(acc);
    if (lane == 0) C[i] = acc;
  }
}
__device__ __noinline__ void row_product(const float2* A, const float2* B, float2* C, int n, int k) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int j = threadIdx.x >> 5; j < n; j += NT / 32) {
    // The sums of eight warps of which each takes 32 terms in turn.
    float2 part = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int w = 0; w < 8 && 32 * w < k; ++w) {
      float2 acc = make_float2(0.f, 0.f);
      for (int kk = 32 * w + lane; kk < k; kk += 256) acc = cfma(A[kk], B[kk * n + j], acc);
      acc = warp_sum(acc);
      if (lane == w) part = acc;
    }
    part = warp_sum(part);
    if (lane == 0) C[j] = part;
  }
}

// Index x with its bit b moved to bit to[b], the destinations unpacked once per
// operation.
struct BitMoves {
  std::uint32_t to[16];
  __device__ __forceinline__ explicit BitMoves(const SmallOp& op) {
    const uint2* w = reinterpret_cast<const uint2*>(op.to);
    const uint2 lo = w[0], hi = w[1];
    const std::uint32_t word[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
    for (int b = 0; b < 16; ++b) to[b] = (word[b / 4] >> (8 * (b % 4))) & 31u;
  }
  __device__ __forceinline__ std::uint32_t operator()(std::uint32_t x) const {
    std::uint32_t y = 0;
#pragma unroll
    for (int b = 0; b < 16; ++b) y |= ((x >> b) & 1u) << to[b];
    return y;
  }
};

template <bool kCompensated>
__global__ void __launch_bounds__(NT, 1)
    small_program_kernel(const SmallProgram p, const std::uint8_t* __restrict__ init_bits,
                         const std::uint8_t* __restrict__ final_bits, double2* __restrict__ amps) {
  extern __shared__ __align__(16) std::uint8_t raw[];
  float2* arena = reinterpret_cast<float2*>(raw);
  float2* mats = arena + p.arena_elems;
  float2* mats_lo = mats + p.n_mats;
  StepDesc* steps = reinterpret_cast<StepDesc*>(mats_lo + (kCompensated ? p.n_mats : 0));
  ColumnDesc* cols = reinterpret_cast<ColumnDesc*>(steps + p.n_steps);
  SmallOp* ops = reinterpret_cast<SmallOp*>(cols + p.n_cols);
  std::uint32_t* at_k = reinterpret_cast<std::uint32_t*>(ops + p.n_ops);  // kMaxK of them
  const int t = threadIdx.x, string = blockIdx.x;
  auto fetch = [&](void* dst, const void* src, std::size_t bytes) {
    for (std::size_t i = t; i < bytes / 8; i += NT)
      reinterpret_cast<uint2*>(dst)[i] = __ldg(reinterpret_cast<const uint2*>(src) + i);
  };
  fetch(mats, p.mats, p.n_mats * sizeof(float2));
  if (kCompensated) fetch(mats_lo, p.mats_lo, p.n_mats * sizeof(float2));
  fetch(steps, p.steps, p.n_steps * sizeof(StepDesc));
  fetch(cols, p.cols, p.n_cols * sizeof(ColumnDesc));
  fetch(ops, p.ops, p.n_ops * sizeof(SmallOp));
  init_bits += std::size_t(string) * p.n_cols;
  final_bits += std::size_t(string) * p.n_cols;
  __syncthreads();

  // Grid tensors: warps take pieces of 128 elements of a column, four per
  // lane, so that four gate chains run side by side.
  {
    const int lane = t & 31;
    std::uint32_t piece = t >> 5;
    for (std::uint32_t c = 0; c < p.n_cols; ++c) {
      const ColumnDesc cd = cols[c];
      const std::uint32_t size = 1u << cd.size_log2, pieces = (size + 127) / 128;
      for (; piece < pieces; piece += NT / 32) {
        std::uint32_t e[4];
        float2 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) e[u] = piece * 128 + u * 32 + lane;
        const bool final_bit = final_bits[c] != 0;
        column_elements<kCompensated, 4>(cd, steps, mats, mats_lo, init_bits[c] != 0, e, v, [&](int u) {
          return cd.o_shift >= 0 ? ((e[u] >> cd.o_shift) & 1) != 0 : final_bit;
        });
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (e[u] < size) arena[cd.out_offset + e[u]] = v[u];
      }
      piece -= pieces;
    }
  }
  __syncthreads();

  for (std::uint32_t o = 0; o < p.n_ops; ++o) {
    const SmallOp& op = ops[o];
    const float2* A = arena + op.a;
    float2* C = arena + op.c;
    const BitMoves move(op);
    if (op.k == 0) {  // permutation of m elements
      for (std::uint32_t e = t; e < op.m; e += NT) C[move(e)] = A[e];
    } else {
      const float2* B = arena + op.b;
      const int m = op.m, n = op.n, k = op.k;
      const std::uint32_t* col = nullptr;
      if (op.bits) {  // A through a permutation: `to` is operand digit -> source digit
        for (int kk = t; kk < k; kk += NT) at_k[kk] = move(kk);
        col = at_k;
        __syncthreads();
      }
      auto row = [&](int r) {
        return op.bits ? move(std::uint32_t(r) * k) : std::uint32_t(r) * k;
      };
      // Neighbouring lanes take columns, then neighbouring rows: A's rows
      // through a permutation mostly lie side by side, in different banks.
      // (256 x 16 x 16: 7000 cycles; four neighbouring rows per thread 8200,
      // two rows per thread 7300.)
      const int cols4 = (n + 3) / 4, rows4 = (m + 3) / 4;
      const bool even = ((op.b | op.c | n) & 1) == 0;
      if (n == 1 && k > 32) {
        column_product(A, B, C, m, k);
      } else if (m == 1 && n > 1 && n < 256) {
        row_product(A, B, C, n, k);
      } else if (m * n >= 2048) {
        for (int i = t; i < rows4 * cols4; i += NT)
          tile_product<4, 4>(A, B, C, m, n, k, i / cols4, rows4, i % cols4 * 4, even, col, row);
      } else if (m * n >= 512) {
        for (int i = t; i < m * cols4; i += NT)
          tile_product<1, 4>(A, B, C, m, n, k, i / cols4, 1, i % cols4 * 4, even, col, row);
      } else {
        for (int i = t; i < m * n; i += NT) tile_product<1, 1>(A, B, C, m, n, k, i / n, 1, i % n, even, col, row);
      }
    }
    __syncthreads();
  }

  for (std::uint32_t a = t; a < p.n_amps; a += NT) {
    double re = 0, im = 0;
    for (std::uint32_t q = p.ptr[a]; q < p.ptr[a + 1]; ++q) {
      const float2 v = arena[p.results + p.leaves[q]];
      re += double(v.x);
      im += double(v.y);
    }
    amps[std::size_t(string) * p.n_amps + a] = make_double2(re, im);
  }
}

}  // namespace

std::size_t small_program_smem(const SmallProgram& p) {
  const std::size_t mats = p.n_mats * sizeof(float2) * (p.mats_lo ? 2 : 1);
  return p.arena_elems * sizeof(float2) + mats + p.n_steps * sizeof(StepDesc) + p.n_cols * sizeof(ColumnDesc) +
         p.n_ops * sizeof(SmallOp) + SmallProgram::kMaxK * sizeof(std::uint32_t);
}

void launch_small_program(const SmallProgram& p, const std::uint8_t* init_bits, const std::uint8_t* final_bits,
                          double2* amps, int batch, cudaStream_t s) {
  const std::size_t smem = small_program_smem(p);
  static PerDevice raised;
  raised([] {
    for (auto* kernel : {small_program_kernel<false>, small_program_kernel<true>})
      raise_smem_limit(kernel, (int)SmallProgram::kMaxSmem);
    return 1;
  });
  auto run = [&](auto* kernel) {
    kernel<<<(unsigned)batch, NT, smem, s>>>(p, init_bits, final_bits, amps);
  };
  if (p.mats_lo)
    run(small_program_kernel<true>);
  else
    run(small_program_kernel<false>);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    throw std::string("ERROR (qflex_gb300: launch small_program) --> ") + cudaGetErrorString(e);
}

}  // namespace qfx
