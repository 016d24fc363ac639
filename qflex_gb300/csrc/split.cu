// Splitting complex64 operands into the planes that the tensor-core products
// load (tc_gemm.cu, tc_direct.cu), from rows of k values or from the columns
// of a row-major k x n matrix.
//
// All three kinds share the work split: a thread takes the consecutive values
// of k that make a 16-byte unit of every plane (eight, four for TF32), and two
// neighbouring threads fill a 32-byte plane row, so every store instruction
// writes whole sectors. (A thread writing both halves of TF32 rows took 3 to 6
// times as long.)
//
// Bound by HBM: 8 B read and 8 (3xFP16; 12 with the negated copy of the
// imaginary planes), 12 (BF16x3) or 16 (3xTF32; 24) B written per element.
// Measured at 4096 x 4096, against two values per thread, a second pass over
// every 3xFP16 row, and a permutation (42 us) before the rows of a row-major B:
//   3xFP16 rows 100 -> 50 us, columns 142 -> 87 us (with the negated copy), in
//   one pass (without) 63; at 1100 x 690 8.4 -> 6.4 us and two launches fewer
//   3xTF32 rows  79 -> 74 us, columns 134 -> 83 us (with the negated copy)
//   BF16x3 rows  68 -> 57 us, columns 110 -> 52 us
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <string>

#include "half_split.cuh"
#include "per_device.h"
#include "tc_common.cuh"

namespace qfx {
namespace {

// The exponent e of a 3xFP16 row whose largest component has the bit pattern
// `mb`: max * 2^e in [2^14, 2^15). Rows of zeros, and rows with infinities or
// NaN, keep 0.
__device__ __forceinline__ int scale_exponent(std::uint32_t mb) {
  const int be = int(mb >> 23);
  if (be > 0 && be < 255) return 141 - be;
  if (be != 0 || mb == 0) return 0;
  int ex;
  frexpf(__uint_as_float(mb), &ex);  // subnormal
  return 15 - ex;
}

// Values of a unit: one 16-byte piece of a plane.
template <int KIND>
constexpr int unit_values() {
  return KIND == KIND_TF32 ? 4 : 8;
}

// Values kk .. kk + V - 1 of a row of k, zero beyond it.
template <int V>
__device__ __forceinline__ void load_unit(const float2* row, std::uint64_t k, std::uint64_t kk, bool vec,
                                          float2 (&v)[V]) {
  if (vec && kk + V <= k) {
#pragma unroll
    for (int j = 0; j < V / 2; ++j) {
      const float4 q = __ldg(reinterpret_cast<const float4*>(row + kk) + j);
      v[2 * j] = make_float2(q.x, q.y);
      v[2 * j + 1] = make_float2(q.z, q.w);
    }
  } else {
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] = kk + j < k ? row[kk + j] : make_float2(0.f, 0.f);
  }
}
template <int V>
__device__ __forceinline__ std::uint32_t largest(const float2 (&v)[V]) {
  std::uint32_t m = 0;
#pragma unroll
  for (int j = 0; j < V; ++j)
    m = max(m, max(__float_as_uint(v[j].x) & 0x7fffffffu, __float_as_uint(v[j].y) & 0x7fffffffu));
  return m;
}

template <typename T>
__device__ __forceinline__ uint4 as_unit(const T (&p)[4]) {
  static_assert(sizeof(T) == 4, "a unit is four 32-bit words");
  const std::uint32_t* w = reinterpret_cast<const std::uint32_t*>(p);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Writes the planes of the unit at value kk of row `row` of `rows`. Layouts per batch entry: 3xFP16 [k / 16][row][plane][16] fp16
// (re hi, lo, im hi, lo; with NP = 6 also -im hi, lo) of the values times 2^e;
// 3xTF32 [k / 8][row][plane][8] fp32, the same planes; BF16x3 main
// [k / 16][row][re0, re1, im0, im1][16] and tail [k / 16][row][re2, im2][16].
template <int KIND, int NP>
__device__ __forceinline__ void emit(const float2 (&v)[unit_values<KIND>()], int e, void* main_planes, void* tail_planes,
                                     std::uint64_t rows, std::uint64_t row, std::uint64_t kk) {
  if constexpr (KIND == KIND_FP16) {
    // Scaling by 2^e is exact; two steps when 2^e is no normal float.
    const float s1 = __uint_as_float(std::uint32_t(min(e, 127) + 127) << 23);
    const float s2 = __uint_as_float(std::uint32_t(max(e - 127, 0) + 127) << 23);
    std::uint32_t rh[4], rl[4], ih[4], il[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float r0 = v[2 * j].x * s1, i0 = v[2 * j].y * s1, r1 = v[2 * j + 1].x * s1, i1 = v[2 * j + 1].y * s1;
      if (e > 127) {
        r0 *= s2;
        i0 *= s2;
        r1 *= s2;
        i1 *= s2;
      }
      split_pair(r0, r1, rh[j], rl[j]);
      split_pair(i0, i1, ih[j], il[j]);
    }
    uint4* o = reinterpret_cast<uint4*>(static_cast<__half*>(main_planes) + ((kk / 16) * rows + row) * (16 * NP) +
                                        kk % 16);
    o[0] = as_unit(rh);
    o[2] = as_unit(rl);
    o[4] = as_unit(ih);
    o[6] = as_unit(il);
    if constexpr (NP == 6) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        ih[j] ^= 0x80008000u;
        il[j] ^= 0x80008000u;
      }
      o[8] = as_unit(ih);
      o[10] = as_unit(il);
    }
  } else if constexpr (KIND == KIND_TF32) {
    float4* o = reinterpret_cast<float4*>(static_cast<float*>(main_planes) + ((kk / 8) * rows + row) * (8 * NP) +
                                          kk % 8);
    float rh[4], ih[4], rl[4], il[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      rh[j] = tf32_rn(v[j].x);
      ih[j] = tf32_rn(v[j].y);
      rl[j] = tf32_rn(v[j].x - rh[j]);
      il[j] = tf32_rn(v[j].y - ih[j]);
    }
    o[0] = make_float4(rh[0], rh[1], rh[2], rh[3]);
    o[2] = make_float4(rl[0], rl[1], rl[2], rl[3]);
    o[4] = make_float4(ih[0], ih[1], ih[2], ih[3]);
    o[6] = make_float4(il[0], il[1], il[2], il[3]);
    if constexpr (NP == 6) {
      o[8] = make_float4(-ih[0], -ih[1], -ih[2], -ih[3]);
      o[10] = make_float4(-il[0], -il[1], -il[2], -il[3]);
    }
  } else {
    std::uint32_t r0[4], r1[4], r2[4], i0[4], i1[4], i2[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      split_bf16(v[2 * j].x, v[2 * j + 1].x, r0[j], r1[j], r2[j]);
      split_bf16(v[2 * j].y, v[2 * j + 1].y, i0[j], i1[j], i2[j]);
    }
    const std::uint64_t at = (kk / 16) * rows + row;
    uint4* o = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(main_planes) + at * 64 + kk % 16);
    o[0] = as_unit(r0);
    o[2] = as_unit(r1);
    o[4] = as_unit(i0);
    o[6] = as_unit(i1);
    uint4* t = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(tail_planes) + at * 32 + kk % 16);
    t[0] = as_unit(r2);
    t[2] = as_unit(i2);
  }
}

// Rows of k values: G = 2^g_log2 threads per row (a power of two up to 32, or
// the whole block of 256), thread g of a row on units g, g + G, ... For 3xFP16
// up to four units per thread stay in registers between the row's maximum and
// its planes; longer rows are read a second time.
template <int KIND>
constexpr int kept_units() {
  return KIND == KIND_FP16 ? 4 : 1;
}
template <int KIND, int NP>
__global__ void __launch_bounds__(256) split_rows_kernel(const float2* __restrict__ src, void* __restrict__ main_planes,
                                                         void* __restrict__ tail_planes, int* __restrict__ exps,
                                                         std::uint64_t rows, std::uint64_t k, std::uint64_t kpad,
                                                         std::uint64_t src_stride, std::uint64_t main_stride,
                                                         std::uint64_t tail_stride, int g_log2) {
  __shared__ std::uint32_t part[8];
  const std::uint64_t b = blockIdx.y;
  src += b * src_stride;
  main_planes = static_cast<char*>(main_planes) + b * main_stride;
  tail_planes = static_cast<char*>(tail_planes) + b * tail_stride;
  const int G = 1 << g_log2, per_block = 256 >> g_log2;
  const int g = threadIdx.x & (G - 1);
  constexpr int V = unit_values<KIND>(), KEEP = kept_units<KIND>();
  const std::uint64_t units = kpad / V;
  for (std::uint64_t first = std::uint64_t(blockIdx.x) * per_block; first < rows;
       first += std::uint64_t(gridDim.x) * per_block) {
    const std::uint64_t row = first + (threadIdx.x >> g_log2);
    const bool here = row < rows;
    const float2* r = src + (here ? row : 0) * k;
    const bool vec = (reinterpret_cast<std::uintptr_t>(r) & 15) == 0;
    float2 v[KEEP][V];
#pragma unroll
    for (int i = 0; i < KEEP; ++i) {
      const std::uint64_t o = g + std::uint64_t(i) * G;
      if (here && o < units) load_unit(r, k, o * V, vec, v[i]);
    }
    int e = 0;
    if constexpr (KIND == KIND_FP16) {
      std::uint32_t mx = 0;
#pragma unroll
      for (int i = 0; i < KEEP; ++i)
        if (here && g + std::uint64_t(i) * G < units) mx = max(mx, largest(v[i]));
      if (here)
        for (std::uint64_t o = g + std::uint64_t(KEEP) * G; o < units; o += G) {
          float2 w[V];
          load_unit(r, k, o * V, vec, w);
          mx = max(mx, largest(w));
        }
      for (int o = min(G, 32) / 2; o; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (G > 32) {
        __syncthreads();  // the previous row's maxima are read
        if ((threadIdx.x & 31) == 0) part[threadIdx.x / 32] = mx;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < 8; ++w) mx = max(mx, part[w]);
      }
      e = scale_exponent(mx);
      if (here && g == 0) exps[b * rows + row] = e;
    }
    if (!here) continue;
#pragma unroll
    for (int i = 0; i < KEEP; ++i) {
      const std::uint64_t o = g + std::uint64_t(i) * G;
      if (o < units) emit<KIND, NP>(v[i], e, main_planes, tail_planes, rows, row, o * V);
    }
    for (std::uint64_t o = g + std::uint64_t(KEEP) * G; o < units; o += G) {
      float2 w[V];
      load_unit(r, k, o * V, vec, w);
      emit<KIND, NP>(w, e, main_planes, tail_planes, rows, row, o * V);
    }
  }
}

// Columns of a row-major k x n matrix become the rows of planes. 3xFP16, whose
// scale is a column's, in one pass: a cluster of CTAs holds 16 columns, each a
// run of `deep` values of k, in shared memory, exchanges the largest
// components and writes the planes. Rows of 17 elements: the two halves of a
// k-step, 8 rows apart, lie in different banks.
constexpr int SLAB = 16, PITCH = SLAB + 1;
template <int NP>
__global__ void __launch_bounds__(256, 3) split_cols_cluster_kernel(const float2* __restrict__ src,
                                                                 void* __restrict__ main_planes, int* __restrict__ exps,
                                                                 std::uint64_t n, std::uint64_t k, std::uint64_t kpad,
                                                                 std::uint64_t src_stride, std::uint64_t main_stride,
                                                                 int deep, int ranks) {
  extern __shared__ float2 slab[];
  __shared__ std::uint32_t part[8][SLAB], top[SLAB];
  __shared__ int scale[SLAB];
  const std::uint64_t b = blockIdx.y;
  src += b * src_stride;
  main_planes = static_cast<char*>(main_planes) + b * main_stride;
  const std::uint32_t rank = cluster_rank();
  const std::uint64_t n0 = std::uint64_t(blockIdx.x / ranks) * SLAB, k0 = std::uint64_t(rank) * deep;
  {
    const int c = threadIdx.x % SLAB, w = threadIdx.x / 32;
    const bool in = n0 + c < n;
    const float2* s = src + n0 + c;
    std::uint32_t mx = 0;
    for (int r0 = threadIdx.x / SLAB; r0 < deep; r0 += 256) {  // 16 rows in flight
      float2 v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int r = r0 + 16 * i;
        v[i] = in && r < deep && k0 + r < k ? __ldg(s + (k0 + r) * n) : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (r0 + 16 * i < deep) slab[(r0 + 16 * i) * PITCH + c] = v[i];
        mx = max(mx, max(__float_as_uint(v[i].x) & 0x7fffffffu, __float_as_uint(v[i].y) & 0x7fffffffu));
      }
    }
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, SLAB));
    if (threadIdx.x % 32 < SLAB) part[w][c] = mx;
  }
  __syncthreads();
  if (threadIdx.x < SLAB) {
    std::uint32_t mx = part[0][threadIdx.x];
#pragma unroll
    for (int w = 1; w < 8; ++w) mx = max(mx, part[w][threadIdx.x]);
    top[threadIdx.x] = mx;
  }
  __syncthreads();
  cluster_sync();
  if (threadIdx.x < SLAB) {
    std::uint32_t mx = 0;
    for (int q = 0; q < ranks; ++q) {
      std::uint32_t v;
      asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer_addr(&top[threadIdx.x], q)) : "memory");
      mx = max(mx, v);
    }
    const int e = scale_exponent(mx);
    scale[threadIdx.x] = e;
    if (rank == 0 && n0 + threadIdx.x < n) exps[b * n + n0 + threadIdx.x] = e;
  }
  __syncthreads();
  // No CTA ends while another still reads its maxima: waited for below.
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  const int c = (threadIdx.x >> 1) % SLAB;
  if (n0 + c < n) {
    const int e = scale[c];
    for (int at = (threadIdx.x >> 5) * 16 + (threadIdx.x & 1) * 8; at < deep && k0 + at < kpad; at += 128) {
      float2 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = slab[(at + j) * PITCH + c];
      emit<KIND_FP16, NP>(v, e, main_planes, nullptr, n, n0 + c, k0 + at);
    }
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Columns longer than the clusters hold with three CTAs on an SM (4096
// values; with one CTA on an SM 13000 x 1000 took 127 us, this way 62). The
// largest component of every column first (bit patterns, by integer maxima): blocks
// of 32 columns x `depth` rows.
__global__ void __launch_bounds__(256) column_max_kernel(const float2* __restrict__ src, std::uint32_t* __restrict__ top,
                                                         std::uint64_t n, std::uint64_t k, std::uint64_t src_stride,
                                                         std::uint64_t depth) {
  __shared__ std::uint32_t part[8][32];
  const std::uint64_t b = blockIdx.z;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const std::uint64_t col = std::uint64_t(blockIdx.x) * 32 + lane;
  const std::uint64_t k0 = std::uint64_t(blockIdx.y) * depth, k1 = min(k0 + depth, k);
  std::uint32_t mx = 0;
  if (col < n) {
    const float2* s = src + b * src_stride + col;
#pragma unroll 8
    for (std::uint64_t kk = k0 + w; kk < k1; kk += 8) {
      const float2 v = __ldg(s + kk * n);
      mx = max(mx, max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu));
    }
  }
  part[w][lane] = mx;
  __syncthreads();
  if (w == 0 && col < n) {
#pragma unroll
    for (int q = 1; q < 8; ++q) mx = max(mx, part[q][lane]);
    if (mx) atomicMax(top + b * n + col, mx);
  }
}

// Then tiles of 64 values of k x 32 columns through shared memory: read as
// rows of 256 bytes, thread (half, column, plane row) writes a unit.
template <int KIND, int NP>
__global__ void __launch_bounds__(256) split_cols_kernel(const float2* __restrict__ src, void* __restrict__ main_planes,
                                                         void* __restrict__ tail_planes,
                                                         const std::uint32_t* __restrict__ top, int* __restrict__ exps,
                                                         std::uint64_t n, std::uint64_t k, std::uint64_t kpad,
                                                         std::uint64_t src_stride, std::uint64_t main_stride,
                                                         std::uint64_t tail_stride) {
  __shared__ float2 tile[64][33];
  const std::uint64_t b = blockIdx.y;
  src += b * src_stride;
  main_planes = static_cast<char*>(main_planes) + b * main_stride;
  tail_planes = static_cast<char*>(tail_planes) + b * tail_stride;
  const unsigned deep = unsigned((kpad + 63) / 64);
  const std::uint64_t k0 = std::uint64_t(blockIdx.x % deep) * 64, n0 = std::uint64_t(blockIdx.x / deep) * 32;
  {
    const int c = threadIdx.x & 31, r0 = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = r0 + 8 * i;
      tile[r][c] = k0 + r < k && n0 + c < n ? __ldg(src + (k0 + r) * n + n0 + c) : make_float2(0.f, 0.f);
    }
  }
  __syncthreads();
  constexpr int V = unit_values<KIND>();
  const int c = (threadIdx.x >> 1) & 31;
  const std::uint64_t col = n0 + c;
  if (col >= n) return;
  int e = 0;
  if constexpr (KIND == KIND_FP16) {
    e = scale_exponent(top[b * n + col]);
    if (k0 == 0 && threadIdx.x < 64 && !(threadIdx.x & 1)) exps[b * n + col] = e;
  }
#pragma unroll
  for (int i = 0; i < 8 / V; ++i) {
    const int at = ((threadIdx.x >> 6) + 4 * i) * 2 * V + (threadIdx.x & 1) * V;
    if (k0 + at >= kpad) break;
    float2 v[V];
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] = tile[at + j][c];
    emit<KIND, NP>(v, e, main_planes, tail_planes, n, col, k0 + at);
  }
}

void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw std::string("ERROR (qflex_gb300: CUDA ") + what + ") --> " + cudaGetErrorString(e);
}

struct Strides {
  std::size_t kpad, main_bytes, tail_bytes;  // of one batch entry
};
template <int KIND, int NP>
Strides strides(std::size_t rows, std::size_t k) {
  if (KIND == KIND_TF32) {
    const std::size_t kpad = (k + 7) / 8 * 8;
    return {kpad, rows * kpad * NP * 4, 0};
  }
  const std::size_t kpad = (k + 15) / 16 * 16;
  return {kpad, rows * kpad * NP * 2, KIND == KIND_BF16 ? rows * kpad * 4 : 0};
}

template <int KIND, int NP>
void run_split(const SplitOut& out, const float2* src, std::size_t rows, std::size_t k, std::uint64_t src_stride,
               int batch, bool columns, cudaStream_t s) {
  const Strides st = strides<KIND, NP>(rows, k);
  if (!columns) {
    int g = 0;
    constexpr unsigned V = unit_values<KIND>();
    // Half a warp per row where there are rows enough: a store then touches
    // fewer k-steps and more neighbouring rows, which lie together (3xTF32,
    // 65536 x 256 x 4: 312 -> 228 us; 8 threads per row: 232 us). Few long
    // rows need the threads (4096 x 2048: 33 us with 32, 38 us with 16).
    const int most = KIND != KIND_FP16 && rows >= 16384 ? 4 : 5;
    while (g < most && (V << g) < st.kpad) ++g;
    // A row that a warp's registers do not hold takes a block.
    if (KIND == KIND_FP16 && st.kpad > 32 * V * kept_units<KIND>()) g = 8;
    const std::uint64_t blocks = (rows + (256u >> g) - 1) >> (8 - g);
    dim3 grid((unsigned)std::min<std::uint64_t>(blocks, 152 * 32), (unsigned)batch);
    split_rows_kernel<KIND, NP><<<grid, 256, 0, s>>>(src, out.main, out.tail, out.exps, rows, k, st.kpad, src_stride,
                                                     st.main_bytes, st.tail_bytes, g);
    check(cudaGetLastError(), "split_rows");
    return;
  }
  const unsigned cols = (unsigned)((rows + 31) / 32);
  if constexpr (KIND == KIND_FP16) {
    // As many CTAs as keep three on an SM (512 values of k each), then as many
    // as give every SM two, of at least 32 values.
    const std::size_t slabs = (rows + SLAB - 1) / SLAB * (std::size_t)batch;
    int ranks = 1;
    while (ranks < 8 && (st.kpad > 512u * ranks || (slabs * ranks < 304 && st.kpad >= 64u * ranks))) ranks *= 2;
    const std::size_t deep = (st.kpad / 16 + ranks - 1) / ranks * 16, bytes = deep * PITCH * sizeof(float2);
    if (deep <= 512) {
      auto* kernel = split_cols_cluster_kernel<NP>;
      static PerDevice raised;
      raised([&] {
        raise_smem_limit(kernel, 512 * PITCH * (int)sizeof(float2));
        return 1;
      });
      cudaLaunchConfig_t lc = {};
      lc.gridDim = dim3((unsigned)((rows + SLAB - 1) / SLAB * ranks), (unsigned)batch, 1);
      lc.blockDim = dim3(256, 1, 1);
      lc.dynamicSmemBytes = bytes;
      lc.stream = s;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = (unsigned)ranks;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      lc.attrs = at;
      lc.numAttrs = 1;
      check(cudaLaunchKernelEx(&lc, kernel, src, out.main, out.exps, (std::uint64_t)rows, (std::uint64_t)k,
                               (std::uint64_t)st.kpad, src_stride, (std::uint64_t)st.main_bytes, (int)deep, ranks),
            "split_cols_cluster");
      return;
    }
    check(cudaMemsetAsync(out.top, 0, rows * (std::size_t)batch * sizeof(std::uint32_t), s), "cudaMemsetAsync");
    // Deep enough to amortize a block, shallow enough for several on each SM.
    const std::size_t want = std::max<std::size_t>(1, 152 * 8 / ((std::size_t)cols * batch));
    const std::size_t depth = std::max<std::size_t>(64, (k + want - 1) / want);
    dim3 grid(cols, (unsigned)((k + depth - 1) / depth), (unsigned)batch);
    column_max_kernel<<<grid, 256, 0, s>>>(src, out.top, rows, k, src_stride, depth);
    check(cudaGetLastError(), "column_max");
  }
  dim3 grid((unsigned)((st.kpad + 63) / 64 * cols), (unsigned)batch);
  split_cols_kernel<KIND, NP><<<grid, 256, 0, s>>>(src, out.main, out.tail, out.top, out.exps, rows, k, st.kpad,
                                                   src_stride, st.main_bytes, st.tail_bytes);
  check(cudaGetLastError(), "split_cols");
}

}  // namespace

void launch_split(SplitKind kind, int nplanes, const SplitOut& out, const float2* src, std::size_t rows,
                  std::size_t k, std::uint64_t src_stride, int batch, bool columns, cudaStream_t s) {
  if (kind == KIND_FP16)
    nplanes == 6 ? run_split<KIND_FP16, 6>(out, src, rows, k, src_stride, batch, columns, s)
                 : run_split<KIND_FP16, 4>(out, src, rows, k, src_stride, batch, columns, s);
  else if (kind == KIND_TF32)
    nplanes == 6 ? run_split<KIND_TF32, 6>(out, src, rows, k, src_stride, batch, columns, s)
                 : run_split<KIND_TF32, 4>(out, src, rows, k, src_stride, batch, columns, s);
  else
    run_split<KIND_BF16, 4>(out, src, rows, k, src_stride, batch, columns, s);
}

}  // namespace qfx
