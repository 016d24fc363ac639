// What the tensor-core translation units share: PTX wrappers (mbarriers with
// bounded waits, TMA copies, shared-memory and instruction descriptors,
// tcgen05 issue and TMEM loads), the operand kinds and the truncation-bias
// compensation.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstddef>
#include <cstdint>

#include "tc_gemm.h"

namespace qfx {

// Host helpers, defined in tc_gemm.cu next to the plane layouts.
CUtensorMap plane_map(const float* base, std::uint64_t rows, std::uint64_t kpad, int batch, int box_rows,
                      int row_floats = 32, int box_inner = 32);
CUtensorMap plane_map_bf16(const __nv_bfloat16* base, std::uint64_t rows, std::uint64_t kpad, int batch,
                           int box_rows, int inner, int box_inner);
// Map over complex64 elements (`dims`, byte `strides` of the dimensions from
// the second on) for boxes with rows of 16 elements, 128-byte swizzle.
CUtensorMap element_map(const float2* base, int rank, const std::uint64_t* dims, const std::uint64_t* strides,
                        const std::uint32_t* box);
CUtensorMap plane_map_f16(const __half* base, std::uint64_t rows, std::uint64_t kpad, int batch, int box_rows,
                          int row_halves, int box_inner = 32);
bool output_map(float2* C, std::size_t m, std::size_t n, std::uint64_t batch_stride, int batch, CUtensorMap* map,
                bool narrow = false);
unsigned persistent_grid(std::size_t tiles);
// Splits `batch` operands into planes (split.cu): `rows` rows of k values, or
// with `columns` the columns of a row-major k x rows matrix. `nplanes` 4, or 6
// with the negated imaginary planes (not BF16). `top` holds rows * batch words
// for 3xFP16 columns.
struct SplitOut {
  void* main;
  void* tail;          // BF16x3: the third pieces
  int* exps;           // 3xFP16: one exponent per row
  std::uint32_t* top;
};
void launch_split(SplitKind kind, int nplanes, const SplitOut& out, const float2* src, std::size_t rows,
                  std::size_t k, std::uint64_t src_stride, int batch, bool columns, cudaStream_t s);

namespace {

constexpr unsigned long long WAIT_NS = 2000000000ull;  // 2 s per wait

__device__ __forceinline__ std::uint32_t smem_u32(const void* p) {
  return static_cast<std::uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(std::uint64_t* bar, std::uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(std::uint64_t* bar, std::uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_test(std::uint64_t* bar, std::uint32_t parity) {
  std::uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Limit of a pipeline wait: the 64-bit value the host keeps after the error
// code in the error-flag buffer (err[2..3], written when the buffer is
// created and by the "tc_wait_ns" option), or WAIT_NS when it is 0. Read
// only once a wait has to spin. The drains on the abort path keep WAIT_NS.
__device__ __forceinline__ unsigned long long wait_limit_ns(const int* err) {
  const unsigned long long v = *reinterpret_cast<const volatile unsigned long long*>(err + 2);
  return v ? v : WAIT_NS;
}
// Bounded wait: false (and an error code) when the phase does not complete
// within the wait limit or another warp of the CTA has already given up.
__device__ __forceinline__ bool mbar_wait(std::uint64_t* bar, std::uint32_t parity, volatile int* abort_flag,
                                          int* err, int code) {
  if (mbar_test(bar, parity)) return true;  // the common case reads no timer
  const unsigned long long t0 = now_ns(), limit = wait_limit_ns(err);
  while (!mbar_test(bar, parity)) {
    if (*abort_flag) return false;
    if (now_ns() - t0 > limit) {
      *abort_flag = 1;
      atomicExch(err, code);
      return false;
    }
  }
  return true;
}

__device__ __forceinline__ void tma_load_4d(const CUtensorMap* map, std::uint64_t* bar, void* dst, int c0,
                                            int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
      "%5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<std::uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tma_load_3d(const CUtensorMap* map, std::uint64_t* bar, std::uint32_t dst, int c0,
                                            int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          dst),
      "l"(reinterpret_cast<std::uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}
// Box at the origin of the first four dimensions.
__device__ __forceinline__ void tma_load_5d(const CUtensorMap* map, std::uint64_t* bar, std::uint32_t dst, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %2, %2, %2, %3}], "
      "[%4];" ::"r"(dst),
      "l"(reinterpret_cast<std::uint64_t>(map)), "r"(0), "r"(c4), "r"(smem_u32(bar))
      : "memory");
}

// Bulk tensor store of a shared-memory box to global memory (C tiles), its
// commit group, and the waits for the box's shared-memory reads / for the
// global writes to finish.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(
                   reinterpret_cast<std::uint64_t>(map)),
               "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(src))
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// v * 2^e, exact unless the result leaves the normal range (then rounded
// like ldexpf): a multiply by the power of two when 2^e is a normal float.
__device__ __forceinline__ float scale2(float v, int e) {
  return (e >= -126 && e <= 127) ? v * __uint_as_float(std::uint32_t(e + 127) << 23) : ldexpf(v, e);
}

// Shared-memory matrix descriptor: K-major operand inside rows of 128 bytes
// in the 128-byte swizzle (the start address may sit 32, 64 or 96 bytes into
// the row, as for a K offset), 8-row groups 1024 bytes apart.
__device__ __forceinline__ std::uint64_t smem_desc_sw128(std::uint32_t addr) {
  std::uint64_t d = 0;
  d |= std::uint64_t((addr & 0x3FFFF) >> 4);       // start address
  d |= std::uint64_t(1) << 16;                     // leading byte offset (unused here)
  d |= std::uint64_t(1024 >> 4) << 32;             // stride byte offset
  d |= std::uint64_t(1) << 46;                     // descriptor version
  d |= std::uint64_t(2) << 61;                     // 128-byte swizzle
  return d;
}

// The same for rows of 64 bytes in the 64-byte swizzle (8-row groups 512
// bytes apart); the BF16x3 kernel keeps its third pieces there.
__device__ __forceinline__ std::uint64_t smem_desc_sw64(std::uint32_t addr) {
  std::uint64_t d = 0;
  d |= std::uint64_t((addr & 0x3FFFF) >> 4);
  d |= std::uint64_t(1) << 16;
  d |= std::uint64_t(512 >> 4) << 32;
  d |= std::uint64_t(1) << 46;
  d |= std::uint64_t(4) << 61;                     // 64-byte swizzle
  return d;
}

// Rows of 32 bytes in the 32-byte swizzle (8-row groups 256 bytes apart).
__device__ __forceinline__ std::uint64_t smem_desc_sw32(std::uint32_t addr) {
  std::uint64_t d = 0;
  d |= std::uint64_t((addr & 0x3FFFF) >> 4);
  d |= std::uint64_t(1) << 16;
  d |= std::uint64_t(256 >> 4) << 32;
  d |= std::uint64_t(1) << 46;
  d |= std::uint64_t(6) << 61;                     // 32-byte swizzle
  return d;
}

// Instruction descriptor, kind::tf32: D = F32, A = B = TF32, both K-major.
__host__ __device__ constexpr std::uint32_t idesc_tf32(int m, int n, bool negate_a) {
  return (1u << 4) | (2u << 7) | (2u << 10) | (negate_a ? (1u << 13) : 0u) |
         (std::uint32_t(n >> 3) << 17) | (std::uint32_t(m >> 4) << 24);
}

__device__ __forceinline__ void umma_tf32(std::uint32_t d_tmem, std::uint64_t a, std::uint64_t b,
                                          std::uint32_t idesc, std::uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}
// Instruction descriptor, kind::f16 with FP16 A and B (format 0), F32 D.
__host__ __device__ constexpr std::uint32_t idesc_f16(int m, int n, bool negate_a) {
  return (1u << 4) | (negate_a ? (1u << 13) : 0u) | (std::uint32_t(n >> 3) << 17) | (std::uint32_t(m >> 4) << 24);
}
__device__ __forceinline__ void umma_f16(std::uint32_t d_tmem, std::uint64_t a, std::uint64_t b, std::uint32_t idesc,
                                         std::uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}
// kind::f16 with BF16 A and B (format 1), F32 D.
__host__ __device__ constexpr std::uint32_t idesc_bf16(int m, int n, bool negate_a) {
  return idesc_f16(m, n, negate_a) | (1u << 7) | (1u << 10);
}
template <int KIND>
__host__ __device__ constexpr std::uint32_t idesc_kind(int m, int n, bool negate_a) {
  return KIND == KIND_TF32 ? idesc_tf32(m, n, negate_a)
                           : (KIND == KIND_FP16 ? idesc_f16(m, n, negate_a) : idesc_bf16(m, n, negate_a));
}
// True in one lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  std::uint32_t r;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
  return r != 0;
}
__device__ __forceinline__ void umma_commit(std::uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

#define TMEM_LD16(taddr, r)                                                                            \
  asm volatile(                                                                                        \
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];" \
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),          \
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),       \
        "=r"(r[14]), "=r"(r[15])                                                                      \
      : "r"(taddr))

__device__ __forceinline__ void mbar_arrive(std::uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// ---- Pairs of CTAs (clusters of two, cta_group::2) ---------------------------

__device__ __forceinline__ std::uint32_t cluster_rank() {
  std::uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Shared::cluster address of the same shared-memory offset in CTA `rank`.
__device__ __forceinline__ std::uint32_t peer_addr(const void* p, std::uint32_t rank) {
  std::uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool mbar_test_cluster(std::uint64_t* bar, std::uint32_t parity) {
  std::uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_cluster(std::uint64_t* bar, std::uint32_t parity, volatile int* abort_flag,
                                                  int* err, int code) {
  if (mbar_test_cluster(bar, parity)) return true;
  const unsigned long long t0 = now_ns(), limit = wait_limit_ns(err);
  while (!mbar_test_cluster(bar, parity)) {
    if (*abort_flag) return false;
    if (now_ns() - t0 > limit) {
      *abort_flag = 1;
      atomicExch(err, code);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void mbar_arrive_remote(std::uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load into this CTA's shared memory that completes on a barrier of
// either CTA of the pair (`bar` is a shared::cluster address).
__device__ __forceinline__ void tma_load_4d_pair(const CUtensorMap* map, std::uint32_t bar, void* dst, int c0, int c1,
                                                 int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, "
      "%4, %5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<std::uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}
// Commit of the issuing thread's MMAs, arriving on `bar` in both CTAs.
__device__ __forceinline__ void umma_commit_pair(std::uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(std::uint16_t(3))
      : "memory");
}

// Compensation of the truncation bias. The tensor core's FP32 accumulation
// rounds toward zero, so every product comes out smaller by a fraction beta
// of itself that depends on the split kind and on how many k-steps a TMEM
// chunk accumulates (not on the shape). Measured on GB300 against complex128
// products of Gaussian operands (python -m qflex_gb300.kernel_bench bias), for
// chunks of one and two k-steps; other chunk lengths are not compensated.
// With err[1] != 0 (option "tc_debias") every output x becomes x + beta x,
// one fused multiply-add rounded to nearest (1 + beta itself is not a float:
// beta is below the float spacing at 1).
template <int KIND>
__device__ __forceinline__ float debias_beta(const int* err, int chunk, int kblocks) {
  if (*reinterpret_cast<const volatile int*>(err + 1) == 0) return 0.f;
  const int c = chunk < kblocks ? chunk : kblocks;
  if (c == 1) return KIND == KIND_FP16 ? 5.53e-8f : KIND == KIND_BF16 ? 4.47e-8f : 5.39e-8f;
  if (c == 2) return KIND == KIND_FP16 ? 1.535e-7f : KIND == KIND_BF16 ? 2.226e-7f : 1.52e-7f;
  return 0.f;
}

}  // namespace
}  // namespace qfx
