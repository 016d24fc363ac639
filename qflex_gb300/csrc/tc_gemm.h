// Split-precision complex64 products on the tcgen05 tensor cores.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace qfx {

// Operand kinds: 3xTF32 planes (8 values of 4
// bytes per plane and k-step) or 3xFP16 planes (16 values of 2 bytes, rows
// scaled by powers of two).
// BF16x3: three BF16 pieces per value (x = b0 + b1 + b2 to ~24 bits).
enum SplitKind : int { KIND_TF32 = 0, KIND_FP16 = 1, KIND_BF16 = 2 };

// Shapes that a contraction gives to the tensor-core kernels (smaller products
// stay on the CUDA-core kernels).
bool tc_eligible(std::size_t m, std::size_t n, std::size_t k);
// Shapes the kernels can run.
bool tc_runs(std::size_t m, std::size_t n, std::size_t k);
// How B lies in memory: n rows of k values, or k rows of n.
enum class BLayout { nk, kn };
// 3xTF32 products of 17 to 32 terms with many columns and outputs: loading both
// operands' planes, with the real and imaginary parts in MMAs of their own, is
// then ahead of splitting A inside the kernel, as a tile's store bounds both.
bool tf32_separate(std::size_t m, std::size_t n, std::size_t k);
// The same of BF16x3 with 33 to 64 terms.
bool bf16_separate(std::size_t m, std::size_t n, std::size_t k);
// fp32 elements of split planes one batch entry needs (A and B of any split kind).
std::size_t tc_workspace_elems(std::size_t m, std::size_t n, std::size_t k);

// Kernel choice of one product.
struct TcConfig {
  int chunk = 2;     // k-steps per TMEM accumulation chunk, 1..64 (QFLEX_TC_CHUNK)
  int variant = 0;   // 0: the product that splits A itself (tc_direct.cu) where it runs, else single
                     // CTA; 1: CTA pair from planes; -1: CTA pair when m >= 256, else single;
                     // 2: 3xFP16 single CTA with five stages; 3: 3xFP16 single CTA with 16
                     // epilogue warps; 4: 3xFP16 single CTA with 64-column tiles and four
                     // TMEM chunk buffers (others: single CTA)
};
// Defaults: chunk from QFLEX_TC_CHUNK, variant -1 when QFLEX_TC_PAIR=1, 2 when
// QFLEX_TC_DEEP=1.
TcConfig tc_default_config();

// C[m,n] = A[m,k] * B (complex64, B in either layout), 3xTF32 split, FP32
// accumulation. Batch entry b reads A + b * ac_stride, B + b * b_stride and
// writes C + b * ac_stride. `workspace` holds
// batch * tc_workspace_elems fp32; `err` (device int) receives a nonzero
// code if a pipeline wait expired.
void launch_cgemm_tf32x3(const float2* A, const float2* B, BLayout b_layout, float2* C, std::size_t m,
                         std::size_t n, std::size_t k, std::uint64_t ac_stride, std::uint64_t b_stride, int batch,
                         float* workspace, int* err, const TcConfig& cfg, cudaStream_t s);

// Where the 3xFP16 product keeps its operands in `workspace` (batch entries
// after each other in every region): A planes, Bt planes, the row exponents
// of A and of Bt, and the block exponents of an A operand that arrives as
// planes (one per 32 values of a row).
struct Fp16Workspace {
  void* a_planes;
  void* b_planes;
  int* a_exps;
  int* b_exps;
  int* a_block_exps;
  std::uint32_t* b_top;  // largest components of B's columns while it is split
};
Fp16Workspace fp16_workspace(float* workspace, std::size_t m, std::size_t n, std::size_t k, int batch);

// The same product with 3xFP16 planes: every row of A and of Bt is scaled by
// a power of two so that its largest component lies in [2^14, 2^15), split
// into FP16 hi + lo, multiplied as hi*hi + hi*lo + lo*hi on kind::f16
// tensor cores (twice the TF32 rate) and unscaled in the epilogue. Always
// the single-CTA kernel; cfg.variant is ignored.
// With `a_in_planes` the A planes and block exponents are already in the
// workspace (written by launch_permute_fp16_planes; k a power of two >= 32,
// cfg.chunk <= 2 so that a TMEM chunk never spans two exponent blocks) and
// A is not read.
void launch_cgemm_fp16x3(const float2* A, const float2* B, BLayout b_layout, float2* C, std::size_t m,
                         std::size_t n, std::size_t k, std::uint64_t ac_stride, std::uint64_t b_stride, int batch,
                         float* workspace, int* err, const TcConfig& cfg, cudaStream_t s,
                         bool a_in_planes = false);

// Where the direct products find A: TMA boxes or, where no box fits,
// cp.async copies (16 bytes: two elements adjacent in the source; 8 bytes for
// plain rows on odd addresses) fill a block of 128 rows x 32 values, copy
// u = lt + 64 i by loader thread lt. Offsets of sources are in elements and
// add up, offsets into the block are in bytes and combine by XOR. With boxes
// one thread issues two copies or one a block, where 64 threads spent 2000
// cycles issuing 32 each: (65536, 256, 256) x 4 323 -> 308 us, (3001, 690,
// 1100) 63 -> 42 us.
struct AGather {
  static constexpr int kBits = 26;
  std::uint64_t copy_src[32];   // copy i's part of the source offset
  std::uint64_t lane_src[6];    // part of each bit of lt
  std::uint64_t tile_src[kBits];   // of each bit of the row-tile number (not plain)
  std::uint64_t block_src[kBits];  // of each bit of the 32-value block number (not plain)
  std::uint32_t copy_dst[32];   // the same two in the block
  std::uint32_t lane_dst[6];
  std::uint32_t row_at[7];      // of each bit of a row, where its values are read
  std::uint32_t value_at[32];   // of each value of a row
  std::int32_t plain;           // rows of k values: tiles and blocks by arithmetic
  std::int32_t pairs;           // values 2 j and 2 j + 1 of a row are adjacent
  std::int32_t copies_real;     // copies i below this exist (16 when k = 16)
  // TMA boxes instead of copies. Plain: two boxes of 128 rows x 16 values.
  // Otherwise one box whose dimensions are the 16 lowest digits' values (rows
  // of 128 bytes), then `runs` of neighbouring digits.
  std::int32_t boxes;
  std::int32_t run_bits[3];
  std::uint64_t run_src[3];     // source offset of a run's lowest digit
  std::int32_t nbits;           // digits of the source (not plain)
};
// A as m rows of k values; `aligned`: base, row and batch strides are
// multiples of 16 bytes.
AGather make_a_rows(std::size_t k, bool aligned);
// A as a tensor of 2^nbits elements whose digit p goes to digit perm[p] of
// the row-major m x k operand (k = 2^j >= 16, m >= 128): the product reads it
// where it lies. False when the permutation cannot be read that way (the
// source's low digits outside a block); the base and the batch stride have to
// be multiples of 16 bytes.
bool make_a_gather(int nbits, const std::uint8_t* perm, std::size_t m, std::size_t k, AGather* g);
// The gather's copies and reads on host buffers, block by block, with bounds
// checks: dst is the m x k operand the product sees. Tests use it.
void a_gather_on_host(const AGather& g, std::size_t m, std::size_t k, const float2* src, float2* dst);

// Whether the direct product of m rows and k terms runs on pairs of CTAs
// (BF16x3: whether it runs).
bool tc_direct_pair(SplitKind kind, std::size_t m, std::size_t k);
// fp32 elements that launch_cgemm_direct's workspace takes per batch entry.
std::size_t tc_direct_workspace_elems(SplitKind kind, std::size_t n, std::size_t k);
// The split product with A split inside the kernel: A is read as
// complex64 through `gather` (3xFP16: every 32 values of a row scaled by their
// own power of two), and no A planes exist in memory. cfg.chunk 2 (a TMEM chunk
// is one of A's blocks); cfg.variant is ignored. With `watch` != 0 err[4] takes
// that value when a sum is an infinity or NaN.
void launch_cgemm_direct(SplitKind kind, const float2* A, const AGather& gather, const float2* B, BLayout b_layout,
                         float2* C, std::size_t m, std::size_t n, std::size_t k, std::uint64_t ac_stride,
                         std::uint64_t b_stride, int batch, float* workspace, int* err, const TcConfig& cfg,
                         cudaStream_t s, int watch = 0);

// The same product with BF16x3 planes: x = b0 + b1 + b2 in BF16 (no
// scaling: BF16 has the FP32 exponent range), six products per real
// product (x0y0, x0y1, x1y0, x0y2, x1y1, x2y0) on kind::f16 tensor cores.
// Single-CTA kernel; cfg.variant is ignored.
void launch_cgemm_bf16x3(const float2* A, const float2* B, BLayout b_layout, float2* C, std::size_t m,
                         std::size_t n, std::size_t k, std::uint64_t ac_stride, std::uint64_t b_stride, int batch,
                         float* workspace, int* err, const TcConfig& cfg, cudaStream_t s);

}  // namespace qfx
