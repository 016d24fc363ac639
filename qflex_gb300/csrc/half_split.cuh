// Splitting FP32 values into FP16 hi + lo and three BF16 pieces, rounding them
// to TF32.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

namespace qfx {
namespace {

__device__ __forceinline__ float tf32_rn(float x) {
  std::uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// hi = fp16(x), lo = fp16(x - hi), both to nearest, for two values: a packs
// into the low halves, b into the high ones. x - hi is one mixed-precision FMA
// (hi * -1 + x, exact) instead of a conversion back to FP32 and a subtraction:
// 18 instead of 10 pairs per cycle and SM.
__device__ __forceinline__ void split_pair(float a, float b, std::uint32_t& hi, std::uint32_t& lo) {
  asm("{\n .reg .b16 l, h, m;\n .reg .f32 x, y;\n"
      " cvt.rn.f16x2.f32 %0, %3, %2;\n mov.b32 {l, h}, %0;\n mov.b16 m, 0xBC00;\n"
      " fma.rn.f32.f16 x, l, m, %2;\n fma.rn.f32.f16 y, h, m, %3;\n cvt.rn.f16x2.f32 %1, y, x;\n}\n"
      : "=&r"(hi), "=r"(lo)
      : "f"(a), "f"(b));
}

// x = p0 + p1 + p2 in BF16, each piece what is left rounded to nearest, for two
// values: a packs into the low halves, b into the high ones.
__device__ __forceinline__ void split_bf16(float a, float b, std::uint32_t& p0, std::uint32_t& p1, std::uint32_t& p2) {
  const __nv_bfloat162 h0 = __floats2bfloat162_rn(a, b);
  const float2 f0 = __bfloat1622float2(h0), r0 = make_float2(a - f0.x, b - f0.y);
  const __nv_bfloat162 h1 = __floats2bfloat162_rn(r0.x, r0.y);
  const float2 f1 = __bfloat1622float2(h1);
  const __nv_bfloat162 h2 = __floats2bfloat162_rn(r0.x - f1.x, r0.y - f1.y);
  p0 = reinterpret_cast<const std::uint32_t&>(h0);
  p1 = reinterpret_cast<const std::uint32_t&>(h1);
  p2 = reinterpret_cast<const std::uint32_t&>(h2);
}

}  // namespace
}  // namespace qfx
