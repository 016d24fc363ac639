// One element of a qubit column's 2D tensor, shared by the flatten kernel and
// the one-kernel program, and the complex64 helpers.
#pragma once

#include <cstdint>

#include "kernels.h"

namespace qfx {
namespace {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 c) {
  c.x = fmaf(a.x, b.x, c.x);
  c.x = fmaf(-a.y, b.y, c.x);
  c.y = fmaf(a.x, b.y, c.y);
  c.y = fmaf(a.y, b.x, c.y);
  return c;
}

// ---------------------------------------------------------------------------
// Column flatten.
// ---------------------------------------------------------------------------
// Float-float numbers (an unevaluated sum h + l of two floats, ~44
// significant bits) built from the classic error-free transformations:
// Knuth's two-sum and the FMA-based exact product.
struct ff {
  float h, l;
};
__device__ __forceinline__ ff ff_add(ff a, ff b) {
  const float s = a.h + b.h;
  const float bb = s - a.h;
  float e = (a.h - (s - bb)) + (b.h - bb);
  e += a.l + b.l;
  const float h = s + e;
  return {h, e - (h - s)};
}
__device__ __forceinline__ ff ff_mul(ff a, ff b) {
  const float p = a.h * b.h;
  float e = fmaf(a.h, b.h, -p);
  e = fmaf(a.h, b.l, e);
  e = fmaf(a.l, b.h, e);
  const float h = p + e;
  return {h, e - (h - p)};
}
__device__ __forceinline__ ff ff_neg(ff a) { return {-a.h, -a.l}; }
struct cff {
  ff re, im;
};
__device__ __forceinline__ cff cff_mul(cff a, cff b) {
  return {ff_add(ff_mul(a.re, b.re), ff_neg(ff_mul(a.im, b.im))),
          ff_add(ff_mul(a.re, b.im), ff_mul(a.im, b.re))};
}
__device__ __forceinline__ cff cff_add(cff a, cff b) { return {ff_add(a.re, b.re), ff_add(a.im, b.im)}; }
__device__ __forceinline__ cff cff_load(const float2* hi, const float2* lo, std::uint32_t i) {
  const float2 h = hi[i], l = lo[i];
  return {{h.x, l.x}, {h.y, l.y}};
}

// Element e of a column's 2D tensor: <bit| G_K ... G_1 |one> with every
// two-qubit half reading its virtual digit of e. Plain FP32 repeats the
// reference's complex<float> arithmetic on its float gate constants; the
// compensated form carries float-float values and gate constants (hi + lo
// of the double-precision gate) and rounds once at the end.
// U elements of a column at a time: their chains are independent and share the
// step descriptors. out[u] gets the component `bit(u)` selects.
template <bool kCompensated, int U, typename E, typename Bit>
__device__ __forceinline__ void column_elements(const ColumnDesc& cd, const StepDesc* steps, const float2* mats,
                                                const float2* mats_lo, bool one, const E (&e)[U],
                                                float2 (&out)[U], Bit bit) {
  float2 p0[U], p1[U];
  cff f0[U], f1[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    p0[u] = make_float2(one ? 0.f : 1.f, 0.f);
    p1[u] = make_float2(one ? 1.f : 0.f, 0.f);
    f0[u] = {{p0[u].x, 0.f}, {0.f, 0.f}};
    f1[u] = {{p1[u].x, 0.f}, {0.f, 0.f}};
  }
  for (std::uint32_t s = cd.step_begin; s < cd.step_end; ++s) {
    const StepDesc sd = steps[s];
    const bool half = sd.kind == 2;
    const std::uint32_t row = half ? 2 * sd.V : 2;  // distance between input rows of the gate data
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const std::uint32_t g = sd.mat + (half ? 2 * (std::uint32_t(e[u] >> sd.shift) & (sd.V - 1)) : 0);
      if constexpr (kCompensated) {
        const cff q0 = cff_add(cff_mul(f0[u], cff_load(mats, mats_lo, g)),
                               cff_mul(f1[u], cff_load(mats, mats_lo, g + row)));
        const cff q1 = cff_add(cff_mul(f0[u], cff_load(mats, mats_lo, g + 1)),
                               cff_mul(f1[u], cff_load(mats, mats_lo, g + row + 1)));
        f0[u] = q0;
        f1[u] = q1;
      } else {
        const float2 q0 = cfma(p1[u], mats[g + row], cmul(p0[u], mats[g]));
        const float2 q1 = cfma(p1[u], mats[g + row + 1], cmul(p0[u], mats[g + 1]));
        p0[u] = q0;
        p1[u] = q1;
      }
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if constexpr (kCompensated) {
      p0[u] = make_float2(f0[u].re.h + f0[u].re.l, f0[u].im.h + f0[u].im.l);
      p1[u] = make_float2(f1[u].re.h + f1[u].re.l, f1[u].im.h + f1[u].im.l);
    }
    out[u] = bit(u) ? p1[u] : p0[u];
  }
}

}  // namespace
}  // namespace qfx
