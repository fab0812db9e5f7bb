// srs_comp.h — compact storage of the Euler compensation terms.
//
// The FP32 engines keep, per element and species, the rounding error c of
// the last compensated Euler update t = u + y (Kahan: c = (t - u) - y), and
// subtract it from the next increment.  |c| <= ulp(t) / 2.  The FP32
// engines store c as an IEEE half of c * 2^24 (round to nearest even,
// saturated to the largest finite half; a NaN stays a NaN): the plain engine
// in HBM, the resident engine in shared memory, where the smaller footprint
// lets more CTAs share an SM.  10 bytes per element for the five species
// instead of 20:
//   q = half(clamp(c * 2^24, +-65504)),   c' = float(q) * 2^-24.
// Concentrations stay below 2^15 uM, so |c * 2^24| <= 2^15 and the clamp only
// matters for a diverged state; c' keeps 11 significant bits of c (the
// accumulator keeps about 35), down to |c| = 2^-38 (c * 2^24 >= 2^-14, the
// half's normal range), i.e. for states above about 6e-5 uM.  Both scalings
// are exact powers of two, and the conversion is IEEE round-to-nearest-even
// (the device's conversion; the CPU oracle restates it with the compiler's
// _Float16), and reading back is exact on host and device alike.
#pragma once
#include <stdint.h>

namespace srs {

constexpr float kCompScale = 16777216.0f;          // 2^24
constexpr float kCompInvScale = 1.0f / 16777216.0f;  // 2^-24

#ifdef __CUDACC__
// Device side.  cvt.rn.satfinite rounds to nearest even and saturates to
// +-65504 (a NaN stays a NaN): the clamp of the encoding, then the rounding;
// two species per conversion (the scalings are exact: powers of two).
__device__ __forceinline__ uint32_t comp_encode2(float lo, float hi) {
  uint32_t q;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(q) : "f"(hi * kCompScale), "f"(lo * kCompScale));
  return q;
}
// the two halves of q as floats (exact), not yet scaled
__device__ __forceinline__ float2 comp_halves2(uint32_t q) {
  float lo, hi;
  asm("{\n\t.reg .f16 l, h;\n\tmov.b32 {l, h}, %2;\n\tcvt.f32.f16 %0, l;\n\tcvt.f32.f16 %1, h;\n\t}"
      : "=f"(lo), "=f"(hi)
      : "r"(q));
  return make_float2(lo, hi);
}
__device__ __forceinline__ float2 comp_decode2(uint32_t q) {
  const float2 h = comp_halves2(q);
  return make_float2(h.x * kCompInvScale, h.y * kCompInvScale);
}

// the stored layout: ushort4 (x, y, z, w) of the four mobile species (read
// and written as one 8-byte word), ushort of the immobile buffer
__device__ __forceinline__ float4 comp_load4(const ushort4* p) {
  const uint2 q = *reinterpret_cast<const uint2*>(p);
  const float2 a = comp_decode2(q.x), b = comp_decode2(q.y);
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void comp_store4(ushort4* p, float4 c) {
  *reinterpret_cast<uint2*>(p) = make_uint2(comp_encode2(c.x, c.y), comp_encode2(c.z, c.w));
}
// The same with the scalings as packed FP32 multiplies (identical values):
// faster in the plain adjoint's reverse step (0.831 against 0.846 ms per
// large-mesh step), slower in the 40-register forward update (0.454 against
// 0.439 ms), which uses the scalar forms above.
__device__ __forceinline__ float4 comp_load4_x2(const ushort4* p) {
  const uint2 q = *reinterpret_cast<const uint2*>(p);
  const float2 s = make_float2(kCompInvScale, kCompInvScale);
  const float2 a = __fmul2_rn(comp_halves2(q.x), s), b = __fmul2_rn(comp_halves2(q.y), s);
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void comp_store4_x2(ushort4* p, float4 c) {
  const float2 s = make_float2(kCompScale, kCompScale);
  const float2 a = __fmul2_rn(make_float2(c.x, c.y), s), b = __fmul2_rn(make_float2(c.z, c.w), s);
  uint32_t qa, qb;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(qa) : "f"(a.y), "f"(a.x));
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(qb) : "f"(b.y), "f"(b.x));
  *reinterpret_cast<uint2*>(p) = make_uint2(qa, qb);
}
__device__ __forceinline__ float comp_load1(unsigned short q) {
  float v;
  asm("{\n\t.reg .f16 h;\n\tmov.b16 h, %1;\n\tcvt.f32.f16 %0, h;\n\t}" : "=f"(v) : "h"(q));
  return v * kCompInvScale;
}
__device__ __forceinline__ unsigned short comp_store1(float c) {
  unsigned short q;
  asm("cvt.rn.satfinite.f16.f32 %0, %1;" : "=h"(q) : "f"(c * kCompScale));
  return q;
}
// (double)f on the integer units: conversions share the FP64 pipe, which issues
// one warp instruction in 64 cycles on sm_103a (and a conversion on a branch that
// the compiler turns into a predicate is issued all the same).
__device__ __forceinline__ double widen(float f) {
  const uint32_t b = __float_as_uint(f);
  uint32_t m = b & 0x7fffffffu;
  uint32_t rebias = m >= 0x7f800000u ? 0x70000000u : 0x38000000u;  // 1151 (infinity, NaN) or 896 exponents
  if (m < 0x00800000u) {  // zero, or a denormal: normalise
    const int s = __clz((int)m) - 8;
    m = m ? m << s : 0u;
    rebias = m ? rebias - ((uint32_t)s << 20) : 0u;
  }
  return __hiloint2double((int)((b & 0x80000000u) | ((m >> 3) + rebias)), (int)(m << 29));
}
#endif

}  // namespace srs
