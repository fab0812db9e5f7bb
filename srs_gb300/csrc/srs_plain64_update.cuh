// srs_plain64_update.cuh — pieces of the FP64 element update shared by the
// one-launch-per-step kernel (k_plain64.cu) and the looping kernel
// (k_plain_loop.cu).
//
// Every piece keeps the reference's association order and the units that
// include this file are compiled with -fmad=false, so results are the
// reference's bit for bit.  An FP64 warp instruction occupies its pipe for 64
// cycles on this part (two lanes a cycle and SM), whatever else the kernel
// does, so the pieces avoid FP64 instructions whose result is known: constant
// factors are formed on the host in the same operations, divisions by a
// constant use its reciprocal, buffers that are absent are not divided by, and
// signs, zeros and non-finite values are tested on the bits.
#pragma once
#include "srs_engine.h"

namespace srs {

__device__ __forceinline__ uint64_t bits64(double x) { return (uint64_t)__double_as_longlong(x); }

__device__ __forceinline__ bool finite64(double x) {
  return ((bits64(x) >> 52) & 0x7ff) != 0x7ff;
}

// x + 0.0: x, and +0 for -0
__device__ __forceinline__ double plus_zero(double x) {
  return bits64(x) == 0x8000000000000000ull ? 0.0 : x;
}

// a / b for a constant b with y = 1 / b rounded to nearest: the quotient a y is
// corrected twice by its remainder; after the first correction it is within
// one ulp, so the second one rounds it correctly (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990).  The
// operands' exponents are kept away from the ends of the range (y is zero
// where b's is not: the division proper then).
__device__ __forceinline__ double div_by_const(double a, double b, double y) {
  const uint32_t e = (uint32_t)(bits64(a) >> 52) & 0x7ff;
  if (e - 523u > 1000u || y == 0.0) return a / b;  // |a| outside 2^-500 .. 2^500
  double q = __dmul_rn(a, y);
  q = __fma_rn(__fma_rn(-b, q, a), y, q);
  return __fma_rn(__fma_rn(-b, q, a), y, q);
}

// Diffusion of one species (cpu/RunSimulation.cpp:44-67):
// D (c a0 + s1 a1 + s2 a2 + s3 a3 + s4 a4) + br, left to right.
__device__ __forceinline__ double diffuse64(double D, double c, double s1, double s2, double s3,
                                            double s4, const double* a, double br) {
  return D * (c * a[0] + s1 * a[1] + s2 * a[2] + s3 * a[3] + s4 * a[4]) + br;
}

// Buffer reaction kon (B - b) c - koff b (cpu/RunSimulation.cpp:78-118)
__device__ __forceinline__ double react64(double kon, double B, double koff, double b, double c) {
  return kon * (B - b) * c - koff * b;
}

// SERCA uptake (cpu/RunSimulation.cpp:83-91); its K_sr terms come from the host
// (plain64_consts).
__device__ __forceinline__ double serca64(const Plain64Args& a, double c) {
  double K_i = div_by_const(c, a.p[49], a.inv_kdi);
  K_i = K_i * K_i;
  const double D = a.sd0 + K_i * a.sd1 + K_i * K_i * a.sd2;
  const double v = (K_i * K_i * 3.24873e12 + K_i * a.sn1 - a.sn0) / D;
  return (2e-3) * v * a.p[51];
}

// UpdateFastBuffer (cpu/RunSimulation.cpp:15-22).  Without either buffer B is
// exactly one (unless a denominator vanishes).
__device__ __forceinline__ double fast_buffer64(const Plain64Args& a, double b_ca, double c,
                                                double bhi, double blo) {
  const double khi = a.p[28], klo = a.p[30];
  if (((bits64(bhi) | bits64(blo)) << 1) == 0 && bits64(c) != bits64(-khi) && bits64(c) != bits64(-klo))
    return b_ca;
  const double B = 1 + (bhi * khi / ((khi + c) * (khi + c))) + (blo * klo / ((klo + c) * (klo + c)));
  return b_ca / B;
}

}  // namespace srs
