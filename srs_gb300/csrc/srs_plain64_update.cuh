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

// ---- the update dealt to four warps ----------------------------------------------
// 32 elements, one per lane of each of four warps; each warp has its share (its
// "role"), because an FP64 warp instruction occupies a quarter of an SM for 64
// cycles: 112 of them in one warp are 3.5 us, dealt to four 1.2.
//   role 0: Ca -- diffusion; after the others, the sums of Ca's rate in the
//           reference's order, channel fluxes, rapid buffer, Euler;
//   role 1: troponin C or calsequestrin, SERCA;  role 2: dye and ATP;
//   role 3: calmodulin.
struct Geo64 {
  double ac[5];
  int n1, n2, n3, n4, fl;
};
__device__ __forceinline__ Geo64 geometry64(const Plain64Args& a, int e) {
  Geo64 g;
#pragma unroll
  for (int q = 0; q < 5; ++q) g.ac[q] = __ldg(a.aij + 5 * (size_t)e + q);
  const int32_t* nn = a.nij + 4 * (size_t)e;
  g.n1 = __ldg(nn);
  g.n2 = __ldg(nn + 1);
  g.n3 = __ldg(nn + 2);
  g.n4 = __ldg(nn + 3);
  g.fl = __ldg(a.flags + e);
  return g;
}
// First of the species whose value a role holds in x0 and, roles 1 and 2, x1.
__device__ __forceinline__ int role64_x0(int role) { return role == 0 ? 0 : role == 1 ? 3 : role == 2 ? 5 : 2; }
__device__ __forceinline__ int role64_x1(int role) { return role == 1 ? 4 : 1; }

// A role's share of one element from the state src (read past L1) and the
// element's Ca c.  Returns Ca's diffusion (role 0); advances x0, x1 (the
// others) and leaves the reactions in rate: immobile buffer, SERCA, dye, ATP,
// CMDN.
__device__ __forceinline__ double role64(const Plain64Args& a, int role, const Geo64& g, int e, int lane,
                                         const double* src, double c, double& x0, double& x1,
                                         double (*rate)[32]) {
  const double* p = a.p;
  const double dt = a.P.dt;
  const size_t n = a.N;
  const bool jsr = g.fl & 1, trop = !jsr && (g.fl & 2);
  auto diffuse = [&](const double* f, double D, double x, double br) {
    return diffuse64(D, x, __ldcg(f + g.n1), __ldcg(f + g.n2), __ldcg(f + g.n3), __ldcg(f + g.n4), g.ac, br);
  };
  if (role == 0) return diffuse(src, p[5], c, __ldg(a.br + e));
  if (role == 1) {
    double r = 0.0, y0 = plus_zero(x0), y1 = plus_zero(x1);
    if (trop) {
      r = react64(p[26], p[24], p[25], x0, c);
      rate[1][lane] = serca64(a, c);
      y0 = x0 + r * dt;
    } else if (jsr) {
      r = react64(p[39], p[34], p[40], x1, c);
      y1 = x1 + r * dt;
    }
    rate[0][lane] = r;
    x0 = y0;
    x1 = y1;
  } else if (role == 2) {
    double b_dye = diffuse(src + 5 * n, p[11], x0, __ldg(a.br + 3 * n + e));
    double b_atp = diffuse(src + n, p[7], x1, __ldg(a.br + n + e));
    if (!jsr) {
      const double rd = react64(p[33], p[31], p[32], x0, c), ra = react64(p[20], p[18], p[19], x1, c);
      rate[2][lane] = rd;
      rate[3][lane] = ra;
      b_dye += rd;
      b_atp += ra;
    }
    x0 = x0 + b_dye * dt;
    x1 = x1 + b_atp * dt;
  } else {
    double b_cmdn = diffuse(src + 2 * n, p[8], x0, __ldg(a.br + 2 * n + e));
    if (!jsr) {
      const double rm = react64(p[23], p[21], p[22], x0, c);
      rate[4][lane] = rm;
      b_cmdn += rm;
    }
    x0 = x0 + b_cmdn * dt;
  }
  return 0.0;
}
// Ca's rate with the reactions added to its diffusion b_ca (role 0).
__device__ __forceinline__ double sum64(const Plain64Args& a, int fl, int lane, double c, double b_ca,
                                        double (*rate)[32]) {
  if (!(fl & 1)) {
    if (fl & 2) {
      b_ca += -rate[0][lane];
      b_ca -= rate[1][lane];
    }
    b_ca += -rate[2][lane];
    b_ca += -rate[3][lane];
    b_ca += -rate[4][lane];
  } else {
    b_ca += -rate[0][lane];
    b_ca += (a.nsr - c) * a.p[36];
  }
  return b_ca;
}

}  // namespace srs
