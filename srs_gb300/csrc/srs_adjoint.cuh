// srs_adjoint.cuh — per-element pieces of the reverse sweep shared by the
// adjoints of the resident and the plain FP32 engines.
#pragma once
#include "srs_engine.h"
#include "srs_fp32_update.cuh"

namespace srs {

// A thread's parameter gradients.  The sums of the two packed halves of an
// element, (Ca, ATP) and (CMDN, dye), are packed too.
struct AdjGrad {
  float2 d_xy, d_zw;      // diffusion coefficients
  float2 on_zw, off_zw;   // kon, koff of (CMDN, dye)
  float on_atp, off_atp, on_trpn, off_trpn, on_csqn, off_csqn;
  float v_ryr, a_p, b_tot_sl, k_d_sl;
  __device__ __forceinline__ void clear() {
    d_xy = d_zw = on_zw = off_zw = make_float2(0.0f, 0.0f);
    on_atp = off_atp = on_trpn = off_trpn = on_csqn = off_csqn = v_ryr = a_p = b_tot_sl = k_d_sl = 0.0f;
  }
  __device__ __forceinline__ void get(float (&g)[SRS_N_ADJ]) const {
    g[SRS_ADJ_D_CA] = d_xy.x;
    g[SRS_ADJ_D_ATP] = d_xy.y;
    g[SRS_ADJ_D_CMDN] = d_zw.x;
    g[SRS_ADJ_D_DYE] = d_zw.y;
    g[SRS_ADJ_K_ON_CMDN] = on_zw.x;
    g[SRS_ADJ_K_ON_DYE] = on_zw.y;
    g[SRS_ADJ_K_OFF_CMDN] = off_zw.x;
    g[SRS_ADJ_K_OFF_DYE] = off_zw.y;
    g[SRS_ADJ_K_ON_ATP] = on_atp;
    g[SRS_ADJ_K_OFF_ATP] = off_atp;
    g[SRS_ADJ_K_ON_TRPN] = on_trpn;
    g[SRS_ADJ_K_OFF_TRPN] = off_trpn;
    g[SRS_ADJ_K_ON_CSQN] = on_csqn;
    g[SRS_ADJ_K_OFF_CSQN] = off_csqn;
    g[SRS_ADJ_V_RYR] = v_ryr;
    g[SRS_ADJ_A_P] = a_p;
    g[SRS_ADJ_B_TOT_SL] = b_tot_sl;
    g[SRS_ADJ_K_D_SL] = k_d_sl;
  }
};

// Compensated update of lambda, s += dt o (Kahan), in negated form: ny = -y,
// t = s - ny, c = (t - s) + ny.
__device__ __forceinline__ void kadd(float& s, float& c, float ndt, float o) {
  const float ny = fmaf(ndt, o, c);
  const float t = s - ny;
  c = (t - s) + ny;
  s = t;
}
__device__ __forceinline__ void kadd(float2& s, float2& c, float2 ndt, float2 o) {
  const float2 ny = p_fma(ndt, o, c);
  const float2 t = p_sub(s, ny);
  c = p_add(p_sub(t, s), ny);
  s = t;
}

// Sums of N values over the warp: lane p returns the sum of value p (lanes from N
// on: anything).  Each exchange halves the values a lane carries (of 32, the ones
// from N on zero), 31 shuffles for 18 values instead of five a value; the sum of
// each value is taken over the same tree (lanes 16, 8, 4, 2, 1 apart), so it is the
// same number.
template <int N>
__device__ __forceinline__ float warp_sums(const float (&g)[N], int lane) {
  float v[32];
#pragma unroll
  for (int p = 0; p < 32; ++p) v[p] = p < N ? g[p] : 0.0f;
#pragma unroll
  for (int h = 16; h >= 1; h >>= 1) {
    const bool up = (lane & h) != 0;
#pragma unroll
    for (int p = 0; p < h; ++p) {
      if (p >= N) continue;  // nothing in either half
      const float keep = up ? v[p + h] : v[p], give = up ? v[p] : v[p + h];
      v[p] = keep + __shfl_xor_sync(0xffffffffu, give, h);
    }
  }
  return v[0];
}

// One buffer reaction r = kon (B - b) c - koff b of an element: adds its
// Jacobian-transpose terms and its kon/koff gradient terms.
__device__ __forceinline__ void adj_buffer(const Consts32& k, const AdjConsts& ak, int q, float c,
                                           float ub, float lb, float w, float& ob, float& oc,
                                           float& dG, float& g_on, float& g_off) {
  const float free = k.bfree[q] - ub;
  const float alpha = k.kon[q] * free;
  const float beta = fmaf(k.kon[q], c, k.koff[q]);
  dG -= alpha;            // dF_Ca/dCa (times B)
  ob = fmaf(beta, w - lb, ob);  // dF_Ca/db * lambda_Ca + dF_b/db * lambda_b
  oc = fmaf(alpha, lb, oc);      // dF_b/dCa * lambda_b
  const float d = lb - w;
  g_on = fmaf(d * free, c, g_on);                  // dr/dkon = (B - b) c
  g_off = fmaf(-d, ak.brest[q] + ub, g_off);       // dr/dkoff = -b
}

// 1 / B(c), B the rapid-buffer factor of UpdateFastBuffer
// (cpu/RunSimulation.cpp:15-22).
__device__ __forceinline__ float sl_inv_factor(const Consts32& k, float bsl, float c) {
  if (bsl == 0.0f) return 1.0f;
  const float kc = k.khi + c;
  const float kc2 = kc * kc;
  return __fdividef(kc2, kc2 + bsl);
}

// The reverse-step terms of one element but its channels and the rapid buffer:
// the transposed diffusion S = sum_k aT_k lambda(nb_k) - (sum_k a_k) lambda(self)
// over the neighbours' slots n0..n3, the diffusion-coefficient gradients, the
// buffer reactions and SERCA (cpu/RunSimulation.cpp:70-118), and the JSR
// refill.  x/xim: state x_{n-1}; me: the element's published slot (lambda_Ca / B,
// lambda_ATP, lambda_CMDN, lambda_dye); li: lambda of the immobile buffer.
// Returns the adjoint rates (Ca's before the rapid-buffer factor) and dG,
// d(Ca rate)/dCa times B.  What the species share is done two at a time, as in
// the forward update (tet_update_x2).
struct AdjTerms {
  float2 oxy, ozw;  // (Ca, ATP), (CMDN, dye)
  float oi, dG, c;
};
__device__ __forceinline__ AdjTerms adj_local(const Consts32& k, const AdjConsts& ak, const float4& x,
                                              float xim, const float4& me, float li, bool jsr,
                                              bool trpn, const float4& at, float sa, const float4& n0,
                                              const float4& n1, const float4& n2, const float4& n3, AdjGrad& g) {
  float2 b = p_bc(at.x);
  float2 Sxy = p_mul(b, lo2(n0)), Szw = p_mul(b, hi2(n0));
  b = p_bc(at.y);
  Sxy = p_fma(b, lo2(n1), Sxy);
  Szw = p_fma(b, hi2(n1), Szw);
  b = p_bc(at.z);
  Sxy = p_fma(b, lo2(n2), Sxy);
  Szw = p_fma(b, hi2(n2), Szw);
  b = p_bc(at.w);
  Sxy = p_fma(b, lo2(n3), Sxy);
  Szw = p_fma(b, hi2(n3), Szw);
  b = p_bc(-sa);
  Sxy = p_fma(b, lo2(me), Sxy);
  Szw = p_fma(b, hi2(me), Szw);
  // D gradients: sum_j lambda_j (L u)_j = sum_j u_j (L^T lambda)_j
  g.d_xy = p_fma(lo2(x), Sxy, g.d_xy);
  g.d_zw = p_fma(hi2(x), Szw, g.d_zw);
  AdjTerms o;
  o.oxy = p_mul(make_float2(k.D[0], k.D[1]), Sxy);
  o.ozw = p_mul(make_float2(k.D[2], k.D[3]), Szw);
  o.oi = 0.0f;
  const float w = me.x;
  o.dG = 0.0f;
  const float c = (jsr ? k.c0j : k.c0) + x.x;
  o.c = c;
  if (!jsr) {
    // adj_buffer of CMDN and dye
    const float2 kon = make_float2(k.kon[2], k.kon[0]);
    const float2 free = p_sub(make_float2(k.bfree[2], k.bfree[0]), hi2(x));
    const float2 alpha = p_mul(kon, free);
    const float2 beta = p_fma(kon, p_bc(c), make_float2(k.koff[2], k.koff[0]));
    const float2 nd = p_sub(p_bc(w), hi2(me));
    o.ozw = p_fma(beta, nd, o.ozw);
    g.on_zw = p_fma(p_mul(nd, free), p_bc(-c), g.on_zw);
    g.off_zw = p_fma(nd, p_add(make_float2(ak.brest[2], ak.brest[0]), hi2(x)), g.off_zw);
    o.dG -= alpha.y;
    o.oxy.x = fmaf(alpha.y, me.w, o.oxy.x);
    adj_buffer(k, ak, 1, c, x.y, me.y, w, o.oxy.y, o.oxy.x, o.dG, g.on_atp, g.off_atp);
    o.dG -= alpha.x;
    o.oxy.x = fmaf(alpha.x, me.z, o.oxy.x);
    if (trpn) {
      adj_buffer(k, ak, 3, c, xim, li, w, o.oi, o.oxy.x, o.dG, g.on_trpn, g.off_trpn);
      // SERCA v(Ki), Ki = (c / K_D_i)^2 (cpu/RunSimulation.cpp:83-91)
      float Ki = c * k.inv_kdi;
      Ki = Ki * Ki;
      const float den = fmaf(Ki * Ki, k.sd2, fmaf(Ki, k.sd1, k.sd0));
      const float num = fmaf(Ki * Ki, 3.24873e12f, fmaf(Ki, k.sn1, -k.sn0));
      const float iden = __fdividef(1.0f, den);
      const float v = num * iden;
      const float dnum = fmaf(2.0f * Ki, 3.24873e12f, k.sn1);
      const float dden = fmaf(2.0f * Ki, k.sd2, k.sd1);
      const float dv = (dnum - v * dden) * iden * (2.0f * c * k.inv_kdi * k.inv_kdi);
      o.dG = fmaf(-k.serca_scale, dv, o.dG);
      g.a_p = fmaf(-w * ak.serca_per_ap, v, g.a_p);
    }
  } else {
    adj_buffer(k, ak, 4, c, xim, li, w, o.oi, o.oxy.x, o.dG, g.on_csqn, g.off_csqn);
    o.dG -= k.refill_v;
  }
  return o;
}

// dG into lambda_Ca's rate, then the rapid SL buffer (cpu/RunSimulation.cpp:
// 15-22): F_Ca = G / B(c), so -G B'(c) / B^2 lambda_Ca = 2 bsl G w / (B kc^3),
// with its B_TOT_SL and K_D_SL gradient terms.  w: lambda_Ca / B.
__device__ __forceinline__ void adj_rapid(const Consts32& k, const AdjConsts& ak, float bsl, float c,
                                          float G, float w, float dG, float& oc, AdjGrad& g) {
  oc = fmaf(dG, w, oc);
  if (bsl != 0.0f) {
    const float kc = k.khi + c;
    const float ikc = __fdividef(1.0f, kc);
    const float bk2 = bsl * ikc * ikc;           // B - 1
    const float GB = __fdividef(G, 1.0f + bk2);  // G / B
    const float t3 = GB * bk2 * ikc;             // G bsl / (B kc^3)
    oc = fmaf(2.0f * t3, w, oc);
    g.b_tot_sl = fmaf(-w * GB, bk2 * ak.inv_btot_sl, g.b_tot_sl);
    g.k_d_sl = fmaf(-w * t3, (c - k.khi) * ak.inv_khi, g.k_d_sl);
  }
}

}  // namespace srs
