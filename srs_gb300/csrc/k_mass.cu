// k_mass.cu — total Ca per compartment, accumulated in FP64.
//
// Total Ca of an element (uM): free Ca + Ca bound to every buffer state
// variable (ATP, calmodulin, troponin C, dye in the cytosol; calsequestrin in
// the JSR) + Ca bound to the rapid sarcolemmal buffers of UpdateFastBuffer
// (cpu/RunSimulation.cpp:15-22), which are at equilibrium with the free Ca:
// b_hi c / (K_hi + c) + b_lo c / (K_lo + c).  The rapid-buffer Euler form
// dc/dt = G / B with B = 1 + d(bound)/dc makes this the conserved quantity
// of the reaction and diffusion terms.  Per realization the kernel returns
// sum_j V0_j total_j (uM um^3) over the cytosol and over the JSR, summed in
// double precision whatever the precision of the state.
#include "srs_comp.h"
#include "srs_engine.h"
#include "srs_math.h"

namespace srs {

// Rapid-buffer part b c / (K + c).
__device__ __forceinline__ double sl_bound(double b, double K, double c) { return b * c / (K + c); }
// c at which a buffer of no capacity binds nothing: finite, not -K (tests on the
// bits: the FP64 pipe issues one warp instruction in 64 cycles here)
__device__ __forceinline__ bool plain_ca(const MassArgs& a, double c) {
  return (__double2hiint(c) & 0x7ff00000) != 0x7ff00000 && __double_as_longlong(c) != __double_as_longlong(-a.khi) &&
         __double_as_longlong(c) != __double_as_longlong(-a.klo);
}

// The FP32 engines' state of one element: deviation less compensation, widened
// on the integer units.
__device__ __forceinline__ double dev_ca(const MassArgs& a, size_t o) {
  const float c = a.CMq ? comp_load4(a.CMq + o).x : a.CM[o].x;
  return widen(a.M[o].x) - widen(c);
}

// Grid: x over blocks of one realization's elements, y over realizations.  A
// block per realization alone leaves a few large realizations on a few SMs.
// The bound is the FP64 pipe, so an FP32 engine's element takes twelve of its
// instructions: the five deviations less their compensation, their sum on top of
// the summed resting values, Ca for its test and the volume's multiply-add.  The
// rapid buffers, a division each for the one element in ten at the membrane,
// follow over the list of those, so that whole warps divide.
// 32 x 542,376 elements: 11.4 ms a call by one block a realization, 1.25 with
// the split, 0.49 with this count and list.  Each block writes its two sums;
// k_total_ca_sum adds them in order (a launch that one block a realization spares:
// 384 elements 30 us a call with it, 28.7 without).
__global__ void __launch_bounds__(256) k_total_ca(MassArgs a) {
  const int r = blockIdx.y;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  const double* S = a.S64 ? a.S64 + (size_t)r * 6 * a.n_state : nullptr;
  const size_t ro = (size_t)r * a.n_state;
  double acc[2] = {0.0, 0.0};
  for (int e = t0; e < a.n_state; e += nt) {
    const double v0 = a.v0[e];
    if (__double_as_longlong(v0) == 0) continue;  // padding slot
    double c, sum;
    if (S) {
      const size_t n = a.n_state;
      c = S[e];
      sum = c + (S[n + e] + S[2 * n + e] + S[3 * n + e] + S[4 * n + e] + S[5 * n + e]);
    } else {
      const size_t o = ro + e;
      const float4 m = a.M[o];
      const float im = a.I[o];
      float4 cm;
      float ci;
      if (a.CMq) {  // compact compensation (srs_comp.h)
        cm = comp_load4(a.CMq + o);
        ci = comp_load1(a.CIq[o]);
      } else {
        cm = a.CM[o];
        ci = a.CI[o];
      }
      const double dx = widen(m.x) - widen(cm.x), dy = widen(m.y) - widen(cm.y), dz = widen(m.z) - widen(cm.z),
                   dw = widen(m.w) - widen(cm.w), di = widen(im) - widen(ci);
      c = a.rest_ca[e] + dx;
      sum = a.rest_sum[e] + (((dx + dy) + (dz + dw)) + di);
    }
    if (!plain_ca(a, c)) sum += sl_bound(a.bhi[e], a.khi, c) + sl_bound(a.blo[e], a.klo, c);
    if (a.jsr[e]) acc[1] = fma(v0, sum, acc[1]);
    else acc[0] = fma(v0, sum, acc[0]);
  }
  for (int q = t0; q < a.n_sl; q += nt) {
    const int e = a.sl[q];
    const double c = S ? S[e] : a.rest_ca[e] + dev_ca(a, ro + e);
    if (!plain_ca(a, c)) continue;  // above
    double b = 0.0;
    const double bhi = a.bhi[e], blo = a.blo[e];
    if (__double_as_longlong(bhi) != 0) b = sl_bound(bhi, a.khi, c);
    if (__double_as_longlong(blo) != 0) b += sl_bound(blo, a.klo, c);
    if (a.jsr[e]) acc[1] = fma(a.v0[e], b, acc[1]);
    else acc[0] = fma(a.v0[e], b, acc[0]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
    acc[1] += __shfl_xor_sync(0xffffffffu, acc[1], o);
  }
  __shared__ double red[8][2];
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[warp][0] = acc[0];
    red[warp][1] = acc[1];
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double v = 0.0;
    for (int q = 0; q < 8; ++q) v += red[q][threadIdx.x];
    a.part[((size_t)r * gridDim.x + blockIdx.x) * 2 + threadIdx.x] = v;
  }
}

__global__ void k_total_ca_sum(const double* part, double* out, int n, int blocks) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // realization * 2 + compartment
  if (i >= n) return;
  double v = 0.0;
  for (int b = 0; b < blocks; ++b) v += part[((size_t)(i >> 1) * blocks + b) * 2 + (i & 1)];
  out[i] = v;
}

// Blocks per realization: enough in all for eight per SM, with at least four
// elements a thread.
int total_ca_blocks(int n_state, int R, int n_sm) {
  const int most = (n_state + 1023) / 1024, want = (8 * n_sm + R - 1) / R;
  return most < want ? (most > 0 ? most : 1) : want;
}

int launch_total_ca(const MassArgs& a, int R, int blocks, cudaStream_t st) {
  if (blocks == 1) {  // the one block's sums are the result
    MassArgs m = a;
    m.part = a.out;
    k_total_ca<<<dim3(1, R), 256, 0, st>>>(m);
  } else {
    k_total_ca<<<dim3(blocks, R), 256, 0, st>>>(a);
    k_total_ca_sum<<<(2 * R + 127) / 128, 128, 0, st>>>(a.part, a.out, 2 * R, blocks);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// The compact compensation codec of srs_comp.h on the device: out[i] is in[i]
// after its round trip through the stored half.  Each thread takes five
// consecutive values, the first four through the four-species form (packed
// scalings when `packed`, as the plain adjoint stores them), the fifth
// through the single form.
__global__ void k_comp_round_trip(const float* in, float* out, int64_t n, int packed) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 5;
  if (i >= n) return;
  float v[5];
  for (int k = 0; k < 5; ++k) v[k] = i + k < n ? in[i + k] : 0.0f;
  ushort4 q;
  float4 c4;
  if (packed) {
    comp_store4_x2(&q, make_float4(v[0], v[1], v[2], v[3]));
    c4 = comp_load4_x2(&q);
  } else {
    comp_store4(&q, make_float4(v[0], v[1], v[2], v[3]));
    c4 = comp_load4(&q);
  }
  const float r[5] = {c4.x, c4.y, c4.z, c4.w, comp_load1(comp_store1(v[4]))};
  for (int k = 0; k < 5; ++k)
    if (i + k < n) out[i + k] = r[k];
}

// srs_div_in_range against the division: all 2^23 significands of a, of both
// signs in turn, over n_b of b (blockIdx.y; step b_step), a times 2^ea, b 2^eb.
// wrong: quotients, then reciprocals of every b, then quotients (m - 1) / (m + 1)
// of srs_logf over every float m from 1/2 to 2 (the last two by blocks of y 0).
__global__ void __launch_bounds__(256) k_division_check(int32_t b_first, int32_t b_step, int32_t n_b, int32_t ea,
                                                        int32_t eb, int64_t* wrong) {
  constexpr uint32_t n = 1u << 23;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  auto scaled = [](uint32_t significand, int e) {
    return __uint_as_float((uint32_t)(127 + e) << 23 | (significand & (n - 1)));
  };
  int64_t q = 0, y = 0, l = 0;
  for (int32_t i = blockIdx.y; i < n_b; i += gridDim.y) {
    const float b = scaled((uint32_t)b_first + (uint32_t)i * (uint32_t)b_step, eb);
    for (uint32_t s = t; s < n; s += nt) {
      const float a = s & 1 ? -scaled(s, ea) : scaled(s, ea);
      q += srs_div_in_range(a, b) != __fdiv_rn(a, b);
    }
  }
  if (blockIdx.y == 0) {
    for (uint32_t s = t; s < n; s += nt) y += srs_rcp_newton(scaled(s, eb)) != __frcp_rn(scaled(s, eb));
    for (uint32_t s = t; s < 2 * n; s += nt) {
      const float m = scaled(s, s < n ? -1 : 0);
      const float a = __fsub_rn(m, 1.0f), b = __fadd_rn(m, 1.0f);
      l += srs_div_in_range(a, b) != __fdiv_rn(a, b);
    }
  }
  auto add = [&](int k, int64_t v) {
    if (v) atomicAdd(reinterpret_cast<unsigned long long*>(wrong + k), (unsigned long long)v);
  };
  add(0, q);
  add(1, y);
  add(2, l);
}
int launch_division_check(int32_t b_first, int32_t b_step, int32_t n_b, int32_t ea, int32_t eb, int64_t* wrong,
                          cudaStream_t st) {
  k_division_check<<<dim3(128, n_b < 256 ? n_b : 256), 256, 0, st>>>(b_first, b_step, n_b, ea, eb, wrong);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_comp_round_trip(const float* in, float* out, int64_t n, int packed, cudaStream_t st) {
  const int64_t groups = (n + 4) / 5;
  const int64_t blocks = (groups + 255) / 256;
  if (blocks > 0x7fffffff) return -1;
  k_comp_round_trip<<<(unsigned)blocks, 256, 0, st>>>(in, out, n, packed);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace srs
