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

namespace srs {

// Rapid-buffer part b c / (K + c).  The division is skipped where it gives
// zero (elements off the membrane, about nine in ten): the FP64 pipe issues
// one warp instruction in 64 cycles here, and the two divisions were half of
// an element's work.
__device__ __forceinline__ double sl_bound(double b, double K, double c) {
  return b == 0.0 && isfinite(c) && c != -K ? 0.0 : b * c / (K + c);
}

// Grid: x over blocks of one realization's elements, y over realizations.  A
// block per realization alone leaves a few large realizations on a few SMs
// (32 x 542,376 elements: 11.4 ms a call; with the split and without the
// empty divisions 1.24, bound by the FP64 pipe).  Each block writes its two sums; k_total_ca_sum adds them in order.
__global__ void __launch_bounds__(256) k_total_ca(MassArgs a) {
  const int r = blockIdx.y;
  double acc[2] = {0.0, 0.0};
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < a.n_state; e += gridDim.x * blockDim.x) {
    const double v0 = a.v0[e];
    if (v0 == 0.0) continue;  // padding slot
    double c, bound;
    if (a.S64) {
      const double* S = a.S64 + (size_t)r * 6 * a.n_state;
      const size_t n = a.n_state;
      c = S[e];
      bound = S[n + e] + S[2 * n + e] + S[3 * n + e] + S[4 * n + e] + S[5 * n + e];
    } else {
      const size_t o = (size_t)r * a.n_state + e;
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
      const double* rs = a.rest4 + 4 * (size_t)e;
      c = rs[0] + ((double)m.x - (double)cm.x);
      bound = (rs[1] + ((double)m.y - (double)cm.y)) + (rs[2] + ((double)m.z - (double)cm.z)) +
              (rs[3] + ((double)m.w - (double)cm.w)) + (a.rest_imm[e] + ((double)im - (double)ci));
    }
    const double sl = sl_bound(a.bhi[e], a.khi, c) + sl_bound(a.blo[e], a.klo, c);
    acc[a.jsr[e] ? 1 : 0] += v0 * (c + bound + sl);
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
  k_total_ca<<<dim3(blocks, R), 256, 0, st>>>(a);
  k_total_ca_sum<<<(2 * R + 127) / 128, 128, 0, st>>>(a.part, a.out, 2 * R, blocks);
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

int launch_comp_round_trip(const float* in, float* out, int64_t n, int packed, cudaStream_t st) {
  const int64_t groups = (n + 4) / 5;
  const int64_t blocks = (groups + 255) / 256;
  if (blocks > 0x7fffffff) return -1;
  k_comp_round_trip<<<(unsigned)blocks, 256, 0, st>>>(in, out, n, packed);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace srs
