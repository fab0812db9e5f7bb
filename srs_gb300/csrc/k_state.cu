// k_state.cu — a realization's state in the caller's form, and the reset of all
// realizations, on the device.
//
// srs_sim_get_state returns absolute concentrations in the reference's
// numbering; the FP32 engines hold deviations from rest in their own.  The
// conversion (one FP64 addition a value) runs here and writes the caller's
// form, into pinned host memory for states of up to a few MB: a host loop over
// 542,376 elements after four copies took 6.4 ms, one over 15,288 0.2.
#include "srs_comp.h"
#include "srs_engine.h"

namespace srs {

__global__ void __launch_bounds__(256) k_export_state(ExportArgs a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  if (a.S) {
    const size_t N = a.N;
    if (a.S64) {
      for (size_t i = t; i < 6 * N; i += nt) a.S[i] = a.S64[i];
    } else {
      for (int j = t; j < a.N; j += nt) {
        const int e = a.eng_of_ref[j];
        const uint32_t fl = a.flags[(size_t)e * a.flag_stride];
        const bool jsr = fl & 1u, trop = fl & 2u;
        const double f = jsr ? 0.0 : 1.0;
        const float4 m = a.M[e];
        const float4 c = a.CMq ? comp_load4(a.CMq + e) : a.CM[e];
        const float im = a.I[e], ci = a.CIq ? comp_load1(a.CIq[e]) : a.CI[e];
        // the state is u - comp (the compensation holds the rounding error of
        // the last update)
        const double imm = (jsr ? a.rest[4] : trop ? a.rest[3] : 0.0) + ((double)im - (double)ci);
        a.S[j] = (jsr ? a.rest_ca_jsr : a.rest[0]) + ((double)m.x - (double)c.x);
        a.S[N + j] = f * a.rest[1] + ((double)m.y - (double)c.y);
        a.S[2 * N + j] = f * a.rest[2] + ((double)m.z - (double)c.z);
        a.S[3 * N + j] = jsr ? 0.0 : imm;
        a.S[4 * N + j] = jsr ? imm : 0.0;
        a.S[5 * N + j] = f * a.rest[5] + ((double)m.w - (double)c.w);
      }
    }
  }
  if (blockIdx.x == 0) {
    for (int i = threadIdx.x; i < a.NR && a.ryr_out; i += blockDim.x) a.ryr_out[i] = a.ryr[i];
    for (int i = threadIdx.x; i < a.NL && a.lcc_out; i += blockDim.x) a.lcc_out[i] = a.lcc[i];
    for (int i = threadIdx.x; i < a.NL && a.lccv_out; i += blockDim.x) a.lccv_out[i] = a.lccv[i];
    for (int i = threadIdx.x; i < a.NR + a.NL && a.res_out; i += blockDim.x) a.res_out[i] = a.res[i];
  }
}

int launch_export_state(const ExportArgs& a, cudaStream_t st) {
  const int most = (a.N + 255) / 256;
  k_export_state<<<most < 608 ? most : 608, 256, 0, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// dL/d(initial state) of realizations blockIdx.y in the caller's numbering, from
// lambda and its compensation (the host's pass over 21 x 15,288 elements after
// four copies took 4.3 ms).
__global__ void __launch_bounds__(256) k_export_lambda(ExportLambdaArgs a) {
  const size_t N = a.N, o = (size_t)blockIdx.y * a.NE;
  double* g = a.g + (size_t)blockIdx.y * 6 * N;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < a.N; j += gridDim.x * blockDim.x) {
    const int e = a.eng_of_ref[j];
    const uint32_t fl = a.flags[(size_t)e * a.flag_stride];
    const bool jsr = fl & 1u, trop = fl & 2u;
    const float4 m = a.lam[o + e];
    const float4 c = a.c4q ? comp_load4(a.c4q + o + e) : a.c4[o + e];
    const float im = a.lam_im[o + e], ci = a.cimq ? comp_load1(a.cimq[o + e]) : a.cim[o + e];
    const double li = (double)im - (double)ci;
    g[j] = (double)m.x - (double)c.x;
    g[N + j] = (double)m.y - (double)c.y;
    g[2 * N + j] = (double)m.z - (double)c.z;
    g[3 * N + j] = !jsr && trop ? li : 0.0;
    g[4 * N + j] = jsr ? li : 0.0;
    g[5 * N + j] = (double)m.w - (double)c.w;
  }
}
int launch_export_lambda(const ExportLambdaArgs& a, int R, cudaStream_t st) {
  const int most = (a.N + 255) / 256;
  k_export_lambda<<<dim3(most < 608 ? most : 608, R), 256, 0, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// One state for every realization: dst[r][i] = src[i].
template <class T>
__global__ void __launch_bounds__(256) k_broadcast_state(const T* src, T* dst, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[blockIdx.y * n + i] = src[i];
}
template <class T>
int launch_broadcast_state(const T* src, T* dst, size_t n, int R, cudaStream_t st) {
  const size_t most = (n + 255) / 256;
  k_broadcast_state<<<dim3((unsigned)(most < 304 ? most : 304), R), 256, 0, st>>>(src, dst, n);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
template int launch_broadcast_state(const double*, double*, size_t, int, cudaStream_t);
template int launch_broadcast_state(const float*, float*, size_t, int, cudaStream_t);

}  // namespace srs
