// k_linescan.cu — confocal line scan of the bound dye on the device.
//
// The reference's post-processing tool (linescan/main.cpp:197-225) forms, for
// each sample point x_i on a line, the PSF-weighted sum
//   F_i = sum_j V0_j * [CaDye]_j * N(r_ij; sigma)      (|r_ij|^2 < r_thresh)
// over mesh cells and padding voxels held at the resting fluorescence.  The
// host folds the cell volumes and PSF values into a sparse weight matrix
// (samples x elements, engine numbering) and the constant padding sum into an
// offset; this kernel evaluates the sum from the state in HBM for every
// realization, accumulating in double precision.
#include <type_traits>

#include "srs_comp.h"
#include "srs_engine.h"

namespace srs {

// One block per (sample, realization).  With few blocks a term's chain of loads
// and conversions is what a thread waits for, so four terms' are in flight: one
// realization of 69,696 elements 82 us a call (141 with one term at a time), 256
// realizations 4.9 ms (7.0).
__global__ void k_linescan(LinescanArgs a) {
  const int i = blockIdx.x, r = blockIdx.y;
  const int end = a.ptr[i + 1], stride = blockDim.x;
  double acc = 0.0;
  // adds the terms q, q + stride, ...: N of them, whose loads are in flight together
  auto terms = [&](int q, auto n) {
    constexpr int N = decltype(n)::value;
    int e[N];
    double w[N], dye[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      e[k] = a.col[q + k * stride];
      w[k] = a.w[q + k * stride];
    }
    if (a.S64) {
#pragma unroll
      for (int k = 0; k < N; ++k) dye[k] = a.S64[(size_t)r * 6 * a.n_state + 5 * (size_t)a.n_state + e[k]];
    } else {
      float u[N], c[N];
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const size_t o = (size_t)r * a.n_state + e[k];
        u[k] = a.M[o].w;
        c[k] = a.CMq ? comp_load1(a.CMq[o].w) : a.CM[o].w;
        dye[k] = a.rest_dye[e[k]];
      }
#pragma unroll
      for (int k = 0; k < N; ++k) dye[k] += widen(u[k]) - widen(c[k]);
    }
#pragma unroll
    for (int k = 0; k < N; ++k) acc += w[k] * dye[k];
  };
  int q = a.ptr[i] + threadIdx.x;
  for (; q + 3 * stride < end; q += 4 * stride) terms(q, std::integral_constant<int, 4>{});
  for (; q < end; q += stride) terms(q, std::integral_constant<int, 1>{});
  __shared__ double red[256];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) a.out[(size_t)r * a.n_samples + i] = a.pad[i] + red[0];
}

// Tiled form for an ensemble: lanes over 32 realizations, each warp eight
// samples.  A block stages the dye of LINESCAN_CHUNK elements of its 32
// realizations in shared memory (one conversion to double per element and
// realization, where the form above does it once per sample) and every warp
// adds them into its eight sums, one multiply-add per weight.  The bound is
// the FP64 pipe: 1024 realizations of the 10,368-element dyad, 40 samples,
// about 330 M weighted terms, 0.52 ms at 2 DFMA per clock and SM; the call
// took 3.19 ms untiled and takes 0.73.  The chunks are dealt to a.splits blocks
// (a.split: by their work) whose partial sums k_linescan_sum adds in order.
__global__ void __launch_bounds__(256) k_linescan_tile(LinescanArgs a, int R) {
  __shared__ double s_dye[LINESCAN_CHUNK][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = blockIdx.z * (blockDim.x >> 5) + warp;  // sample group
  const bool live = g * 8 < a.n_samples;
  const int r0 = blockIdx.y * 32, nr = min(32, R - r0);
  double acc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.0;
  const int32_t* tp = a.tptr + (size_t)(live ? g : 0) * (a.n_chunk + 1);
  const int c0 = a.split[blockIdx.x], c1 = a.split[blockIdx.x + 1];
  for (int c = c0; c < c1; ++c) {
    const int e0 = c * LINESCAN_CHUNK;
    __syncthreads();
    for (int q = threadIdx.x; q < LINESCAN_CHUNK * 32; q += blockDim.x) {
      const int k = q & (LINESCAN_CHUNK - 1), rr = q / LINESCAN_CHUNK, e = e0 + k;
      double dye = 0.0;
      if (rr < nr && e < a.n_state) {
        const int r = r0 + rr;
        if (a.S64) {
          dye = a.S64[(size_t)r * 6 * a.n_state + 5 * (size_t)a.n_state + e];
        } else {
          const size_t o = (size_t)r * a.n_state + e;
          const float u = a.M[o].w;
          const float cm = a.CMq ? comp_load1(a.CMq[o].w) : a.CM[o].w;
          dye = a.rest_dye[e] + (widen(u) - widen(cm));
        }
      }
      s_dye[k][rr] = dye;
    }
    __syncthreads();
    if (live) {
      for (int q = tp[c]; q < tp[c + 1]; ++q) {
        const uint32_t t = a.tent[q];
        const double dye = s_dye[t & 0xffffffu][lane];
        const double2* w = reinterpret_cast<const double2*>(a.tw + (size_t)q * 8);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const double2 v = __ldg(w + k);
          // an element a sample does not weigh adds nothing, whatever its value
          if (t >> (24 + 2 * k) & 1u) acc[2 * k] = fma(v.x, dye, acc[2 * k]);
          if (t >> (25 + 2 * k) & 1u) acc[2 * k + 1] = fma(v.y, dye, acc[2 * k + 1]);
        }
      }
    }
  }
  if (live && lane < nr) {
    double* out = a.part + ((size_t)blockIdx.x * R + r0 + lane) * a.n_samples + g * 8;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (g * 8 + k < a.n_samples) out[k] = acc[k];
  }
}

__global__ void k_linescan_sum(LinescanArgs a, int R) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= R * a.n_samples) return;
  double v = 0.0;
  for (int s = 0; s < a.splits; ++s) v += a.part[(size_t)s * R * a.n_samples + i];
  a.out[i] = a.pad[i % a.n_samples] + v;
}

// Warps of a tiled block: one per sample group, eight at most.
static int tile_warps(int n_samples) { return (n_samples + 7) / 8 < 8 ? (n_samples + 7) / 8 : 8; }

// Blocks that share the chunks of one tile of realizations: eight per SM in
// all (six or twelve measured up to a tenth longer), at least one chunk each.
int linescan_splits(int n_samples, int n_state, int R, int n_sm) {
  const int chunks = (n_state + LINESCAN_CHUNK - 1) / LINESCAN_CHUNK;
  const int tiles = (R + 31) / 32 * (((n_samples + 7) / 8 + 7) / 8);
  const int want = (8 * n_sm + tiles - 1) / tiles;
  return chunks < want ? chunks : want;
}

int launch_linescan(const LinescanArgs& a, int R, cudaStream_t st) {
  if (a.tptr) {
    const int w = tile_warps(a.n_samples), groups = (a.n_samples + 7) / 8;
    k_linescan_tile<<<dim3(a.splits, (R + 31) / 32, (groups + w - 1) / w), 32 * w, 0, st>>>(a, R);
    k_linescan_sum<<<(unsigned)(((size_t)R * a.n_samples + 127) / 128), 128, 0, st>>>(a, R);
  } else {
    k_linescan<<<dim3(a.n_samples, R), 256, 0, st>>>(a);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace srs
