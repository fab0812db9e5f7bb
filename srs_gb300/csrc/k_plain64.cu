// k_plain64.cu — FP64 spark step in the reference's operation order.
//
// One fused launch per time step: every thread advances one element of one
// realization through the whole of ExplicitStep (cpu/RunSimulation.cpp:
// 591-654) — ELL-4 diffusion of the four mobile species, buffer reactions,
// SERCA, JSR refill, RyR/LCC flux, rapid SL buffer, Euler update — reading
// the state of step n and writing step n+1 (double buffered).  The last
// block of each realization to finish then runs channel gating and the
// protocol work of the next step, so a step is a single launch.
//
// Every expression keeps the reference's association order and this file is
// compiled with -fmad=false, so with identical inputs the result matches the
// reference's FP64 step bit for bit.  This engine is the FP64 oracle run of
// the GPU path; the FP32 engines are measured against it.
#include <cmath>

#include "srs_engine.h"
#include "srs_pdl.cuh"
#include "srs_plain64_update.cuh"
#include "srs_protocol.cuh"

namespace srs {


// Channel fluxes of element j (UpdateRyRFlux / UpdateLCCFlux, :127-164) added
// to its Ca rate in the reference's order.
__device__ __forceinline__ double channels64(const Plain64Args& a, const double* Sca, int j, double c_ca,
                                             double b_ca, const int32_t* ryr, const int32_t* lcc,
                                             const int32_t* lccv, int v) {
  for (int q = a.chan_ptr[j]; q < a.chan_ptr[j + 1]; ++q) {
    ChanEntry e = a.chan_list[q];
    if (e.kind < 2) {
      if (ryr[e.ch]) {
        double J = a.P.v_ryr * (Sca[a.C.ryr_jsr[e.ch]] - Sca[a.C.ryr_cleft[e.ch]]) * a.P.v_cell;
        if (e.kind == 0) b_ca += J / a.v0[j];
        else b_ca -= J / a.v0[j];
      }
    } else if ((lcc[e.ch] == 6 || lcc[e.ch] == 12) && lccv[e.ch] == 2) {
      double J = a.P.lccA[v] * (c_ca * a.P.lccE[v] - a.P.lccB) / a.P.lccEm1[v] / a.v0[j];
      b_ca += J;
    }
  }
  return b_ca;
}

// The last block of realization r to get here gates its channels from the new
// Ca and runs the protocol of the next step.  chan: this block holds channel
// elements, whose new Ca the last block must see.
__device__ __forceinline__ void plain64_tail(const Plain64Args& a, int r, const RealCtl& ctl0, const double* Sn,
                                             bool chan) {
  __shared__ int s_last;
  __shared__ int32_t s_nb[1024];
  if (chan) {
    __threadfence();
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    unsigned int done = atomicAdd(a.counters + r, 1u);
    s_last = (done == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  RealCtl ctl = ctl0;
  auto ca = [&](int e) -> double { return *((volatile const double*)(Sn + e)); };
  int32_t* ryr_w = a.CS.ryr + (size_t)r * a.C.NR;
  int32_t* lcc_w = a.CS.lcc + (size_t)r * a.C.NL;
  int32_t* lccv_w = a.CS.lccv + (size_t)r * a.C.NL;
  double* res = a.CS.res + (size_t)r * (a.C.NR + a.C.NL);
  if (!a.P.nogating) {
    gate_all(a.P, a.C, ctl.vsel, ctl.seed, ctl.step, ryr_w, lcc_w, lccv_w, res, s_nb,
             threadIdx.x, blockDim.x, ca, []() { __syncthreads(); });
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    a.counters[r] = 0;  // as the next step finds it
    ctl.step += 1;
    ctl.t += a.P.dt;
    prestep(a.P, a.C, ctl, ryr_w, lcc_w, lccv_w,
            a.CS.rows + (size_t)r * a.P.row_cap * a.P.row_w, ca);
    RealCtl* c = a.CS.ctl + r;
    ctl.status |= c->status;  // bits of the other blocks
    *c = ctl;
    __threadfence();
  }
}

// One thread per element.  64-thread blocks: with 256 the last wave is longer (115,000
// elements of 300 realizations 53 us a step, 39 so; 236,000 of eight 76 and 72).
__global__ void __launch_bounds__(256) k_plain64_step(Plain64Args a) {
  pdl_wait();
  pdl_next();
  const int r = blockIdx.y;
  RealCtl* ctlp = a.CS.ctl + r;
  if (ctlp->done) return;  // uniform per realization
  const int N = a.N;
  const double* S = a.S_in + (size_t)r * 6 * N;
  double* So = a.S_out + (size_t)r * 6 * N;
  const int32_t* ryr = a.CS.ryr + (size_t)r * a.C.NR;
  const int32_t* lcc = a.CS.lcc + (size_t)r * a.C.NL;
  const int32_t* lccv = a.CS.lccv + (size_t)r * a.C.NL;
  const double* p = a.p;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < N) {
    const double* Sca = S + 0 * N;
    const double* Satp = S + 1 * N;
    const double* Scmdn = S + 2 * N;
    const double* Strpn = S + 3 * N;
    const double* Scsqn = S + 4 * N;
    const double* Sdye = S + 5 * N;
    double c_ca = Sca[j];
    double a0 = a.aij[5 * j], a1 = a.aij[5 * j + 1], a2 = a.aij[5 * j + 2];
    double a3 = a.aij[5 * j + 3], a4 = a.aij[5 * j + 4];
    int n1 = a.nij[4 * j], n2 = a.nij[4 * j + 1], n3 = a.nij[4 * j + 2], n4 = a.nij[4 * j + 3];
    // UpdateReactionTerms (cpu/RunSimulation.cpp:25-125)
    const double ac[5] = {a0, a1, a2, a3, a4};
    const double dye = Sdye[j], atp = Satp[j], cmdn = Scmdn[j];
    double b_ca = diffuse64(p[5], c_ca, Sca[n1], Sca[n2], Sca[n3], Sca[n4], ac, a.br[0 * N + j]);
    double b_dye = diffuse64(p[11], dye, Sdye[n1], Sdye[n2], Sdye[n3], Sdye[n4], ac, a.br[3 * N + j]);
    double b_atp = diffuse64(p[7], atp, Satp[n1], Satp[n2], Satp[n3], Satp[n4], ac, a.br[1 * N + j]);
    double b_cmdn = diffuse64(p[8], cmdn, Scmdn[n1], Scmdn[n2], Scmdn[n3], Scmdn[n4], ac, a.br[2 * N + j]);
    const int fl = a.flags[j];
    const double dt = a.P.dt;
    // the immobile buffers: a rate of zero leaves the value (-0 becomes +0)
    double o_trpn = plus_zero(Strpn[j]), o_csqn = plus_zero(Scsqn[j]);
    double r_net;
    if (!(fl & 1)) {
      if (fl & 2) {
        const double t = Strpn[j];
        r_net = react64(p[26], p[24], p[25], t, c_ca);
        b_ca += -r_net;
        o_trpn = t + r_net * dt;
        b_ca -= serca64(a, c_ca);
      }
      r_net = react64(p[33], p[31], p[32], dye, c_ca);
      b_ca += -r_net;
      b_dye += r_net;
      r_net = react64(p[20], p[18], p[19], atp, c_ca);
      b_ca += -r_net;
      b_atp += r_net;
      r_net = react64(p[23], p[21], p[22], cmdn, c_ca);
      b_ca += -r_net;
      b_cmdn += r_net;
    } else {
      const double q = Scsqn[j];
      r_net = react64(p[39], p[34], p[40], q, c_ca);
      b_ca += -r_net;
      o_csqn = q + r_net * dt;
      b_ca += (a.nsr - c_ca) * p[36];
    }
    if (fl & 4) b_ca = channels64(a, S, j, c_ca, b_ca, ryr, lcc, lccv, ctlp->vsel);
    b_ca = fast_buffer64(a, b_ca, c_ca, a.bhi[j], a.blo[j]);
    // Euler update (:640-644)
    double* O = So;
    const double ca_new = c_ca + b_ca * dt;
    O[0 * N + j] = ca_new;
    O[1 * N + j] = atp + b_atp * dt;
    O[2 * N + j] = cmdn + b_cmdn * dt;
    O[3 * N + j] = o_trpn;
    O[4 * N + j] = o_csqn;
    O[5 * N + j] = dye + b_dye * dt;
    if (!finite64(ca_new)) atomicOr(&ctlp->status, 1u);
  }
  plain64_tail(a, r, *ctlp, So, __syncthreads_or(j < N && (a.flags[j] & 4) != 0) != 0);
}

// The same for problems of few elements: 32 elements a block, the update dealt
// to four warps (srs_plain64_update.cuh).  KEYS: the allocation-free form, whose
// step and seeds come with the launch (Plain64Keys) instead of from RealCtl and
// whose gating is a launch of its own (k_plain64_gate).
template <bool KEYS>
__global__ void __launch_bounds__(128) k_plain64_split(const __grid_constant__ Plain64Args a,
                                                       const __grid_constant__ Plain64Keys<KEYS> keys) {
  __shared__ double s_rate[5][32];
  pdl_wait();
  pdl_next();
  const int r = blockIdx.y;
  RealCtl ctl{};
  unsigned* status;
  if constexpr (KEYS) {
    ctl.step = keys.step;
    ctl.seed = keys.seeds[r];
    ctl.lcc_close_step = -1;
    status = keys.status;
  } else {
    ctl = a.CS.ctl[r];
    status = &a.CS.ctl[r].status;
    if (ctl.done) return;  // uniform per realization
  }
  const int N = a.N, lane = threadIdx.x & 31, role = ((threadIdx.x >> 5) + blockIdx.x) & 3;
  const int j = blockIdx.x * 32 + lane;
  const int e = min(j, N - 1);  // the last element stands in
  const size_t n = N, ro = (size_t)r * 6 * N;
  const double* S = a.S_in + ro;
  double* So = a.S_out + ro;
  const Geo64 g = geometry64(a, e);
  const double c = S[e];
  double x0 = S[role64_x0(role) * n + e], x1 = S[role64_x1(role) * n + e];
  const double b0 = role64(a, role, g, e, lane, S, c, x0, x1, s_rate);
  if (j < N && role > 0) {
    So[role64_x0(role) * n + e] = x0;
    if (role < 3) So[role64_x1(role) * n + e] = x1;
  }
  __syncthreads();
  if (role == 0) {
    double b_ca = sum64(a, g.fl, lane, c, b0, s_rate);
    if (g.fl & 4) {
      const int32_t* ryr = a.CS.ryr + (size_t)r * a.C.NR;
      const int32_t* lcc = a.CS.lcc + (size_t)r * a.C.NL;
      const int32_t* lccv = a.CS.lccv + (size_t)r * a.C.NL;
      b_ca = channels64(a, S, e, c, b_ca, ryr, lcc, lccv, ctl.vsel);
    }
    b_ca = fast_buffer64(a, b_ca, c, a.bhi[e], a.blo[e]);
    const double ca_new = c + b_ca * a.P.dt;
    if (j < N) {
      So[e] = ca_new;
      if (!finite64(ca_new) && status) atomicOr(status, 1u);
    }
  }
  if constexpr (!KEYS) plain64_tail(a, r, ctl, So, __syncthreads_or(g.fl & 4) != 0);
}

// Gating of an allocation-free step, one block a realization.  It is not left to
// the last block of the update: that block finds itself by a counter in device
// memory, and one that all calls share carries the error of two overlapping calls
// into every later one.  As a chained launch (srs_pdl.cuh) it is the shorter way
// besides: 64 steps of 3 x 384 elements 680 us against 761 with the counter, its
// fences and the reload.
__global__ void __launch_bounds__(128) k_plain64_gate(const __grid_constant__ Plain64Args a,
                                                      const __grid_constant__ Plain64Keys<true> keys) {
  __shared__ int32_t s_nb[1024];
  const int r = blockIdx.x, NR = a.C.NR, NL = a.C.NL;
  // the channels' elements, which no step writes, before the wait
  int e0 = 0, e1 = 0;
  auto elements = [&](int i) {
    e0 = i < NR ? __ldcg(a.C.ryr_cleft + i) : __ldcg(a.C.lcc_ele + i - NR);
    e1 = i < NR ? __ldcg(a.C.ryr_jsr + i) : e0;
  };
  const int i0 = threadIdx.x;
  if (i0 < NR + NL) elements(i0);
  pdl_wait();
  pdl_next();
  const double* Sn = a.S_out + (size_t)r * 6 * a.N;
  int32_t* ryr = a.CS.ryr + (size_t)r * NR;
  int32_t* lcc = a.CS.lcc + (size_t)r * NL;
  int32_t* lccv = a.CS.lccv + (size_t)r * NL;
  double* res = a.CS.res + (size_t)r * (NR + NL);
  const srs_gate_consts* g = &a.P.gc[0];
  if (g->ryr_astar_half != 0.0f) {  // coupled gating
    gate_all(a.P, a.C, 0, keys.seeds[r], keys.step, ryr, lcc, lccv, res, s_nb, threadIdx.x, blockDim.x,
             [&](int e) { return Sn[e]; }, []() { __syncthreads(); });
    return;
  }
  for (int i = i0; i < NR + NL; i += blockDim.x) {
    if (i != i0) elements(i);
    const float c0 = (float)Sn[e0], c1 = (float)Sn[e1];
    double q = res[i];
    if (i < NR) {
      ryr[i] = srs_gate_ryr(g, ryr[i], c0, c1, 0, 0, &q, keys.seeds[r], (uint32_t)i, (uint64_t)keys.step);
    } else {
      int st = lcc[i - NR], vs = lccv[i - NR];
      srs_gate_lcc(g, &st, &vs, c0, &q, keys.seeds[r], (uint32_t)i, (uint64_t)keys.step);
      lcc[i - NR] = st;
      lccv[i - NR] = vs;
    }
    res[i] = q;
  }
}

// Protocol work before the first step of a run (and the t = 0 row).
__global__ void k_plain64_prestep(Plain64Args a, int write_initial_row) {
  const int r = blockIdx.x;
  if (threadIdx.x != 0) return;
  RealCtl ctl = a.CS.ctl[r];
  const double* S = a.S_in + (size_t)r * 6 * a.N;
  auto ca = [&](int e) -> double { return S[e]; };
  int32_t* ryr = a.CS.ryr + (size_t)r * a.C.NR;
  int32_t* lcc = a.CS.lcc + (size_t)r * a.C.NL;
  int32_t* lccv = a.CS.lccv + (size_t)r * a.C.NL;
  float* rows = a.CS.rows + (size_t)r * a.P.row_cap * a.P.row_w;
  if (write_initial_row && a.P.run_protocol) write_row(a.P, a.C, ctl, ryr, lcc, lccv, rows, ctl.t, ca);
  prestep(a.P, a.C, ctl, ryr, lcc, lccv, rows, ca);
  a.CS.ctl[r] = ctl;
}

// The element-independent terms of the SERCA flux in the reference's
// operations (cpu/RunSimulation.cpp:83-91).
void plain64_consts(Plain64Args* a) {
  double K_sr = a->nsr / a->p[50];
  K_sr = K_sr * K_sr;
  a->sd0 = 0.104217 + 17.923 * K_sr;
  a->sd1 = 1.75583e6 + K_sr * 7.61673e6;
  a->sd2 = 6.08463e11 + K_sr * 4.50544e11;
  a->sn1 = 9.17846e6 - 11478.2 * K_sr;
  a->sn0 = 0.329904 * K_sr;
  const double k = std::fabs(a->p[49]);
  a->inv_kdi = k > 0x1p-500 && k < 0x1p500 ? 1.0 / a->p[49] : 0.0;
}

// Tiles of 32 elements up to which the update is dealt to four warps: six blocks
// per SM.  Beyond, the FP64 pipes are busy anyway and a thread per element
// avoids passing values between warps.
static bool small64(const Plain64Args& a) { return (int64_t)((a.N + 31) / 32) * a.R <= 6 * 152; }
// Dealt to four warps also where the blocks of a thread per element would be a full
// wave (six of 64 threads per SM) and a small part of another: 62,000 elements take
// 27.4 us a step so and 39.5 by a thread each, 92,000 35.0 and 39.7, but 104,000 38.8
// and 40.3, 300 realizations of 384 46.2 and 39.4, 311,000 96.7 and 93.8.
static bool split64(const Plain64Args& a) {
  const int64_t blocks = (int64_t)((a.N + 63) / 64) * a.R;
  return small64(a) || (blocks > 6 * 152 && blocks <= 1600);
}

int launch_plain64_step(const Plain64Args& a, cudaStream_t st) {
  if (split64(a))
    launch_pdl(k_plain64_split<false>, dim3((a.N + 31) / 32, a.R), 128, 0, st, a, Plain64Keys<false>{});
  else
    launch_pdl(k_plain64_step, dim3((a.N + 63) / 64, a.R), 64, 0, st, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

bool plain64_keys_fit(const Plain64Args& a) { return small64(a); }
int launch_plain64_keys(const Plain64Args& a, const Plain64Keys<true>& k, cudaStream_t st) {
  cudaError_t e = launch_pdl(k_plain64_split<true>, dim3((a.N + 31) / 32, a.R), 128, 0, st, a, k);
  if (e == cudaSuccess && !a.P.nogating) e = launch_pdl(k_plain64_gate, a.R, 128, 0, st, a, k);
  return e == cudaSuccess ? 0 : -1;
}
int launch_plain64_prestep(const Plain64Args& a, int write_initial_row, cudaStream_t st) {
  k_plain64_prestep<<<a.R, 32, 0, st>>>(a, write_initial_row);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace srs
