// k_plain_loop.cu — the plain engines' steps in one launch, for problems that
// fit on the chip's threads.
//
// With one launch per time step (k_plain64.cu, k_fp32.cu: chained launches,
// replayed as a graph) a small problem waits: 384 elements take 10.9 us a step in
// FP64 and 6.4 in FP32, 10,368 take 11.5 and 6.9 -- launch, loads, update, a
// counter of finished blocks, and then the last block's gating, one after the
// other.  Here (6.4 and 3.5, 6.9 and 3.4) a cooperative launch keeps all blocks
// resident for many steps:
//   * element blocks hold their elements' geometry, immobile buffer and
//     (FP32) compensation terms in registers; a step reads the neighbours'
//     values from L2 and writes the mobile species, double buffered as before;
//   * one barrier per realization and step: a counter the blocks add to;
//   * a block whose elements carry channels keeps the states of those channels
//     and gates them itself, from the Ca it reads with its neighbours after the
//     barrier.  Two blocks that share a channel (its cleft and its JSR element)
//     gate it both: from the same Ca and the same random number they take the
//     same decision, and neither waits for the other (a flag published by one
//     gating block, which a first form used, was two more trips through L2 on
//     the way from one step to the next: 4.3 us a step in FP32);
//   * one more block per realization gates all channels again, off that path,
//     and runs the protocol: output rows, run's end, final channel states.
// Results are those of the one-launch-per-step kernels bit for bit: the same
// update functions, the same order of sums.
//
// Used where no realization can end early (the parameter set has no fidelity
// criterion, so every realization takes the same steps) and RyRs do not couple
// (RYR_A_STAR = 0, as in every shipped set), on meshes below the split form's
// size, when all blocks fit at once.  Every wait has a limit (PlainLoop::rounds);
// a block that gives up sets status bit 1 and two flags and leaves, and so do the
// others.  The device flag lets later launches leave at once, whose counters
// would start off zero; the host flag makes every call fail that waits for the
// device, until the next reset.
#include <cstdint>

#include "srs_engine.h"
#include "srs_fp32_update.cuh"
#include "srs_plain64_update.cuh"
#include "srs_protocol.cuh"

namespace srs {

namespace {

constexpr uint64_t kClosed = 0x7ff8c105edc105edull;  // a NaN that no arithmetic gives

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_add(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Waits until *p has reached `target`; false: gave up after that many rounds of
// polls.  The polls of a round are of a fixed number, which the compiler unrolls:
// 1500 steps of 5 x 6,000 elements 5.36 ms, 5.52 with a variable number.
__device__ __forceinline__ bool wait_for(const unsigned* p, unsigned target, int rounds) {
  for (int n = 0; n < rounds; ++n)
    for (int i = 0; i < 65536; ++i)
      if ((int)(ld_acquire(p) - target) >= 0) return true;
  return false;
}
__device__ __forceinline__ void give_up(const PlainLoop& l) {
  *l.gave_up = 1u;
  *l.timeout = 1u;
}

// Waits (one thread, for the block) until every element block of a realization
// has arrived; with __syncthreads and a release on the arriving side, the
// blocks' writes before it are visible after it.
__device__ __forceinline__ bool wait_all(const unsigned* bar, unsigned target, int rounds) {
  int ok = 1;
  if (threadIdx.x == 0) ok = wait_for(bar, target, rounds);
  return __syncthreads_and(ok);
}

// Steps of the launch for realization r: a run ends at its last step.  Every
// thread of the block calls it.
template <class Args>
__device__ __forceinline__ int steps_of(const Args& a, const PlainLoop& l, const RealCtl& c) {
  const int done = c.done;  // both loads in flight together with the flag's
  const int64_t step = c.step;
  if (__syncthreads_or(__ldcg(l.gave_up) != 0) || done) return 0;
  return a.P.run_protocol ? (int)max((int64_t)0, min((int64_t)l.steps, a.P.n_steps - step)) : l.steps;
}

// ---- the protocol's block ----------------------------------------------------------
// Shared memory: RealCtl; gating constants; the channel states, residuals.
struct GateSmem {
  RealCtl ctl;
  srs_gate_consts gc[2];
  int64_t next_ev;
};
}  // namespace

// ch_max: most channels an element block gates
size_t plain_loop_smem_bytes(int NR, int NL, int ch_max) {
  size_t g = (sizeof(GateSmem) + 15) & ~(size_t)15;
  g += (size_t)(NR + NL) * sizeof(double) + (size_t)(NR + 2 * NL) * sizeof(int32_t);
  size_t e = (2 * sizeof(srs_gate_consts) + 15) & ~(size_t)15;
  e += (size_t)ch_max * (2 * sizeof(double) + 5 * sizeof(int32_t)) + 8;
  return g > e ? g : e;
}

namespace {

// ca(e, buf): absolute Ca of element e in state buffer buf, from L2.
template <class Args, class Ca>
__device__ void gate_loop(const Args& a, const PlainLoop& l, int r, int steps, Ca ca, unsigned char* smem) {
  GateSmem* g = reinterpret_cast<GateSmem*>(smem);
  double* res = reinterpret_cast<double*>(smem + ((sizeof(GateSmem) + 15) & ~(size_t)15));
  const int NR = a.C.NR, NL = a.C.NL, tid = threadIdx.x, nt = blockDim.x;
  int32_t* ryr = reinterpret_cast<int32_t*>(res + NR + NL);
  int32_t* lcc = ryr + NR;
  int32_t* lccv = lcc + NL;
  const size_t rr = (size_t)r * NR, rl = (size_t)r * NL, rc = (size_t)r * (NR + NL);
  if (tid == 0) g->ctl = a.CS.ctl[r];
  if (tid < 2) g->gc[tid] = a.P.gc[tid];
  for (int i = tid; i < NR; i += nt) ryr[i] = a.CS.ryr[rr + i];
  for (int i = tid; i < NL; i += nt) {
    lcc[i] = a.CS.lcc[rl + i];
    lccv[i] = a.CS.lccv[rl + i];
  }
  for (int i = tid; i < NR + NL; i += nt) res[i] = a.CS.res[rc + i];
  __syncthreads();
  unsigned* bar = l.bar + r;
  if (tid == 0) red_release_add(bar, 1u);
  const int64_t step0 = g->ctl.step;
  int64_t next_ev = 0;
  bool ok = true;
  for (int s = 0; s < steps; ++s) {
    const int64_t step = step0 + s;
    const int out = (s & 1) ^ 1;  // buffer of the state after this step
    const int v = g->ctl.vsel;
    const srs_gate_consts* gc = &g->gc[v];
    const int hold = a.P.run_protocol && a.P.init_ryr != -1 && step + 1 < a.P.hold_end ? a.P.init_ryr : -1;
    ok = wait_all(bar, (unsigned)(s + 1) * (unsigned)(l.blocks + 1), l.rounds);
    if (!ok) break;
    if (tid == 0) g->ctl.t += a.P.dt;
    for (int i = tid; i < NR + NL; i += nt) {
      if (i < NR) {
        int open = ryr[i];
        if (!a.P.nogating) {
          double q = res[i];
          open = srs_gate_ryr(gc, open, (float)ca(a.C.ryr_cleft[i], out), (float)ca(a.C.ryr_jsr[i], out), 0, 0,
                              &q, g->ctl.seed, (uint32_t)i, (uint64_t)step);
          res[i] = q;
        }
        // the RyR hold of the next step's protocol (cpu/RunSimulation.cpp:540-542)
        ryr[i] = open || i == hold;
      } else if (!a.P.nogating) {
        const int k = i - NR;
        double q = res[i];
        int st = lcc[k], vs = lccv[k];
        srs_gate_lcc(gc, &st, &vs, (float)ca(a.C.lcc_ele[k], out), &q, g->ctl.seed, (uint32_t)i, (uint64_t)step);
        lcc[k] = st;
        lccv[k] = vs;
        res[i] = q;
      }
    }
    if (tid == 0) g->ctl.step = step + 1;
    __syncthreads();
    // the protocol runs only at the steps where it has work
    if (step + 1 >= next_ev) {
      if (tid == 0) {
        prestep(a.P, a.C, g->ctl, ryr, lcc, lccv, a.CS.rows + (size_t)r * a.P.row_cap * a.P.row_w,
                [&](int e) { return ca(e, out); });
        g->next_ev = protocol_next_event(a.P, g->ctl, true);
      }
      __syncthreads();
      next_ev = g->next_ev;
    }
    // this block has read the state it needed: the element blocks may finish
    // the next step, after which they overwrite it
    if (tid == 0 && s + 1 < steps) red_release_add(bar, 1u);
  }
  __syncthreads();
  for (int i = tid; i < NR; i += nt) a.CS.ryr[rr + i] = ryr[i];
  for (int i = tid; i < NL; i += nt) {
    a.CS.lcc[rl + i] = lcc[i];
    a.CS.lccv[rl + i] = lccv[i];
  }
  for (int i = tid; i < NR + NL; i += nt) a.CS.res[rc + i] = res[i];
  if (tid == 0) {
    // the element blocks may be adding status bits of their own
    RealCtl* c = a.CS.ctl + r;
    const unsigned bits = g->ctl.status | (ok ? 0u : 2u);
    c->step = g->ctl.step;
    c->n_rows = g->ctl.n_rows;
    c->t = g->ctl.t;
    c->ca_max_tick = g->ctl.ca_max_tick;
    c->done = g->ctl.done;
    c->lcc_open = g->ctl.lcc_open;
    c->n_open_tick = g->ctl.n_open_tick;
    c->tick_idx = g->ctl.tick_idx;
    c->vsel = g->ctl.vsel;
    c->next_tick = g->ctl.next_tick;
    c->tick_cache_idx = g->ctl.tick_cache_idx;
    c->tick_cache_ver = g->ctl.tick_cache_ver;
    if (bits) atomicOr(&c->status, bits);
    if (ok) *bar = 0;  // every block has arrived for the last time
    else give_up(l);
  }
}

// ---- the channels of an element block ---------------------------------------------
// Shared memory of an element block that carries channels: gating constants,
// then per local channel its residual, state, (LCC) voltage gate and elements.
struct LocalChan {
  double* res;
  int32_t *id, *state, *vstate, *e0, *e1;  // id: RyR, or NR + LCC; e0: cleft or LCC element; e1: JSR
  const srs_gate_consts* gc;
  int n;
};

template <class Args>
__device__ LocalChan local_channels(const Args& a, const PlainLoop& l, int r, int b, unsigned char* smem) {
  LocalChan c;
  const int q0 = l.ch_ptr[b];
  c.n = l.ch_ptr[b + 1] - q0;
  srs_gate_consts* gc = reinterpret_cast<srs_gate_consts*>(smem);
  c.gc = gc;
  c.res = reinterpret_cast<double*>(smem + ((2 * sizeof(srs_gate_consts) + 15) & ~(size_t)15));
  c.id = reinterpret_cast<int32_t*>(c.res + l.ch_max);
  c.state = c.id + l.ch_max;
  c.vstate = c.state + l.ch_max;
  c.e0 = c.vstate + l.ch_max;
  c.e1 = c.e0 + l.ch_max;
  if (c.n == 0) return c;
  const int NR = a.C.NR, NL = a.C.NL;
  if (threadIdx.x < 2) gc[threadIdx.x] = a.P.gc[threadIdx.x];
  for (int i = threadIdx.x; i < c.n; i += blockDim.x) {
    const int id = l.ch_id[q0 + i];
    c.id[i] = id;
    c.res[i] = a.CS.res[(size_t)r * (NR + NL) + id];
    if (id < NR) {
      c.state[i] = a.CS.ryr[(size_t)r * NR + id];
      c.vstate[i] = 0;
      c.e0[i] = a.C.ryr_cleft[id];
      c.e1[i] = a.C.ryr_jsr[id];
    } else {
      c.state[i] = a.CS.lcc[(size_t)r * NL + id - NR];
      c.vstate[i] = a.CS.lccv[(size_t)r * NL + id - NR];
      c.e0[i] = a.C.lcc_ele[id - NR];
      c.e1[i] = 0;
    }
  }
  return c;
}

// Protocol state that the gating of an element block follows.
struct LocalProtocol {
  uint64_t seed;
  int64_t step, close_step;  // close_step: LCC closing still to come (-1: none)
  int vsel;
};
template <class Args>
__device__ LocalProtocol local_protocol(const Args& a, const RealCtl& c) {
  LocalProtocol p;
  p.seed = c.seed;
  p.step = c.step;
  p.vsel = c.vsel;
  p.close_step = a.P.run_protocol && a.P.flag_lcc && c.lcc_open ? c.lcc_close_step : -1;
  return p;
}
// prestep of step p.step as far as channels see it (the hold aside):
// returns whether the trigger LCC closes now.
template <class Args>
__device__ bool advance_protocol(const Args& a, LocalProtocol& p) {
  const bool close = p.close_step >= 0 && p.step >= p.close_step;
  if (close) p.close_step = -1;
  if (a.P.run_protocol && a.P.flag_vclamp) p.vsel = p.step < a.P.clamp_end ? 1 : 0;
  return close;
}

// Gates local channel i after step `step` from the Ca u0 (cleft or LCC element)
// and u1 (JSR) and applies the next step's protocol; returns whether it is open.
template <class Args>
__device__ __forceinline__ bool gate_local(const Args& a, const LocalChan& c, int i, const LocalProtocol& p,
                                           int v, bool close, float u0, float u1) {
  const int id = c.id[i], NR = a.C.NR;
  const int64_t step = p.step - 1;  // the step just taken
  if (id < NR) {
    int open = c.state[i];
    if (!a.P.nogating) {
      double q = c.res[i];
      open = srs_gate_ryr(c.gc + v, open, u0, u1, 0, 0, &q, p.seed, (uint32_t)id, (uint64_t)step);
      c.res[i] = q;
    }
    if (a.P.run_protocol && id == a.P.init_ryr && p.step < a.P.hold_end) open = 1;
    c.state[i] = open;
    return open != 0;
  }
  int st = c.state[i], vs = c.vstate[i];
  if (!a.P.nogating) {
    double q = c.res[i];
    srs_gate_lcc(c.gc + v, &st, &vs, u0, &q, p.seed, (uint32_t)id, (uint64_t)step);
    c.res[i] = q;
  }
  if (close && id - NR == a.P.lcc_index) st = 1;  // DEFAULT_STATE_LCC
  c.state[i] = st;
  c.vstate[i] = vs;
  return (st == 6 || st == 12) && vs == 2;
}
__device__ __forceinline__ bool open_local(const LocalChan& c, int i, int NR) {
  return c.id[i] < NR ? c.state[i] != 0 : (c.state[i] == 6 || c.state[i] == 12) && c.vstate[i] == 2;
}

// ---- FP32 ----------------------------------------------------------------------
// Block b of realization r = blockIdx.x / (blocks + 1): the last one is the
// protocol's, the others take E elements a thread.
template <int E>
__global__ void __launch_bounds__(PLAIN_LOOP_T32, 6) k_plain32_loop(const __grid_constant__ Plain32Args a,
                                                                    const __grid_constant__ PlainLoop l) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int r = blockIdx.x / (l.blocks + 1), b = blockIdx.x % (l.blocks + 1);
  const int steps = steps_of(a, l, a.CS.ctl[r]);
  if (steps <= 0) return;
  const int N = a.N;
  const size_t ro = (size_t)r * N;
  float4* M[2] = {const_cast<float4*>(a.M_in) + ro, a.M_out + ro};
  if (b == l.blocks) {
    gate_loop(a, l, r, steps,
              [&](int e, int buf) { return widen(a.rest_ca[e] + __ldcg(&M[buf][e].x)); }, smem);
    return;
  }
  const LocalChan ch = local_channels(a, l, r, b, smem);
  float* J = reinterpret_cast<float*>(ch.e1 + l.ch_max);  // flux of each local channel
  LocalProtocol lp = local_protocol(a, a.CS.ctl[r]);
  const int j0 = b * (PLAIN_LOOP_T32 * E) + threadIdx.x;
  auto element = [&](int t) { return min(j0 + t * PLAIN_LOOP_T32, N - 1); };  // the last one stands in
  auto valid = [&](int t) { return j0 + t * PLAIN_LOOP_T32 < N; };
  struct Geo {
    float4 co;
    int4 nb;
    float bsl, kb;
    uint32_t fl;
  };
  auto geometry = [&](int t) {
    const int e = element(t);
    return Geo{__ldg(a.a + e), __ldg(a.nb + e), __ldg(a.bsl + e), a.kb ? __ldg(a.kb + e) : 0.0f,
               __ldg(a.flags + e)};
  };
  float4 x[E], cm[E];
  float im[E], ci[E];
#pragma unroll
  for (int t = 0; t < E; ++t) {
    const size_t o = ro + element(t);
    x[t] = M[0][element(t)];
    im[t] = a.I_in[o];
    cm[t] = comp_load4(a.CMq + o);
    ci[t] = comp_load1(a.CIq[o]);
  }
  Geo geo = geometry(0);  // kept where a thread has one element
  unsigned* bar = l.bar + r;
  __syncthreads();
  bool ok = true;
  for (int s = 0; s < steps; ++s) {
    const float4* src = (s & 1) ? M[1] : M[0];
    float4* dst = (s & 1) ? M[0] : M[1];
    float4 n0, n1, n2, n3;
    auto neighbours = [&]() {
      n0 = __ldcg(src + geo.nb.x);
      n1 = __ldcg(src + geo.nb.y);
      n2 = __ldcg(src + geo.nb.z);
      n3 = __ldcg(src + geo.nb.w);
    };
    neighbours();
    if (ch.n > 0) {
      const int v = lp.vsel;
      const bool close = s > 0 && advance_protocol(a, lp);
      for (int i = threadIdx.x; i < ch.n; i += blockDim.x) {
        const bool ryr = ch.id[i] < a.C.NR;
        const float u0 = __ldcg(&src[ch.e0[i]].x), u1 = ryr ? __ldcg(&src[ch.e1[i]].x) : 0.0f;
        const float c0 = a.rest_ca[ch.e0[i]] + u0;
        const bool open = s > 0 ? gate_local(a, ch, i, lp, v, close, c0, ryr ? a.rest_ca[ch.e1[i]] + u1 : 0.0f)
                                : open_local(ch, i, a.C.NR);
        float f = 0.0f;
        if (open) f = ryr ? a.k.jr_scale * ((a.k.dc0 + u1) - u0)
                          : a.k.lccA[lp.vsel] * fmaf(c0, a.k.lccE[lp.vsel], -a.k.lccB);
        J[i] = f;
      }
      lp.step += 1;
      __syncthreads();
    }
#pragma unroll
    for (int t = 0; t < E; ++t) {
      if (t > 0) {
        geo = geometry(t);
        neighbours();
      }
      const int e = element(t);
      float flux = 0.0f;
      if (geo.fl & 4u)
        for (int q = a.chan_ptr[e]; q < a.chan_ptr[e + 1]; ++q) flux = fmaf(J[l.loc[q]], a.chan_list[q].s, flux);
      float4 out;
      float imo;
      tet_update(a.k, x[t], im[t], n0, n1, n2, n3, geo.co, geo.fl, geo.bsl, geo.kb, flux, cm[t], ci[t], &out, &imo);
      x[t] = out;
      im[t] = imo;
      // as stored between steps: compact halves
      const uint32_t c0 = comp_encode2(cm[t].x, cm[t].y), c1 = comp_encode2(cm[t].z, cm[t].w);
      const float2 d0 = comp_decode2(c0), d1 = comp_decode2(c1);
      cm[t] = make_float4(d0.x, d0.y, d1.x, d1.y);
      ci[t] = comp_load1(comp_store1(ci[t]));
      if (valid(t)) __stcg(dst + e, x[t]);
    }
    if (E > 1) geo = geometry(0);
    __syncthreads();
    if (threadIdx.x == 0) red_release_add(bar, 1u);
    if (s + 1 < steps && !wait_all(bar, (unsigned)(s + 1) * (unsigned)(l.blocks + 1), l.rounds)) {
      ok = false;
      break;
    }
  }
  unsigned bits = ok ? 0u : 2u;
#pragma unroll
  for (int t = 0; t < E; ++t) {
    if (!valid(t)) continue;
    const size_t o = ro + element(t);
    ((steps & 1) ? a.I_out : const_cast<float*>(a.I_in))[o] = im[t];
    comp_store4(a.CMq + o, cm[t]);
    a.CIq[o] = comp_store1(ci[t]);
    if (!isfinite(x[t].x)) bits |= 1u;
  }
  if (bits) atomicOr(&a.CS.ctl[r].status, bits);
  if (!ok && threadIdx.x == 0) give_up(l);
}

// ---- FP64 ----------------------------------------------------------------------
// A block takes E times 32 elements with four warps in four roles
// (srs_plain64_update.cuh); role 3 also gates the block's channels.  Blocks go
// to the SMs in turn; the roles move on by one warp with each turn, so that the
// blocks of an SM load its quarters evenly.
template <int E>
__global__ void __launch_bounds__(128, 6) k_plain64_loop(const __grid_constant__ Plain64Args a,
                                                         const __grid_constant__ PlainLoop l) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double s_ca[E][32];        // Ca of the block's elements
  __shared__ double s_rate[E][5][32];   // reactions: immobile buffer, SERCA, dye, ATP, CMDN
  const int r = blockIdx.x / (l.blocks + 1), b = blockIdx.x % (l.blocks + 1);
  const int steps = steps_of(a, l, a.CS.ctl[r]);
  if (steps <= 0) return;
  const int N = a.N;
  const size_t ro = (size_t)r * 6 * N;
  double* S[2] = {const_cast<double*>(a.S_in) + ro, a.S_out + ro};
  if (b == l.blocks) {
    gate_loop(a, l, r, steps, [&](int e, int buf) { return __ldcg(S[buf] + e); }, smem);
    return;
  }
  const LocalChan ch = local_channels(a, l, r, b, smem);
  double* J = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(ch.e1 + l.ch_max) + 7) & ~(uintptr_t)7);
  // a closed channel adds nothing to the rate, not even zero
  const double closed = __longlong_as_double((long long)kClosed);
  LocalProtocol lp = local_protocol(a, a.CS.ctl[r]);
  const int lane = threadIdx.x & 31, role = ((threadIdx.x >> 5) + blockIdx.x / l.n_sm) & 3;
  const int j0 = b * (PLAIN_LOOP_TILE64 * E) + lane;
  auto element = [&](int t) { return min(j0 + t * 32, N - 1); };  // the last one stands in
  auto valid = [&](int t) { return j0 + t * 32 < N; };
  const double dt = a.P.dt;
  const size_t n = N;
  const int sp0 = role64_x0(role), sp1 = role64_x1(role);
  double x0[E], x1[E];
#pragma unroll
  for (int t = 0; t < E; ++t) {
    x0[t] = S[0][sp0 * n + element(t)];
    x1[t] = role == 1 || role == 2 ? S[0][sp1 * n + element(t)] : 0.0;
    if (role == 0) s_ca[t][lane] = x0[t];
  }
  Geo64 geo = geometry64(a, element(0));  // kept where a lane has one element
  unsigned* bar = l.bar + r;
  __syncthreads();
  bool ok = true;
  for (int s = 0; s < steps; ++s) {
    const double* src = (s & 1) ? S[1] : S[0];
    double* dst = (s & 1) ? S[0] : S[1];
    double b_ca[E];
#pragma unroll
    for (int t = 0; t < E; ++t) {
      if (t > 0) geo = geometry64(a, element(t));
      const int e = element(t);
      if (role == 3 && t == 0 && ch.n > 0) {
        const int v = lp.vsel;
        const bool close = s > 0 && advance_protocol(a, lp);
        for (int i = lane; i < ch.n; i += 32) {
          const bool ryr = ch.id[i] < a.C.NR;
          const double u0 = __ldcg(src + ch.e0[i]), u1 = ryr ? __ldcg(src + ch.e1[i]) : 0.0;
          const bool open = s > 0 ? gate_local(a, ch, i, lp, v, close, (float)u0, (float)u1)
                                  : open_local(ch, i, a.C.NR);
          double f = closed;
          if (open) {
            const int w = lp.vsel;
            f = ryr ? a.P.v_ryr * (u1 - u0) * a.P.v_cell
                    : a.P.lccA[w] * (u0 * a.P.lccE[w] - a.P.lccB) / a.P.lccEm1[w];
          }
          J[i] = f;
        }
        lp.step += 1;
      }
      b_ca[t] = role64(a, role, geo, e, lane, src, s_ca[t][lane], x0[t], x1[t], s_rate[t]);
      if (role >= 2 && valid(t)) {
        __stcg(dst + sp0 * n + e, x0[t]);
        if (role == 2) __stcg(dst + n + e, x1[t]);
      }
    }
    __syncthreads();
    if (role == 0) {
#pragma unroll
      for (int t = 0; t < E; ++t) {
        const int e = element(t), fl = E > 1 ? __ldg(a.flags + e) : geo.fl;
        const double c = s_ca[t][lane];
        double bc = sum64(a, fl, lane, c, b_ca[t], s_rate[t]);
        if (fl & 4) {
          for (int q = a.chan_ptr[e]; q < a.chan_ptr[e + 1]; ++q) {
            const double f = J[l.loc[q]];
            if (bits64(f) == kClosed) continue;
            if (a.chan_list[q].kind == 1) bc -= f / a.v0[e];
            else bc += f / a.v0[e];
          }
        }
        bc = fast_buffer64(a, bc, c, __ldg(a.bhi + e), __ldg(a.blo + e));
        x0[t] = c + bc * dt;
        s_ca[t][lane] = x0[t];
        if (valid(t)) __stcg(dst + e, x0[t]);
      }
    }
    if (E > 1) geo = geometry64(a, element(0));
    __syncthreads();
    if (threadIdx.x == 0) red_release_add(bar, 1u);
    if (s + 1 < steps && !wait_all(bar, (unsigned)(s + 1) * (unsigned)(l.blocks + 1), l.rounds)) {
      ok = false;
      break;
    }
  }
  double* fin = (steps & 1) ? S[1] : S[0];
  unsigned bits = ok ? 0u : 2u;
#pragma unroll
  for (int t = 0; t < E; ++t) {
    if (!valid(t)) continue;
    if (role == 1) {
      fin[3 * n + element(t)] = x0[t];
      fin[4 * n + element(t)] = x1[t];
    }
    if (role == 0 && !finite64(x0[t])) bits |= 1u;
  }
  if (bits) atomicOr(&a.CS.ctl[r].status, bits);
  if (!ok && threadIdx.x == 0) give_up(l);
}

template <class K>
bool loop_fits(K kernel, int threads, size_t smem, int64_t blocks) {
  int dev = 0, n_sm = 0, per = 0, coop = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  if (!coop || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return blocks <= (int64_t)per * n_sm;
}

}  // namespace

// Whether that many blocks of per_thread elements a thread (FP64: a lane) are
// resident on the device at once.
bool plain_loop_fits(bool f64, int per_thread, int64_t blocks, size_t smem) {
  if (f64)
    return per_thread == 1   ? loop_fits(k_plain64_loop<1>, 128, smem, blocks)
           : per_thread == 2 ? loop_fits(k_plain64_loop<2>, 128, smem, blocks)
                             : loop_fits(k_plain64_loop<4>, 128, smem, blocks);
  return per_thread == 1   ? loop_fits(k_plain32_loop<1>, PLAIN_LOOP_T32, smem, blocks)
         : per_thread == 2 ? loop_fits(k_plain32_loop<2>, PLAIN_LOOP_T32, smem, blocks)
                           : loop_fits(k_plain32_loop<4>, PLAIN_LOOP_T32, smem, blocks);
}

static int launch_loop(const void* kernel, int threads, const void* a, int R, const PlainLoop& l, size_t smem,
                       cudaStream_t st) {
  void* args[] = {const_cast<void*>(a), const_cast<PlainLoop*>(&l)};
  return cudaLaunchCooperativeKernel(kernel, dim3(R * (l.blocks + 1)), dim3(threads), args, smem, st) ==
                 cudaSuccess ? 0 : -1;
}
int launch_plain32_loop(const Plain32Args& a, const PlainLoop& l, size_t smem, cudaStream_t st) {
  const void* k = l.per_thread == 1   ? (const void*)k_plain32_loop<1>
                  : l.per_thread == 2 ? (const void*)k_plain32_loop<2>
                                      : (const void*)k_plain32_loop<4>;
  return launch_loop(k, PLAIN_LOOP_T32, &a, a.R, l, smem, st);
}
int launch_plain64_loop(const Plain64Args& a, const PlainLoop& l, size_t smem, cudaStream_t st) {
  const void* k = l.per_thread == 1   ? (const void*)k_plain64_loop<1>
                  : l.per_thread == 2 ? (const void*)k_plain64_loop<2>
                                      : (const void*)k_plain64_loop<4>;
  return launch_loop(k, 128, &a, a.R, l, smem, st);
}

}  // namespace srs
