// srs_engine.h — host-side declarations of the kernel launchers and the
// argument blocks they take (definitions in k_plain64.cu and k_fp32.cu).
#pragma once
#include "srs_comp.h"
#include <cuda_runtime.h>

#include "../../include/srs_gb300.h"
#include "srs_sim.cuh"

namespace srs {

struct Plain64Args {
  int32_t N, R;
  const double* aij;
  const int32_t* nij;
  const double* br;
  const double* v0;
  const double* bhi;
  const double* blo;
  const int32_t* flags;
  const int32_t* chan_ptr;
  const ChanEntry* chan_list;
  const double* S_in;
  double* S_out;
  double p[56];
  double nsr;
  // terms of the SERCA flux that do not depend on the element, and 1 / K_D_i
  // (zero where its exponent is extreme), filled by plain64_consts
  double sd0, sd1, sd2, sn1, sn0, inv_kdi;
  Protocol P;
  Channels C;
  ChanState CS;
  unsigned int* counters;
};
void plain64_consts(Plain64Args* a);
// Step index, Philox keys and status word of an allocation-free step, with the
// launch itself (empty for the engine's own steps, which read RealCtl).
template <bool KEYS>
struct Plain64Keys {};
template <>
struct Plain64Keys<true> {
  int64_t step;
  unsigned* status;  // may be null
  uint64_t seeds[SRS_NOALLOC_MAX_REALIZATIONS];
};
bool plain64_keys_fit(const Plain64Args& a);
int launch_plain64_keys(const Plain64Args& a, const Plain64Keys<true>& k, cudaStream_t st);
int launch_plain64_step(const Plain64Args& a, cudaStream_t st);
int launch_plain64_prestep(const Plain64Args& a, int write_initial_row, cudaStream_t st);

struct Consts32 {
  float D[4];
  float kon[5], koff[5], bfree[5];
  float c0, c0j;
  float inv_kdi;
  float sd0, sd1, sd2;
  float sn1, sn0;
  float serca_scale;
  float refill_v, refill0;
  float khi;
  float dt;
  float jr_scale;
  float dc0;
  float lccA[2], lccE[2], lccB;
  // |Ca| below which the divisions of the element update stay in the range of
  // srs_div_in_range (srs_math.h); negative: never
  float div_cmax;
};

struct ChanEntry32 {
  int32_t kind;
  int32_t ch;
  float s;
  int32_t pad;
};

struct Plain32Args {
  int32_t N, R;
  const float4* a;
  const int4* nb;
  const float* bsl;
  const float* kb;
  const uint32_t* flags;
  const int32_t* chan_ptr;
  const ChanEntry32* chan_list;
  const float* rest_ca;
  const float4* M_in;
  const float* I_in;
  float4* M_out;
  float* I_out;
  float4* CM;  // [R][N] compensation of the Euler update (mobile species)
  float* CI;   // [R][N] compensation (immobile buffer)
  // compact compensation (srs_comp.h): when set (always, in the plain
  // engine), these hold the compensation and CM / CI are unused.  The
  // kernels keep the float branch: without it the 40-register update
  // measured 6 % slower (0.472 against 0.445 ms per large-mesh step).
  ushort4* CMq;  // [R][N]
  uint16_t* CIq;  // [R][N]
  Consts32 k;
  Protocol P;
  Channels C;
  ChanState CS;
  unsigned int* counters;
  int32_t pf_rows;  // split form: element blocks ahead whose state is prefetched into L2
  // trajectory recording for the adjoint (null: none): the slot of this
  // step, [R][N] x_{n-1} and (immobile buffer, Ca rate before the
  // rapid-buffer factor), and [R][NR + 2 NL + 1] the channel states the step
  // used (RyR, LCC, LCC voltage state, voltage selector)
  float4* traj_u;
  float2* traj_ig;
  int32_t* traj_ch;
  float* traj_ib;  // [R][N] 1 / B(x_{n-1}), B the rapid-buffer factor
};
// Meshes of at least this many elements take the split form of the plain
// FP32 step (element update, then gating, as two launches).
constexpr int PLAIN32_SPLIT_N = 65536;
int plain32_kernels_per_step(const Plain32Args& a);
int launch_plain32_step(const Plain32Args& a, cudaStream_t st);
int launch_plain32_prestep(const Plain32Args& a, int write_initial_row, cudaStream_t st);

// The plain engines' steps in one launch (k_plain_loop.cu).  S_in / M_in / I_in
// are buffer 0 of the state, S_out / M_out / I_out buffer 1; after n steps the
// state is in buffer n % 2.
struct PlainLoop {
  int32_t steps;
  int32_t blocks;         // element blocks per realization
  int32_t per_thread;     // elements a thread (FP64: a lane of each of four warps) takes
  int32_t n_sm;
  int32_t rounds;         // of 65,536 polls in one wait before a block gives up
  unsigned* bar;          // [R] arrivals at the step barriers, zero before and after a launch
  unsigned* gave_up;      // set when a wait gave up: later launches do nothing
  unsigned* timeout;      // pinned host word, set with it
  int32_t ch_max;         // most channels an element block gates
  const int32_t* ch_ptr;  // [blocks + 1] CSR of the channels each block gates
  const int32_t* ch_id;   // RyR, or NR + LCC
  const int32_t* loc;     // per entry of chan_list: the channel's place in its block's list
};
constexpr int PLAIN_LOOP_T32 = 128;
constexpr int PLAIN_LOOP_TILE64 = 32;  // elements of an FP64 block
size_t plain_loop_smem_bytes(int NR, int NL, int ch_max);
bool plain_loop_fits(bool f64, int per_thread, int64_t blocks, size_t smem);
int launch_plain32_loop(const Plain32Args& a, const PlainLoop& l, size_t smem, cudaStream_t st);
int launch_plain64_loop(const Plain64Args& a, const PlainLoop& l, size_t smem, cudaStream_t st);

// Element record of the resident engine.  On the device its two halves lie
// apart (ResidentArgs geo_a, geo_b): a warp's 32 records are then two loads of
// 512 consecutive bytes, eight shared-memory/L1 wavefronts instead of sixteen.
struct __align__(16) TetRec {
  float a[4];
  uint16_t nb[4];
  float bsl;
  uint32_t flags;
};

// Per-element record of the reverse sweep (halves apart on the device, as
// TetRec).
struct __align__(16) AdjRec {
  float aT[4];     // coefficient of this element in each neighbour's row
  uint16_t nb[4];  // neighbour codes of the adjoint's CTA grouping
  float bsl;       // SL capacity x K_D; sign bit set: the element has troponin C
  float sa;        // sum of the element's own off-diagonal coefficients; sign bit
                   // set: JSR element
};

// Largest CTA of the resident engine (its kernel's launch bound).
#define SRS_RESIDENT_MAX_THREADS 640

struct ResidentArgs {
  int32_t R;
  int32_t P;
  int32_t off_bits;
  int32_t steps;
  const float4* geo_a;  // coefficients
  const float4* geo_b;  // neighbour codes, bsl, flags
  int32_t group;          // threads of the channel group (resident_group)
  srs_gate_consts* gc;    // [2] gating constants by potential, written before each launch; null: staged in
                          // shared memory
  int32_t prestep_first;  // run the protocol of the first step before it
  int32_t initial_row;    // ... and write the t = 0 states row
  const int32_t* n_local; // [C] elements in each partition
  const int32_t* n_chtet; // [1] channel elements (partition 0, offsets 0..n-1)
  const int32_t* n_int;   // [C] interior elements (all neighbours in the same
                          // partition), right after the channel elements
  int32_t ch_interior;    // every channel element is interior to partition 0
  int32_t speculate;      // allow updating interior elements before the
                          // barrier completes where no realization can
                          // finish inside the launch (decided per realization)
  const int32_t* ch_ptr;  // [n_chtet+1] CSR of channel entries per channel element
  const ChanEntry32* ch_list;
  const uint16_t* ryr_cleft_code;
  const uint16_t* ryr_jsr_code;
  const uint16_t* lcc_code;
  const float* lcc_rest;
  float4* M;   // [R][C][P] state
  float* I;
  float4* CM;  // [R][C][P] compensation
  float* CI;
  Consts32 k;
  Protocol P_;
  Channels C;
  ChanState CS;
  // Trajectory recording (null: off).  Step s of the launch stores the state
  // it starts from (traj_u slot s and traj_ig.x), its Ca rate before the
  // rapid-buffer factor (traj_ig.y) and the channel states it uses (traj_ch
  // slot s: RyR[NR], LCC[NL], LCC V-gate[NL], voltage selector); slot
  // `steps` of traj_u/traj_ig holds the final state.  Layout [slot][R][C*P].
  float4* traj_u;
  float2* traj_ig;
  int32_t* traj_ch;
  float* traj_ib;  // [R][N] 1 / B(x_{n-1}), B the rapid-buffer factor
};
// Line scan: F[r][i] = pad[i] + sum_q w[q] * dye(col[q]) over ptr[i]..ptr[i+1].
struct LinescanArgs {
  int32_t n_samples;
  int32_t n_state;       // elements per realization in the engine layout
  const int32_t* ptr;    // [n_samples + 1]
  const int32_t* col;    // engine element indices
  const double* w;       // V0 * PSF weight
  const double* pad;     // [n_samples] padding-voxel contribution
  const double* S64;     // FP64 engine state [R][6][N] (or null)
  const float4* M;       // FP32 engines: deviations [R][n_state]
  const float4* CM;      //   and their compensation terms
  const ushort4* CMq;    //   (or in compact form, srs_comp.h)
  const double* rest_dye;  // [n_state] resting bound dye per element
  double* out;           // [R][n_samples]
  // tiled form (linescan_tiled): per group of eight samples the elements that any
  // of them weighs, by element chunk
  int32_t n_chunk;       // chunks of LINESCAN_CHUNK engine elements
  const int32_t* tptr;   // [groups][n_chunk + 1]
  const uint32_t* tent;  // (sample mask << 24) | offset in the chunk
  const double* tw;      // [entry][8]
  int32_t splits;        // blocks the chunks are dealt to
  const int32_t* split;  // [splits + 1] first chunk of each
  double* part;          // [splits][R][n_samples]
};
constexpr int LINESCAN_CHUNK = 64;
int linescan_splits(int n_samples, int n_state, int R, int n_sm);
int launch_linescan(const LinescanArgs& a, int R, cudaStream_t st);

// ---- state exchange (k_state.cu) ----------------------------------------------
struct ExportArgs {
  int32_t N, NR, NL;
  const double* S64;            // FP64 engine: the realization's state [6][N]; or the FP32 engines':
  const float4* M;              // the realization's arrays in engine order
  const float* I;
  const float4* CM;
  const float* CI;
  const ushort4* CMq;           // (compensation compact, when set)
  const uint16_t* CIq;
  const int32_t* eng_of_ref;    // [N]
  const uint32_t* flags;        // bit 0 JSR, bit 1 troponin C, by engine element
  int32_t flag_stride;          // words between elements' flags
  double rest[6], rest_ca_jsr;  // Ca (cytosol), ATP, CMDN, TRPN, CSQN, dye; Ca (JSR)
  const int32_t *ryr, *lcc, *lccv;
  const double* res;
  double* S;                    // outputs (null: not wanted)
  int32_t *ryr_out, *lcc_out, *lccv_out;
  double* res_out;
};
int launch_export_state(const ExportArgs& a, cudaStream_t st);
struct ExportLambdaArgs {
  int32_t N;
  size_t NE;                    // elements per realization in the engine's arrays
  const float4* lam;            // [R][NE]
  const float* lam_im;
  const float4* c4;             // compensation, or compact when c4q / cimq are set
  const float* cim;
  const ushort4* c4q;
  const uint16_t* cimq;
  const int32_t* eng_of_ref;
  const uint32_t* flags;        // as in ExportArgs
  int32_t flag_stride;
  double* g;                    // [R][6][N]
};
int launch_export_lambda(const ExportLambdaArgs& a, int R, cudaStream_t st);
template <class T>  // double, float
int launch_broadcast_state(const T* src, T* dst, size_t n, int R, cudaStream_t st);

// ---- total Ca per compartment (k_mass.cu) ------------------------------------
struct MassArgs {
  int32_t n_state;        // elements per realization in the engine layout
  const double* v0;       // [n_state] volume (0 for padding slots)
  const uint8_t* jsr;     // [n_state] 1 for JSR elements
  const double* bhi;      // [n_state] rapid SL buffer capacities (uM)
  const double* blo;
  double khi, klo;
  int32_t n_sl;           // elements with rapid buffers, and their list
  const int32_t* sl;
  const double* S64;      // FP64 engine state [R][6][n_state], or null
  const float4* M;        // FP32 engines: deviations and compensation
  const float4* CM;
  const float* I;
  const float* CI;
  const ushort4* CMq;     // compact compensation (srs_comp.h), when set
  const uint16_t* CIq;
  const double* rest_ca;  // [n_state] resting Ca
  const double* rest_sum; // [n_state] resting total of the five species
  double* part;           // [R][blocks][2]: the blocks' sums
  double* out;            // [R][2]: cytosol, JSR
};
int total_ca_blocks(int n_state, int R, int n_sm);
int launch_total_ca(const MassArgs& a, int R, int blocks, cudaStream_t st);
int launch_division_check(int32_t b_first, int32_t b_step, int32_t n_b, int32_t ea, int32_t eb, int64_t* wrong,
                          cudaStream_t st);
int launch_comp_round_trip(const float* in, float* out, int64_t n, int packed, cudaStream_t st);

// ---- pathwise adjoint (k_adjoint.cu) ---------------------------------------
// FP32 constants of the Jacobian beyond Consts32.
struct AdjConsts {
  float brest[5];      // resting bound buffer: dye, ATP, CMDN, TRPN, CSQN
  float inv_btot_sl;   // 1 / B_TOT_SL_HI (0 when B_TOT_SL_HI = 0)
  float serca_per_ap;  // dF_Ca/dA_P = -serca_per_ap * v_cycle / B
  float v_cell;        // V_CELL
  float inv_khi;       // 1 / K_D_SL_HI
  // Dirichlet faces hold the mobile buffers at their resting bound level
  // c0 B / (Kd + c0), Kd = koff / kon, so their source D kb Bv depends on kon
  // and koff: d(source)/dkon = kb * kb_on[q], d(source)/dkoff = kb * kb_off[q]
  // (q: dye, ATP, CMDN)
  float kb_on[3];
  float kb_off[3];
};

constexpr int ADJ_MAX_THREADS = 640;  // of a reverse-sweep CTA, at 96 registers
struct AdjArgs {
  int32_t R, P, off_bits;  // P: forward partition stride; off_bits of the codes in geo
  int32_t m_sub;           // forward partitions per CTA (CTA slots m_sub * P)
  int32_t ch_off_bits;     // off_bits of the forward layout (channel codes)
  int32_t n_steps;  // steps of the segment; the kernel runs t = n_steps .. 1
  int64_t s0;       // global index of the state the segment starts from
  const float4* geo_a;  // [C*P] per-element records of the CTA grouping: coefficients
  const float4* geo_b;  // ... neighbour codes, bsl, sa
  const int32_t* n_local;
  const int32_t* n_chtet;
  const int32_t* n_int;    // [C] interior elements after the channel elements
  int32_t ch_interior;     // every channel element is interior to partition 0
  const int32_t* ch_ptr;
  const ChanEntry32* ch_list;
  const uint16_t* ryr_cleft_code;
  const uint16_t* ryr_jsr_code;
  const float* ryr_s_cl;  // +1/V0 of each RyR's cleft element
  const float* ryr_s_js;  // -1/V0 of each RyR's JSR element
  int32_t NR, NL;
  const float4* traj_u;    // trajectory of the segment (ResidentArgs layout)
  const float2* traj_ig;  // (immobile buffer, Ca rate before the rapid-buffer factor)
  const int32_t* traj_ch;
  int32_t tick_every;      // loss ticks at global steps that are multiples
  int32_t n_samples;
  const double* coef;      // [tick slot][R][n_samples] dL/dF at the ticks of the segment
  const int32_t* wt_ptr;   // [C*P + 1] element -> line-scan samples
  const int32_t* wt_idx;
  const double* wt_w;
  float4* lam;   // [R][C*P] (Ca, ATP, CMDN, dye) at segment boundaries
  float* lam_im; // [R][C*P] immobile buffer
  float4* lam_c4;  // Kahan compensation
  float* lam_cim;
  float* lam_c;    // [R][C*P] lambda_Ca within a segment (when not on chip)
  int32_t own_in_smem;  // owner state of lambda in shared memory
  int32_t stage;        // trajectory staged in shared memory by bulk copies
  unsigned int* status; // bit 0: a staging wait gave up
  double* grad;  // [R][SRS_N_ADJ]
  Consts32 k;
  AdjConsts ak;
};

struct AdjTickArgs {
  int32_t n_samples, n_state, n_ticks, R;
  int32_t tick0;        // global index of the segment's first tick
  int32_t n_seg_ticks;  // ticks of the segment (grid z)
  int64_t slot_stride;  // trajectory elements between consecutive ticks
  const int32_t* ptr;
  const int32_t* col;
  const double* w;
  const double* base;    // [n_samples] pad + resting dye part
  const double* f0;
  const double* target;  // [R][n_ticks][n_samples] or null
  const float4* traj_u;  // trajectory slot of the first tick [R][n_state]
  double* coef;          // [n_seg_ticks][R][n_samples]
  double* loss;          // [n_ticks][R][n_samples]: loss terms of every tick
  int32_t mean_trace;    // loss on the realizations' mean trace (target [n_ticks][n_samples])
};

// Reverse step of the plain FP32 engine's adjoint (k_adjoint_plain.cu); all
// arrays [R][N] in the plain engine's numbering unless noted.
struct AdjPlainArgs {
  int32_t N, R, NR, NL, n_samples;
  int32_t last;            // t == 1: write the boundary lambda instead of nxt
  const float4* aT;        // [N] coefficient of this element in each neighbour's row
  const int4* nb;          // [N] neighbours
  const float2* bs;        // [N] (bsl, TropC in the sign bit; sum a + kb, JSR in the sign bit)
  const float* kb;         // [N] Dirichlet rate kb, or null when the mesh has none
  const uint32_t* flags;   // [N] bit 2: the element carries channel entries
  const int32_t* ch_ptr;
  const ChanEntry32* ch_list;
  const int32_t* ryr_cleft;
  const int32_t* ryr_jsr;
  const float* ryr_s_cl;   // +1/V0 of each RyR's cleft element
  const float* ryr_s_js;   // -1/V0 of each RyR's JSR element
  const float4* tu;        // trajectory slot of x_{n-1}
  const float2* tig;       // (immobile buffer, Ca rate) of x_{n-1}
  const float* ib;         // [R][N] 1 / B of the state the published slots divide by:
                           // x_{n-2} (step, t > 1) or x_{s1-1} (publish)
  const int32_t* rec;      // [R][NR + 2 NL + 1] channel states of step n
  const double* coef_cur;  // publish: dL/dF of the tick at s1 ([R][n_samples]) or null
  const double* coef_next; // step: dL/dF of the tick at n - 1 or null
  const int32_t* wt_ptr;   // [N + 1] element -> line-scan samples
  const int32_t* wt_idx;
  const double* wt_w;
  const float4* pub;
  float4* nxt;
  float* lam_c;
  float* lam_im;
  // Kahan compensation of lambda as halves (srs_comp.h), like the forward
  // state's
  ushort4* lam_c4q;
  uint16_t* lam_cimq;
  float4* lam;             // boundary lambda (Ca, ATP, CMDN, dye)
  double* part;            // [R][blocks][SRS_N_ADJ] FP64 gradient rows of the blocks
  Consts32 k;
  AdjConsts ak;
};
int adjp_blocks_per_realization(int N, int R, int n_sm);
int launch_adjp_publish(const AdjPlainArgs& a, int blocks, cudaStream_t st);
int launch_adjp_step(const AdjPlainArgs& a, int blocks, cudaStream_t st);

size_t adjoint_smem_bytes(int P, int n_chtet, int n_entries, bool own_in_smem, bool stage);
int launch_adjoint(const AdjArgs& a, int C, int n_clusters, int threads, size_t smem,
                   cudaStream_t st);
int adjoint_max_clusters(int C, int threads, size_t smem);
int launch_adj_tick(const AdjTickArgs& a, cudaStream_t st);

// Host-side constants (double precision, from the parameter set and the
// membrane potential V): gating rates and the LCC flux terms.
void gate_consts(const srs_params& p, double V, srs_gate_consts* g);
void lcc_flux_consts(const srs_params& p, double V, double* A, double* E, double* Em1, double* B,
                     double* Vg);

size_t resident_smem_bytes(int P, int NR, int NL, int n_chtet, int n_entries, bool gc);
// per cluster size (k_res_*.cu)
#define SRS_RESIDENT_DECLARE(CC)                                                            \
  int launch_resident_c##CC(const ResidentArgs& a, int n_clusters, int threads, size_t smem, \
                            cudaStream_t st);                                              \
  int resident_max_clusters_c##CC(int threads, size_t smem);
SRS_RESIDENT_DECLARE(1)
SRS_RESIDENT_DECLARE(2)
SRS_RESIDENT_DECLARE(3)
SRS_RESIDENT_DECLARE(4)
SRS_RESIDENT_DECLARE(5)
SRS_RESIDENT_DECLARE(6)
SRS_RESIDENT_DECLARE(8)
SRS_RESIDENT_DECLARE(16)
#undef SRS_RESIDENT_DECLARE
// Threads of partition 0 that own the channel elements and gate the channels:
// three warps, the last one for the LCCs, where the step waits for the
// channels (large CTAs: 3.81 -> 2.93 us per step of a 16-CTA cluster of 320
// threads); two where the elements bound it and a third warp is missed there
// (1024 realizations, 8 x 192 threads: 117 against 126 us).  A larger group leaves
// partition 0 fewer elements and the others more: where they do not fit any more
// the group is of two warps (`wide` false).
constexpr int resident_group(int threads, bool wide) {
  return wide && threads >= 320 ? 96 : threads >= 128 ? 64 : 32;
}
int launch_resident(const ResidentArgs& a, int C, int n_clusters, int threads, size_t smem,
                    cudaStream_t st);
int resident_max_clusters(int C, int threads, size_t smem);
bool resident_cluster_supported(int C);

}  // namespace srs
