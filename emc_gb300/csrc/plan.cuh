// The fused-iteration plan: workspace layout and kernels shared by the FP32
// and tensor-core paths.
#pragma once
#include <cuda_fp16.h>

#include <vector>

#include "common.cuh"
#include "kernels.cuh"

// Rotations per E-step tile; LSE partials are kept per tile of this many rows.
#define EMC_RT 128

namespace emc {
struct IterReport;  // what the host reads after an iteration
}

struct emc_plan {
  emc_ctx* ctx = nullptr;
  emc_plan_desc d{};
  int n2 = 0;      // side*side
  int P_eff = 0;   // pixels with mask != 0
  int Kp = 0;      // P_eff padded (128)
  int Np = 0;      // patterns padded (128)
  int Rp = 0;      // rotations padded (128)
  int n_rt = 0;    // rotation tiles of EMC_RT
  bool bound = false;
  bool counts_fp16_exact = false;  // every count is an integer in [0, 2048]
  bool counts_integer = false;     // every count is an integer in [0, 65504]
  int count_max = 0;               // the largest count
  int counts_round = 0;            // tensor path: counts above 2048 rounded to FP16
  // the likelihood's count operands are k and k (k - 1) times this power of two
  // (set at bind; 1 for true Poisson)
  float count_scale = 1.0f / 128.0f;

  // bound inputs (caller owned)
  const float* images = nullptr;
  const int* mask = nullptr;
  const float *x = nullptr, *y = nullptr, *z = nullptr;
  const float* rot = nullptr;
  const float* rotw = nullptr;

  // compacted geometry
  int* pix = nullptr;                          // [Kp], -1 padding
  float *cx = nullptr, *cy = nullptr, *cz = nullptr;  // [Kp]

  // pattern operands, rows of Kp (FP32 path)
  float* Kraw = nullptr;  // k (x c_i when normalising); FP32 plans only
  double* ksum_part = nullptr;  // [N][Kp / 256] block sums of k
  std::vector<int> h_mask, h_pix;  // the bound mask and its compacted pixels (re-binds)
  float fused_scale = 0.0f;  // count_scale of FP16 counts written by the pattern pass (0: none)
  float* Kt = nullptr;    // k if k > 1e-10 else 0
  float* Ksum = nullptr;  // [N] sum_p k
  float* cnorm = nullptr; // [N] c_i (1 when not normalising)

  // pattern operands (tensor-core path), rows of Kp, times count_scale
  __half* Kh = nullptr;      // k
  __half* Jh = nullptr;      // fp16(j), j = k (k - 1): written in blocks with a count above 1
  __half* Jl = nullptr;      // j - Jh: written in blocks where it is not 0
  float *ktot = nullptr, *k2tot = nullptr;  // [Np] sum k, sum k^2 (exact, then rounded)
  // some pattern's sum k^2 or count is beyond FP32 differences (found at bind; the
  // likelihood then sums over the covered pixels): the device's word for it, ours
  int* d_bright = nullptr;
  bool bright = false;
  unsigned char* blk_bits = nullptr;  // [Np/128][Kp/64] what the block holds (es::kJ ..)
  // the blocks each pattern tile (and pair of tiles) has counts in, with their
  // bits: index << 8 | bits, in order; never empty
  uint32_t *pt_list = nullptr, *pp_list = nullptr;
  int *pt_n = nullptr, *pp_n = nullptr;
  unsigned char* blk_live = nullptr;  // [Kp/64] some pattern counts there
  // M-step: [Kp/64][Np/64] the (64-pixel, 64-pattern) block holds a count; per
  // 256-pixel tile the pattern blocks that hold one (never none) as a map and a list
  unsigned char *sub_any = nullptr, *ms_map = nullptr;
  int *ms_list = nullptr, *ms_n = nullptr;
  // [Np/128 + 1] K . H takes H's lo half on the 64-pixel blocks below lo_kb[pt]:
  // the blocks after it hold at most hlo_tail_ppm / 1e6 of every pattern's
  // counts (EMC_OPT_HLO_TAIL; 0: every block); lo_kb[Np/128] is the largest
  int* lo_kb = nullptr;
  int hlo_tail_ppm = 300000;
  int glo_tail_ppm = 1000;  // what EMC_OPT_GLO_TAIL reads: its last value set
  // [2][Rp/128][Kp/64] per iteration: a slice value s <= 0 / in (0, 1e-10) among
  // the tile's rotations and the block's pixels
  unsigned char* rot_flags = nullptr;
  __half* KhT = nullptr;     // [Kp][Np] transposed counts for the M-step

  // rotation side, per iteration
  float* S = nullptr;       // [Rp][Kp] slice at the compacted pixels (FP32 path)
  float* rot_cnt = nullptr; // [Rp] count_r (pixels with s > 0)
  float* rot_A = nullptr;   // [Rp] sum s^2/(s+c) over s > 0
  float* rot_ssum = nullptr;// [Rp] sum max(s, floor) (true Poisson)

  // responsibilities
  float* L = nullptr;      // [R][N] log-likelihood, then normalised responsibility
  float* PHI = nullptr;    // [R][N] scaling
  float* Q = nullptr;      // [R][N] responsibility / scaling (FP32 M-step)
  __half* Qh = nullptr;    // [Rp][Np] hi (tensor-core M-step)
  __half* Ql = nullptr;    // [Rp][Np] lo
  float* qscale = nullptr; // [Rp] 2^-e_r of the Q rows
  float2* part = nullptr;  // [n_rt][N] (max, sumexp) per rotation tile
  double* lse = nullptr;   // [N]
  float2* lse2 = nullptr;  // [N] lse as float hi + lo
  float* lse_shifted = nullptr;  // [4][2][Np] the same in four alignments (LseOut)
  const double* ll_src = nullptr;  // what the report adds (own_loglik)
  int ll_n = 0;
  double* ll_part = nullptr;  // [N/32] sums of lse
  float* T = nullptr;      // [Rp] rotation totals
  double* red = nullptr;   // reduction scratch (small)
  ulonglong2* fix2 = nullptr;  // [s^3] fixed-point (model, weight) sums (deterministic insert)
  float2* acc2 = nullptr;  // [s^3] interleaved (model, weight) sums (float atomics)
  int* flags = nullptr;    // device status words
  float* sigma_dev = nullptr;  // [1] annealing width read by the E-step kernels
  emc::BlurWork blur{};        // plan-owned blur buffers and taps (blur_sigma > 0)

  // pruned iteration (prune.cu): set for the iteration being enqueued
  int2* prune_tiles = nullptr;          // (pattern tile, rotation tile) list, device
  int prune_n_tiles = 0;
  unsigned char* prune_state = nullptr; // [n_pt][n_rt] 0 skipped, 1 evaluated, 2 margin
  double* prune_margin = nullptr;       // [R] responsibility mass in margin tiles
  int* prune_kb_off = nullptr;          // [n_rt + 1] M-step k-blocks per rotation tile
  int* prune_kb_list = nullptr;         // the 64-pattern k-blocks themselves
  void* prune = nullptr;                // PruneState
  // L holds the normalised responsibilities P of the last iteration (true),
  // or still its log-likelihoods (false: mprep left P unwritten; it is formed
  // on request by plan_respons_ready)
  bool p_written = true;
  emc::IterReport* report = nullptr;  // page-locked host memory, written by the device

  // one captured iteration (emc_plan_capture / emc_plan_replay)
  bool graph_p_written = true;  // p_written after one of its replays
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t graph_exec = nullptr;

  // per-phase CUDA events on the context stream (emc_plan_set_profiling)
  static constexpr int kPhases = 6;  // expand, estep, lse, mprep, mstep, finish
  bool profiling = false;
  cudaEvent_t ev[kPhases + 1] = {};

  void* tc = nullptr;  // tensor-core state (tensor maps, rotation operands)
  int estep_gh_lo = -1;   // tensor E-step lo terms: bit 0 G, bit 1 H; -1 auto
  int mstep_q_lo = 0;     // tensor M-step: Q as FP16 hi + lo (1) or hi only (0)
  int estep_raster = 8;     // tensor E-step tile order (EMC_OPT_ESTEP_RASTER)
  int estep_pair = 1;       // full scans on CTA pairs (EMC_OPT_ESTEP_PAIR)
  int mstep_raster = -16;   // tensor M-step tile order (EMC_OPT_MSTEP_RASTER)
  int mstep_aggregate = 0;  // tensor M-step: warp-aggregated float atomics (nearest)
  unsigned debug_spin = 0;  // > 0: polls per tensor-pipeline wait (EMC_OPT_DEBUG_SPIN)
  int mstep_pair = 1;       // tensor M-step full scans on CTA pairs (EMC_OPT_MSTEP_PAIR)

  // sorted-voxel insertion (EMC_INSERT_SORTED, sorted_insert.cu): the M-step
  // stores each pair's value T_r x slice in ins_u [P_eff][ins_ldu] (rotation
  // fastest) and a segmented reduction in voxel order adds them
  float* ins_u = nullptr;
  int ins_ldu = 0;
  void* sorted = nullptr;

  std::vector<void*> allocs;
  size_t bytes = 0;
};

namespace emc {

// Voxel-sum upper bound and fixed-point scale slots in plan->red.
enum RedSlot {
  kRedMass = 1,      // captured responsibility mass
  kRedBad = 2,       // invalid pairs
  kRedBoundM = 3,    // upper bound of inserted model mass
  kRedBoundW = 4,    // upper bound of inserted weight
  kRedMean = 5,      // {sum, count} of positive voxels (2 slots) + partials
  kRedFixScale = 7,  // float2 {model, weight} fixed-point scales (deterministic mode)
  kRedSlots = 8,
};

// Deterministic insertion adds round(value * scale) into 64-bit integers.
// The scale is the power of two 2^(61 - k) with bound <= 2^k (the bound is an
// upper bound of the total inserted mass), so no partial sum leaves the signed
// 64-bit range, value * scale is exact in FP32, and 1 / scale is exact too.
__host__ __device__ inline float fix_scale_pow2(double bound) {
  if (!(bound > 0.0)) return 1.0f;
  int k;
  frexp(bound, &k);  // bound = f 2^k, f in [0.5, 1)
  const int e = 61 - k;
  return ldexpf(1.0f, e < -126 ? -126 : (e > 126 ? 126 : e));
}

#ifdef __CUDACC__
// x rounded to the nearest integer (ties to even) as a signed 64-bit value,
// with FP32 and integer instructions only: below 2^23 the addition of 2^23
// rounds the fraction away; from 2^23 on x is an integer, its mantissa shifted
// by the exponent.  |x| >= 2^62 (never reached under fix_scale_pow2) saturates.
__device__ __forceinline__ long long fixed_from_float(float x) {
  const float a = fabsf(x);
  long long m;
  if (a < 8388608.0f) {
    m = (long long)(__float_as_uint(__fadd_rn(a, 8388608.0f)) - 0x4B000000u);
  } else if (a < 4611686018427387904.0f) {
    const unsigned b = __float_as_uint(a);
    m = (long long)((b & 0x7FFFFFu) | 0x800000u) << ((int)(b >> 23) - 150);
  } else {
    m = 0x4000000000000000LL;
  }
  return x < 0.0f ? -m : m;
}
#endif

int plan_alloc(emc_plan* p, void** ptr, size_t bytes);

// Sorted-voxel insertion (sorted_insert.cu).  sorted_ensure (re)builds the
// voxel map when the plan's rotations or pixel coordinates differ from those
// it was built from (a bind, a change of the rotation order); sorted_reduce
// enqueues the per-iteration reduction of ins_u into acc2.
int sorted_ensure(emc_plan* p);
int sorted_reduce(emc_plan* p);
void sorted_free(emc_plan* p);

// Tensor-core path (tc_gemm.cu).
int tc_bind(emc_plan* p);
int prune_iterate(emc_plan* p, float* model, float* weight, float sigma, emc_iter_stats* stats,
                  bool* handled);
void prune_free(emc_plan* p);
int prune_reset(emc_plan* p);
int tc_pattern_side(emc_plan* p, const int* d_perm, bool counts_done = false);
int tc_ensure_qlo(emc_plan* p);
int tc_ensure_mslo(emc_plan* p);  // M'S lo, where EMC_OPT_ESTEP_GHLO asks for it
int tc_block_lists(emc_plan* p);  // count sums, lo_kb and block lists from the bound counts
__half* tc_tiny_plane(emc_plan* p);  // 1 where 0 < s < 1e-10 (blocks flagged tiny)
int pattern_side(emc_plan* p, const int* d_perm, bool with_tc);
constexpr float kPoisC = 0.02f;  // emc_cuda.cu:205

// Rotation-side FP16 operands of the tensor-core likelihood, written by the
// expand kernel straight from each slice value s (no FP32 slice buffer).
// Reference likelihood: M'S = [s >= 1e-10] s 2^-8, H = 1 / (s + 0.02) with 0
// where s <= 0 (their lo halves in MSl and Hl where those are read), I = [s <= 0] (bright counts:
// V = [s >= 1e-10] in its place), and the flags of the 64-pixel blocks that hold
// pixels with s <= 0 or an s in (0, 1e-10);
// true Poisson: log max(s, 1e-6) as hi + lo in Lh / Ll.  Blocks in which no pattern counts are not
// written (nothing reads them).  flags[0] |= 4 when M'S leaves the FP16 range.
struct RotOps {
  __half *MS = nullptr, *MSl = nullptr, *Hh = nullptr, *Hl = nullptr, *Iv = nullptr;
  __half *Lh = nullptr, *Ll = nullptr;
  int* flags = nullptr;
  const unsigned char* live = nullptr;  // [nkb] (null: no tensor path)
  bool bright = false;                  // V instead of I
  unsigned char *inv = nullptr, *tiny = nullptr;  // [n_rt][nkb]
  int nkb = 0;
  // device int: H lo is read (and written) only in the 64-pixel blocks below
  // it, the largest count-tail bound of the pattern tiles (null: every block)
  const int* hl_end = nullptr;
};

// The operands of four neighbouring pixels e .. e + 3 (e a multiple of 4) as
// 8-byte stores; hv = 1 / (s + 0.02) where s > 0, else 0, computed by the caller.
// BRIGHT: V in I's place; MS_LO: M'S lo too.
template <bool BRIGHT, bool MS_LO>
__device__ __forceinline__ void rot_ops_store4(const RotOps& o, size_t e, const float (&sv)[4],
                                               const float (&hv)[4], bool covered, bool live,
                                               bool h_lo) {
  union H4 {
    __half2 h[2];
    uint2 u;
  } ms4, hh4, iv4;
  float ms[4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
    ms[u] = covered || sv[u] >= 1e-10f ? sv[u] * (1.0f / 256.0f) : 0.0f;
  if (fmaxf(fmaxf(ms[0], ms[1]), fmaxf(ms[2], ms[3])) > 60000.0f) {
    atomicOr(o.flags, 4);
#pragma unroll
    for (int u = 0; u < 4; ++u)  // the operand stays finite: later models may skip this block
      ms[u] = ms[u] > 60000.0f ? 60000.0f : ms[u];
  }
  if (!live) return;
  ms4.h[0] = __floats2half2_rn(ms[0], ms[1]);
  ms4.h[1] = __floats2half2_rn(ms[2], ms[3]);
  hh4.h[0] = __floats2half2_rn(hv[0], hv[1]);
  hh4.h[1] = __floats2half2_rn(hv[2], hv[3]);
  iv4.h[0] = iv4.h[1] = __float2half2_rn(BRIGHT ? 1.0f : 0.0f);
  if (BRIGHT && !covered) {
    iv4.h[0] = __floats2half2_rn(sv[0] >= 1e-10f ? 1.0f : 0.0f, sv[1] >= 1e-10f ? 1.0f : 0.0f);
    iv4.h[1] = __floats2half2_rn(sv[2] >= 1e-10f ? 1.0f : 0.0f, sv[3] >= 1e-10f ? 1.0f : 0.0f);
  } else if (!covered) {
    iv4.h[0] = __floats2half2_rn(sv[0] > 0.0f ? 0.0f : 1.0f, sv[1] > 0.0f ? 0.0f : 1.0f);
    iv4.h[1] = __floats2half2_rn(sv[2] > 0.0f ? 0.0f : 1.0f, sv[3] > 0.0f ? 0.0f : 1.0f);
  }
  *reinterpret_cast<uint2*>(o.MS + e) = ms4.u;
  *reinterpret_cast<uint2*>(o.Hh + e) = hh4.u;
  *reinterpret_cast<uint2*>(o.Iv + e) = iv4.u;
  if (MS_LO) {
    H4 ml4;
    const float2 a = __half22float2(ms4.h[0]), b = __half22float2(ms4.h[1]);
    ml4.h[0] = __floats2half2_rn(ms[0] - a.x, ms[1] - a.y);
    ml4.h[1] = __floats2half2_rn(ms[2] - b.x, ms[3] - b.y);
    *reinterpret_cast<uint2*>(o.MSl + e) = ml4.u;
  }
  if (o.Hl && h_lo) {
    H4 hl4;
    const float2 a = __half22float2(hh4.h[0]), b = __half22float2(hh4.h[1]);
    hl4.h[0] = __floats2half2_rn(hv[0] - a.x, hv[1] - a.y);
    hl4.h[1] = __floats2half2_rn(hv[2] - b.x, hv[3] - b.y);
    *reinterpret_cast<uint2*>(o.Hl + e) = hl4.u;
  }
}

// The same for the true-Poisson likelihood: log max(s, floor) as FP16 hi + lo.
__device__ __forceinline__ void rot_ops_store_pois4(const RotOps& o, size_t e,
                                                    const float (&sv)[4]) {
  union H4 {
    __half2 h[2];
    uint2 u;
  } hi, lo;
  float l[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) l[u] = logf(fmaxf(sv[u], 1e-6f));
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    hi.h[v] = __floats2half2_rn(l[2 * v], l[2 * v + 1]);
    const float2 f = __half22float2(hi.h[v]);
    lo.h[v] = __floats2half2_rn(l[2 * v] - f.x, l[2 * v + 1] - f.y);
  }
  *reinterpret_cast<uint2*>(o.Lh + e) = hi.u;
  *reinterpret_cast<uint2*>(o.Ll + e) = lo.u;
}

// 1 / d for normal d whose reciprocal is normal too: the hardware reciprocal and one
// residual correction (Markstein 1990), at most the last bit off; a fifth of the
// instructions of the general division.
__device__ __forceinline__ float inverse(float d) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
  return __fmaf_rn(r, __fmaf_rn(-d, r, 1.0f), r);
}

RotOps tc_rot_ops(emc_plan* p);  // the plan's operand buffers (all null for FP32 plans)
int tc_estep(emc_plan* p);
int tc_autotune(emc_plan* p, int waves, int* best, float* best_ms);
int tc_estep_tiles(emc_plan* p);    // tiles of the full likelihood grid
int tc_time_estep(emc_plan* p, int raster, int first, int count, float* ms);
int tc_mstep(emc_plan* p, float* model, float* weight);
// What the host reads after an iteration, in host memory: four copies to pageable
// memory, each with a wait of its own, took 45 us of a 48^3 iteration's 200.
struct IterReport {
  double red[kRedSlots];
  double mass, margin;  // sums over the rotations
  double loglik;        // of the patterns' lse
  int flags[8];
  int status;  // of the tensor-core pipelines
};

int plan_wait(emc_plan* p, emc_iter_stats* stats, const double* margin, double* margin_sum);
int* tc_status(emc_plan* p);  // device status word of the tensor-core pipelines
void tc_free(emc_plan* p);
// Forms P = exp(L - lse) over L on the plan's stream when the last iteration
// left it unwritten (p_written false); no-op otherwise.
int plan_respons_ready(emc_plan* p);

}  // namespace emc
