// The fused EMC iteration (emc_plan_* / emc_iterate) and its FP32 kernels.
//
// One iteration restates main.cpp:239-480 for one process on one GPU:
//   expand        slice the model at every rotation, compacted to the
//                 P_eff pixels with mask != 0                       (A4)
//   scaling +     one tiled kernel per 128x128 (rotation, pattern) tile:
//   likelihood    pass 1 accumulates phi = sum k^2 / sum k s, pass 2 the
//                 per-pixel difference sum, the epilogue writes L and phi
//                 and a per-tile (max, sum exp) pair for every pattern (A5, A6)
//   normalise     FP64 log-sum-exp over the tile partials -> lse_i,
//                 P = exp(L - lse), Q = P / phi, T_r = sum_i P      (A7-A9)
//   M-step        tiled GEMM U = Q K over the compacted pixels; its epilogue
//                 inserts T_r * (U / T_r) into the model and T_r into the
//                 weight (nearest or trilinear; float or fixed-point
//                 atomics)                                           (A10, A11)
//   finish        divide by weight, normalise to mean 1 (FP64), blur (A13-A15)
// The MPI exchanges of the reference (main.cpp:367-392, 467-480) have no
// counterpart: the normaliser and the model sums are device reductions.
//
// Semantics of the fused path (the "intended" forms, stated because they
// differ from the drop-in kernels): the scaling denominator is a float sum
// (the reference truncates it to int), the per-pixel term is FP32, pairs with
// no overlap (count_r == 0) or undefined scaling (num or den <= 0) get
// L = -inf and phi = 1, a pattern whose pairs are all invalid gets zero
// responsibility, and the normaliser is FP64.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include "geometry.cuh"
#include "kernels.cuh"
#include "plan.cuh"
#include "ptx.cuh"

namespace emc {

int plan_alloc(emc_plan* p, void** ptr, size_t bytes) {
  if (bytes == 0) bytes = 256;
  cudaError_t e = cudaMalloc(ptr, bytes);
  if (e != cudaSuccess)
    return fail(p->ctx, EMC_ERR_NOMEM, "plan alloc of %zu bytes: %s", bytes, cudaGetErrorString(e));
  p->allocs.push_back(*ptr);
  p->bytes += bytes;
  return EMC_OK;
}

template <typename T>
static int alloc_n(emc_plan* p, T** ptr, size_t n) {
  return plan_alloc(p, (void**)ptr, n * sizeof(T));
}

// ------------------------------------------------------------- bind ------
// fp16(k) times a power of two: exact (k's FP16 form has 11 significant bits,
// and the scale keeps its last one at 2^-17 or above).
__device__ __forceinline__ __half scaled_count(float k, float scale) {
  return __float2half_rn(__half2float(__float2half_rn(k)) * scale);
}

__global__ void gather_coords_kernel(const int* __restrict__ pix, const float* __restrict__ x,
                                     const float* __restrict__ y, const float* __restrict__ z,
                                     float* cx, float* cy, float* cz, int Kp) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= Kp) return;
  const int p = pix[q];
  cx[q] = p >= 0 ? x[p] : 0.0f;
  cy[q] = p >= 0 ? y[p] : 0.0f;
  cz[q] = p >= 0 ? z[p] : 0.0f;
}

// Per-pattern factor of the reference's image normalisation
// (emc_helper.cpp:389-418): c_i = N_2d / (float sum over mask == 1 pixels).
// Pattern position i of the plan holds input pattern perm[i] (perm == nullptr:
// the identity) in this and the other pattern-side kernels.
__global__ void pattern_norm_kernel(const float* __restrict__ images, const int* __restrict__ mask,
                                    int n2, int N, int normalize, float* __restrict__ cnorm,
                                    const int* __restrict__ perm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  float c = 1.0f;
  if (normalize) {
    const float* img = images + (size_t)(perm ? perm[i] : i) * n2;
    float s = 0.0f;
    for (int p = 0; p < n2; ++p)
      if (__ldg(mask + p) == 1) s = __fadd_rn(s, __ldg(img + p));
    c = __fdiv_rn((float)n2, s);
  }
  cnorm[i] = c;
}

// Compacted pattern operands.  flags[0] bit 0: non-finite input; bit 1: a
// count that is not an integer in [0, 65504] (no FP16 form); bit 3: an
// integer count above 2048 (FP16 rounds it); flags[8]: the largest integer
// count.  One block per (pattern, 256 compacted pixels), pixel blocks the
// fast index so that a pattern's row stays in L2 while its blocks run; flags
// and part[i][block] (the block's sum of k, FP64, fixed order) reduced by
// warp shuffles and one barrier.  Kraw / Kt (FP32 path) may be null;
// with Kh non-null the kernel also writes the tensor path's FP16 counts
// (the same values as tc_pattern_ops_kernel with the same scale).
__global__ void pattern_ops_kernel(const float* __restrict__ images, const int* __restrict__ pix,
                                   const float* __restrict__ cnorm, int n2, int N, int Kp,
                                   float* __restrict__ Kraw, float* __restrict__ Kt,
                                   int* __restrict__ flags,
                                   const int* __restrict__ perm, double* __restrict__ part,
                                   __half* __restrict__ Kh, float count_scale) {
  const int nqb = (Kp + 255) / 256;
  const int i = (int)(blockIdx.x / nqb);
  const int q = (int)(blockIdx.x % nqb) * 256 + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool in = q < Kp;
  const int p = in ? pix[q] : -1;
  float v = 0.0f, k = 0.0f;
  int bits = 0, vmax = 0;
  if (p >= 0) {
    v = __ldg(images + (size_t)(perm ? perm[i] : i) * n2 + p);
    if (!isfinite(v)) bits |= 1;
    if (!(v >= 0.0f && v <= 65504.0f && v == rintf(v))) {
      bits |= 2;
    } else {
      if (v > 2048.0f) bits |= 8;
      vmax = (int)v;
    }
    k = __fmul_rn(v, __ldg(cnorm + i));
  }
  // FP32 warp tree (exact for integer counts; FP64 throughput is scarce), FP64 after
  float fsum = k;
  for (int o = 16; o > 0; o >>= 1) fsum += __shfl_down_sync(0xffffffffu, fsum, o);
  const double sum = (double)fsum;
  bits = __reduce_or_sync(0xffffffffu, (unsigned)bits);
  vmax = __reduce_max_sync(0xffffffffu, vmax);
  __shared__ double wsum[8];
  __shared__ int wbits[8], wmax[8];
  if (lane == 0) {
    wsum[warp] = sum;
    wbits[warp] = bits;
    wmax[warp] = vmax;
  }
  if (in) {
    const size_t o = (size_t)i * Kp + q;
    if (Kraw) Kraw[o] = k;
    const float kt = k >= 1e-10f ? k : 0.0f;  // the reference's (double)k > 1e-10
    if (Kt) Kt[o] = kt;
    if (Kh) Kh[o] = scaled_count(v, count_scale);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    int b = 0, m = 0;
    for (int j = 0; j < 8; ++j) {
      t += wsum[j];
      b |= wbits[j];
      m = max(m, wmax[j]);
    }
    part[blockIdx.x] = t;
    if (b) atomicOr(flags, b);
    // the maximum settles early: skip the atomic when this block cannot raise it
    if (m > flags[8]) atomicMax(flags + 8, m);
  }
}

// The same operands, sums and flags as pattern_ops_kernel with one block per
// pattern: the pattern's row is first staged in shared memory with coalesced
// 16-byte loads, then the compacted values are gathered from there in the
// pixel list's (radius) order -- the list scatters over the whole row, and
// gathering it from global memory, one load per thread in flight, took 3.5 ms
// of a 4.2 ms bind at 128^3 x 20,000 patterns.  For rows that fit shared
// memory (pattern_row_smem <= kRowSmemMax).  Ksum[i] is written directly: a
// warp-shuffle tree per 64 pixels in FP32 (exact for integer counts, whose
// sums stay below 2^24; FP64 arithmetic runs at a small fraction of the FP32
// rate on this GPU, and an FP64 tree per pixel took as long as the rest of
// the bind), then the warp sums in pixel order in FP64.
constexpr int kRowThreads = 512;
constexpr int kRowSmemMax = 200 * 1024;

// the row, then the warps' FP64 sums (8-byte aligned: n2 may be odd)
__host__ __device__ inline size_t pattern_row_bytes(int n2) {
  return ((size_t)n2 + (n2 & 1)) * sizeof(float);
}
__host__ __device__ inline size_t pattern_row_smem(int n2, int Kp) {
  return pattern_row_bytes(n2) + (size_t)((Kp + 255) / 256) * 8 * sizeof(double);
}

__global__ void __launch_bounds__(kRowThreads) pattern_row_kernel(
    const float* __restrict__ images, const int* __restrict__ pix, const float* __restrict__ cnorm,
    int n2, int N, int Kp, float* __restrict__ Kraw, float* __restrict__ Kt,
    int* __restrict__ flags, const int* __restrict__ perm,
    float* __restrict__ Ksum, __half* __restrict__ Kh, float count_scale) {
  extern __shared__ __align__(16) unsigned char row_smem[];
  float* srow = reinterpret_cast<float*>(row_smem);
  double* wsum = reinterpret_cast<double*>(row_smem + pattern_row_bytes(n2));
  const int i = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* img = images + (size_t)(perm ? perm[i] : i) * n2;
  if ((n2 & 3) == 0 && ((uintptr_t)img & 15) == 0) {
    const float4* s4 = reinterpret_cast<const float4*>(img);
    float4* d4 = reinterpret_cast<float4*>(srow);
    for (int j = threadIdx.x; j < n2 / 4; j += blockDim.x) d4[j] = __ldg(s4 + j);
  } else {
    for (int j = threadIdx.x; j < n2; j += blockDim.x) srow[j] = __ldg(img + j);
  }
  __syncthreads();
  const float ci = __ldg(cnorm + i);
  int bits = 0, vmax = 0;
  // two neighbouring pixels per thread (Kp is a multiple of 128): the
  // compacted operands go out as 8-byte (float2) and 4-byte (half2) stores
  for (int q = 2 * threadIdx.x; q < Kp; q += 2 * blockDim.x) {
    const int2 pp = __ldg(reinterpret_cast<const int2*>(pix + q));
    const int pv[2] = {pp.x, pp.y};
    float v[2], k[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      v[u] = 0.0f;
      k[u] = 0.0f;
      if (pv[u] >= 0) {
        v[u] = srow[pv[u]];
        if (!isfinite(v[u])) bits |= 1;
        if (!(v[u] >= 0.0f && v[u] <= 65504.0f && v[u] == rintf(v[u]))) {
          bits |= 2;
        } else {
          if (v[u] > 2048.0f) bits |= 8;
          vmax = max(vmax, (int)v[u]);
        }
        k[u] = __fmul_rn(v[u], ci);
      }
    }
    float sum = k[0] + k[1];
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if (lane == 0) wsum[(q - 2 * lane) / 64] = (double)sum;
    const size_t o = (size_t)i * Kp + q;
    if (Kraw) *reinterpret_cast<float2*>(Kraw + o) = make_float2(k[0], k[1]);
    const float kt0 = k[0] >= 1e-10f ? k[0] : 0.0f;  // the reference's (double)k > 1e-10
    const float kt1 = k[1] >= 1e-10f ? k[1] : 0.0f;
    if (Kt) *reinterpret_cast<float2*>(Kt + o) = make_float2(kt0, kt1);
    if (Kh)
      *reinterpret_cast<__half2*>(Kh + o) =
          __halves2half2(scaled_count(v[0], count_scale), scaled_count(v[1], count_scale));
  }
  bits = (int)__reduce_or_sync(0xffffffffu, (unsigned)bits);
  vmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)vmax);
  __shared__ int sbits[kRowThreads / 32], smax[kRowThreads / 32];
  if (lane == 0) {
    sbits[warp] = bits;
    smax[warp] = vmax;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < Kp / 64; ++w) s += wsum[w];
    Ksum[i] = (float)s;
    int bb = 0, m = 0;
    for (int w = 0; w < (int)(blockDim.x / 32); ++w) {
      bb |= sbits[w];
      m = max(m, smax[w]);
    }
    if (bb) atomicOr(flags, bb);
    if (m > flags[8]) atomicMax(flags + 8, m);
  }
}

// Ksum[i] = the sum of pattern i's block partials (in block order).
__global__ void pattern_sums_kernel(const double* __restrict__ part, int N, int nqb,
                                    float* __restrict__ Ksum) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double s = 0.0;
  for (int b = 0; b < nqb; ++b) s += part[(size_t)i * nqb + b];
  Ksum[i] = (float)s;
}

// ------------------------------------------------------------ expand -----
constexpr float kSliceFloor = 1e-6f;  // true-Poisson floor for unknown voxels

// Index arithmetic of the samples without conversion instructions (roundf, floorf
// and the casts run at an eighth of the rate of an addition): adding 2^23 (rounding
// down for the trilinear cell: 1.5 x 2^23) leaves the integer in the low bits.

// The voxel voxel_round(v) where that is 1 .. n, else 0: v + 1/2 rounded towards
// zero does not reach the next integer, and truncates to it.  Values outside, and
// NaN, give bits outside the range.
__device__ __forceinline__ unsigned slice_voxel(float v, unsigned n) {
  const unsigned i =
      __float_as_uint(__fadd_rz(__fadd_rz(v, 0.5f), 8388608.0f)) - 0x4B000000u;
  return i - 1u < n ? i : 0u;
}

template <int INTERP>
__device__ __forceinline__ float plan_sample(const float* __restrict__ model, int side,
                                             const RotMat& R, float x, float y, float z);

template <>
__device__ __forceinline__ float plan_sample<EMC_INTERP_NEAREST>(const float* __restrict__ model,
                                                                  int side, const RotMat& R,
                                                                  float x, float y, float z) {
  const unsigned n = (unsigned)side - 1;  // 1 .. side - 1: the reference's bounds
  const unsigned ix = slice_voxel(voxel_coord(side, rotate_row(R, 0, x, y, z)), n);
  const unsigned iy = slice_voxel(voxel_coord(side, rotate_row(R, 1, x, y, z)), n);
  const unsigned iz = slice_voxel(voxel_coord(side, rotate_row(R, 2, x, y, z)), n);
  if (ix && iy && iz) return __ldg(model + ((iz * side + iy) * side + ix));
  return -1.0f;
}

template <>
__device__ __forceinline__ float plan_sample<EMC_INTERP_TRILINEAR>(const float* __restrict__ model,
                                                                    int side, const RotMat& R,
                                                                    float x, float y, float z) {
  constexpr float kMagic = 12582912.0f;  // 1.5 x 2^23
  const float c[3] = {voxel_coord(side, rotate_row(R, 0, x, y, z)),
                      voxel_coord(side, rotate_row(R, 1, x, y, z)),
                      voxel_coord(side, rotate_row(R, 2, x, y, z))};
  int i0[3];
  float f1[3], f0[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float t = __fadd_rd(c[d], kMagic);
    // a coordinate this far out (or NaN) meets no voxel: neither 2^30 nor 2^30 + 1 does
    const bool near = fabsf(c[d]) < 4194304.0f;
    i0[d] = near ? __float_as_int(t) - __float_as_int(kMagic) : 1 << 30;
    f1[d] = c[d] - (t - kMagic);
    f0[d] = 1.0f - f1[d];
  }
  const unsigned n = (unsigned)side;
  const float xy[4] = {f0[0] * f0[1], f1[0] * f0[1], f0[0] * f1[1], f1[0] * f1[1]};
  float acc = 0.0f, wsum = 0.0f;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const unsigned xi = (unsigned)(i0[0] + (e & 1)), yi = (unsigned)(i0[1] + ((e >> 1) & 1)),
                   zi = (unsigned)(i0[2] + (e >> 2));
    if (xi >= n || yi >= n || zi >= n) continue;
    const float w = xy[e & 3] * ((e >> 2) ? f1[2] : f0[2]);
    const float v = __ldg(model + ((zi * n + yi) * n + xi));
    if (v < 0.0f || w <= 0.0f) continue;
    acc = __fmaf_rn(w, v, acc);
    wsum += w;
  }
  return wsum > 1e-6f ? acc / wsum : -1.0f;
}

// The compacted slice rows S[r][0..Kp) (or their FP16 operands) of
// kSliceRows rotations per block and the per-rotation sums: count_r (s > 0) and
// A_r = sum s^2/(s+c) of the reference likelihood, the floored slice sum of the
// true-Poisson one.  Bound by issue while the model fits near L1 -- with all three
// sums and a division in either case, conversions in the index and every test on every
// pixel a sample took up to 110 instructions: 64^3, 6,300 rotations 56 us, now 42;
// 112^3, 10,860, true Poisson 378, now 302; 96^3 trilinear 1,217, now 1,067 -- and by
// the latency of the gathers in an 8 MB model (128^3, 25,680: 1,116 and 1,113, true
// Poisson 1,078 and 985; two rotations per block with more blocks spill: 1,676).
enum SliceMode {
  kSliceFp32,
  kSliceTcPois,
  kSliceTc,  // and with bright counts, or with M'S lo, or both:
  kSliceTcBright,
  kSliceTcLo,
  kSliceTcBrightLo
};

// rotations per expand block: four with nearest sampling, two with the
// eight-voxel trilinear gather (registers)
template <int INTERP>
__host__ __device__ constexpr int slice_rows_per_block() { return INTERP == EMC_INTERP_NEAREST ? 4 : 2; }

template <int INTERP, int MODE>
__global__ void __launch_bounds__(256) slice_rows_kernel(
    const float* __restrict__ model, int side, const float* __restrict__ rot,
    const int* __restrict__ pix, const float* __restrict__ cx, const float* __restrict__ cy,
    const float* __restrict__ cz, int R, int Kp, float* __restrict__ S,
    float* __restrict__ rot_cnt, float* __restrict__ rot_A, float* __restrict__ rot_ssum,
    RotOps ops) {
  // kSliceRows rotations per block: each thread loads the coordinates of four
  // neighbouring compacted pixels once (16-byte loads) and samples them for
  // every rotation of the block, so coordinate traffic is shared and the
  // model gathers of several rotations are in flight together; the operands
  // go out as 8-byte stores (Kp is a multiple of 128)
  constexpr int kSliceRows = slice_rows_per_block<INTERP>();
  constexpr bool kTc = MODE >= kSliceTc;
  constexpr bool kBright = MODE == kSliceTcBright || MODE == kSliceTcBrightLo;
  constexpr bool kMsLo = MODE == kSliceTcLo || MODE == kSliceTcBrightLo;
  const int r0 = blockIdx.x * kSliceRows;
  const int hl_end = ops.hl_end ? 64 * __ldg(ops.hl_end) : Kp;  // H lo pixels
  const int nr = min(kSliceRows, R - r0);
  __shared__ RotMat sR[kSliceRows];
  if (threadIdx.x < nr) sR[threadIdx.x] = quat_to_matrix(rot + 4 * (size_t)(r0 + threadIdx.x));
  __syncthreads();
  // per-thread FP32 partials (FP64 arithmetic is scarce on this GPU), block sums in FP64
  float cnt[kSliceRows], A[kSliceRows], ss[kSliceRows];
#pragma unroll
  for (int k = 0; k < kSliceRows; ++k) cnt[k] = A[k] = ss[k] = 0.0f;
  for (int q = 4 * threadIdx.x; q < Kp; q += 4 * blockDim.x) {
    const int4 pp = __ldg(reinterpret_cast<const int4*>(pix + q));
    const float4 X = __ldg(reinterpret_cast<const float4*>(cx + q));
    const float4 Y = __ldg(reinterpret_cast<const float4*>(cy + q));
    const float4 Z = __ldg(reinterpret_cast<const float4*>(cz + q));
    const int pv[4] = {pp.x, pp.y, pp.z, pp.w};
    const float xv[4] = {X.x, X.y, X.z, X.w}, yv[4] = {Y.x, Y.y, Y.z, Y.w},
                zv[4] = {Z.x, Z.y, Z.z, Z.w};
    const bool pixels = (pp.x | pp.y | pp.z | pp.w) >= 0;  // none is padding
    const bool live = MODE != kSliceFp32 && __ldg(ops.live + (q >> 6)) != 0;
    int odd = 0;  // bit 0: an s <= 0, bit 1: one in (0, 1e-10)
#pragma unroll
    for (int k = 0; k < kSliceRows; ++k) {
      if (k >= nr) break;  // uniform over the block
      const RotMat Rm = sR[k];
      float sv[4], hv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        sv[u] = pixels || pv[u] >= 0 ? plan_sample<INTERP>(model, side, Rm, xv[u], yv[u], zv[u])
                                     : 0.0f;
      const size_t e = (size_t)(r0 + k) * Kp + q;
      if (!kTc) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (pixels || pv[u] >= 0) ss[k] += fmaxf(sv[u], kSliceFloor);
      }
      if (MODE == kSliceTcPois) {
        if (live) rot_ops_store_pois4(ops, e, sv);
        continue;
      }
      // each value for itself: a minimum would pass over a NaN, which is not covered
      const bool covered = pixels && sv[0] >= 1e-10f && sv[1] >= 1e-10f && sv[2] >= 1e-10f &&
                           sv[3] >= 1e-10f;
      if (covered) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          hv[u] = inverse(sv[u] + kPoisC);  // serves A = s^2 h and the operands
          A[k] = __fmaf_rn(sv[u] * sv[u], hv[u], A[k]);
        }
        cnt[k] += 4.0f;
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          hv[u] = sv[u] > 0.0f ? inverse(sv[u] + kPoisC) : 0.0f;
          if (pv[u] >= 0) {
            if (!(sv[u] >= 1e-10f)) odd |= sv[u] > 0.0f ? 2 : 1;
            if (sv[u] > 0.0f) {
              cnt[k] += 1.0f;
              A[k] = __fmaf_rn(sv[u] * sv[u], hv[u], A[k]);
            }
          }
        }
      }
      // the tensor path takes its FP16 operands straight from s; the FP32
      // path keeps the slices
      if (kTc)
        rot_ops_store4<kBright, kMsLo>(ops, e, sv, hv, covered, live, q < hl_end);
      else
        *reinterpret_cast<float4*>(S + e) = make_float4(sv[0], sv[1], sv[2], sv[3]);
    }
    if (kTc && odd) {  // races store the same value
      const size_t f = (size_t)(r0 >> 7) * ops.nkb + (q >> 6);
      if (odd & 1) ops.inv[f] = 1;
      if (odd & 2) ops.tiny[f] = 1;
    }
  }
  // per row: FP32 warp sums, then FP64 over the warps
  __shared__ double wsum[3][kSliceRows][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < kSliceRows; ++k) {
    float a = cnt[k], b = A[k], c = ss[k];
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, o);
      b += __shfl_down_sync(0xffffffffu, b, o);
      c += __shfl_down_sync(0xffffffffu, c, o);
    }
    if (lane == 0) {
      wsum[0][k][warp] = (double)a;
      wsum[1][k][warp] = (double)b;
      wsum[2][k][warp] = (double)c;
    }
  }
  __syncthreads();
  if (threadIdx.x < nr) {
    const int k = threadIdx.x;
    double a = 0.0, b = 0.0, c = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      a += wsum[0][k][w];
      b += wsum[1][k][w];
      c += wsum[2][k][w];
    }
    rot_cnt[r0 + k] = (float)a;
    rot_A[r0 + k] = (float)b;
    rot_ssum[r0 + k] = (float)c;
  }
}

// The plane T = [0 < s < 1e-10] of the likelihood's rotation operands, in
// the (rotation tile, 64-pixel block) pairs that hold such a value -- none in
// most iterations: a rotation tile's eight blocks look at their flags and exit.
// (With sharp atoms and trilinear slices most blocks hold one: 219 us at 96^3 and
// 10,860 rotations with one block per rotation tile, 82 with eight.)
constexpr int kTinyBlocks = 8;
template <int INTERP>
__global__ void __launch_bounds__(256) tiny_plane_kernel(
    const float* __restrict__ model, int side, const float* __restrict__ rot,
    const int* __restrict__ pix, const float* __restrict__ cx, const float* __restrict__ cy,
    const float* __restrict__ cz, int R, int Kp, const unsigned char* __restrict__ tiny, int nkb,
    __half* __restrict__ T) {
  const int rt = blockIdx.x;
  for (int kb = blockIdx.y; kb < nkb; kb += kTinyBlocks) {
    if (!__ldg(tiny + (size_t)rt * nkb + kb)) continue;  // uniform over the block
    for (int e = threadIdx.x; e < 128 * 64; e += blockDim.x) {
      const int r = rt * 128 + (e >> 6), q = kb * 64 + (e & 63);
      if (r >= R) break;
      const int pv = pix[q];
      float s = 0.0f;
      if (pv >= 0) {
        const RotMat Rm = quat_to_matrix(rot + 4 * (size_t)r);
        s = plan_sample<INTERP>(model, side, Rm, cx[q], cy[q], cz[q]);
      }
      T[(size_t)r * Kp + q] = __float2half_rn(s > 0.0f && s < 1e-10f ? 1.0f : 0.0f);
    }
  }
}

// --------------------------------------------------- FP32 E-step tile ----
// The FP32 contractions: 128 x 128 tiles, 16 steps of the reduction per stage and
// two stages (one barrier each), 8 x 8 results per thread as packed pairs along
// the second operand.  Bound by the FP32 pipe: with scalar
// multiply-adds, two barriers per stage and the coverage as an operand of its own,
// 3,240 rotations x 2,000 patterns at 64^3 took 5,451 us (E-step) and 1,214 (M-step),
// now 4,122 and 1,086.
constexpr int BM = 128, BN = 128, BK = 16, TPB = 256, STG = BK * BM;

using ptx::f32x2;

// Loads a [128 rows][16 cols] tile of a row-major matrix (leading dim ld,
// ld % 4 == 0) into two float4 per thread; rows >= nrows read as zero.
__device__ __forceinline__ void ld_tile(const float* __restrict__ src, size_t ld, int row0,
                                        int nrows, int k0, float4 (&v)[2]) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int f = threadIdx.x + u * TPB;
    const int row = f >> 2, quad = f & 3;
    v[u] = row0 + row < nrows
               ? __ldg(reinterpret_cast<const float4*>(src + (size_t)(row0 + row) * ld + k0) + quad)
               : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// Transposed store of a loaded tile: dst[k][row] = op(v), the row with bits 3 and 4
// flipped by k / 4: a warp's stores (8 rows x 4 quads) meet all banks.
template <typename Op>
__device__ __forceinline__ void st_tile_t(float* dst, const float4 (&v)[2], Op op) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int f = threadIdx.x + u * TPB;
    const int quad = f & 3, at = quad * 4 * BM + ((f >> 2) ^ (quad << 3));
    dst[at] = op(v[u].x);
    dst[at + BM] = op(v[u].y);
    dst[at + 2 * BM] = op(v[u].z);
    dst[at + 3 * BM] = op(v[u].w);
  }
}

// Eight values of row k of such a tile (base: a multiple of 4), as four pairs, or
// each twice in a pair.
__device__ __forceinline__ void ld_pairs(const float* s, int k, int base, f32x2 (&o)[4]) {
  const float* row = s + k * BM + (base ^ ((k >> 2) << 3));
  const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(row);
  const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(row + 64);
  o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}
__device__ __forceinline__ void ld_twice(const float* s, int k, int base, f32x2 (&o)[8]) {
  const float* row = s + k * BM + (base ^ ((k >> 2) << 3));
  const float4 a = *reinterpret_cast<const float4*>(row);
  const float4 b = *reinterpret_cast<const float4*>(row + 64);
  o[0] = ptx::pack2(a.x, a.x); o[1] = ptx::pack2(a.y, a.y);
  o[2] = ptx::pack2(a.z, a.z); o[3] = ptx::pack2(a.w, a.w);
  o[4] = ptx::pack2(b.x, b.x); o[5] = ptx::pack2(b.y, b.y);
  o[6] = ptx::pack2(b.z, b.z); o[7] = ptx::pack2(b.w, b.w);
}

__device__ __forceinline__ int micro_idx(int t4, int i) { return (i < 4 ? 0 : 64) + t4 + (i & 3); }

struct EstepArgs {
  const float* S;      // [Rp][Kp]
  const float* Kraw;   // [N][Kp]
  const float* Kt;
  const float* Ksum;   // [N]
  const float* rot_cnt;
  const float* rot_ssum;
  const float* rotw;   // [R]
  float* L;            // [R][N]
  float* PHI;          // [R][N]
  float2* part;        // [n_rt][N]
  int* bad;            // invalid pair counter
  int R, N, Kp;
  const float* sigma;  // [1] annealing width (device memory)
  int known_intensity;
};

// out[r][n] of the micro-tile.
__device__ __forceinline__ void store_tile(const EstepArgs& a, float* __restrict__ out,
                                           const float (&v)[8][8]) {
  const int ty4 = (threadIdx.x >> 4) * 4, tx4 = (threadIdx.x & 15) * 4;
  const int r0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = r0 + micro_idx(ty4, i);
    if (r >= a.R) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int n = n0 + h * 64 + tx4;
      float* p = out + (size_t)r * a.N + n;
      if (n + 3 < a.N && ((a.N & 3) == 0)) {
        *reinterpret_cast<float4*>(p) =
            make_float4(v[i][4 * h], v[i][4 * h + 1], v[i][4 * h + 2], v[i][4 * h + 3]);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (n + c < a.N) p[c] = v[i][4 * h + c];
      }
    }
  }
}

// Writes L of the micro-tile and the tile's (max, sum exp) per pattern.
__device__ void estep_epilogue(const EstepArgs& a, float (&Lv)[8][8],
                               float* sred /* [16][128] */, float* scol /* [128] */) {
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  const int n0 = blockIdx.x * BN, tx4 = tx * 4;
  store_tile(a, a.L, Lv);
  // per-pattern max over the tile's rotations
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float m = -INFINITY;
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, Lv[i][j]);
    sred[ty * BN + micro_idx(tx4, j)] = m;
  }
  __syncthreads();
  if (threadIdx.x < BN) {
    float m = -INFINITY;
    for (int t = 0; t < 16; ++t) m = fmaxf(m, sred[t * BN + threadIdx.x]);
    scol[threadIdx.x] = m;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float m = scol[micro_idx(tx4, j)];
    float s = 0.0f;
    if (m > -INFINITY) {
#pragma unroll
      for (int i = 0; i < 8; ++i) s += expf(Lv[i][j] - m);
    }
    sred[ty * BN + micro_idx(tx4, j)] = s;
  }
  __syncthreads();
  if (threadIdx.x < BN) {
    const int n = n0 + threadIdx.x;
    float s = 0.0f;
    for (int t = 0; t < 16; ++t) s += sred[t * BN + threadIdx.x];
    if (n < a.N) a.part[(size_t)blockIdx.y * a.N + n] = make_float2(scol[threadIdx.x], s);
  }
}

// Reference-"poisson" likelihood with per-pair scaling, two pixel passes: 1 + 3
// multiply-adds per (rotation, pattern, pixel) where a tile's rotations cover all
// 16 pixels of a stage (s >= 1e-10), 2 + 3 elsewhere.
__global__ void __launch_bounds__(TPB, 1) estep_fp32_kernel(EstepArgs a) {
  __shared__ __align__(16) float sS[2][STG], sG[2][STG], sK[2][STG];
  const int ty4 = (threadIdx.x >> 4) * 4, tx4 = (threadIdx.x & 15) * 4;
  const int r0 = blockIdx.y * BM, n0 = blockIdx.x * BN;

  f32x2 iphi[8][4];
  float4 vr[2], vk[2];
  const int nk = a.Kp / BK;
  int nbad = 0;
  if (!a.known_intensity) {
    // ---- pass 1: num = sum Kt^2 [s >= 1e-10], den = sum Kt s [s >= 1e-10]
    // (s >= 1e-10f is the reference's (double)s > 1e-10 for every float s)
    f32x2 num[8][4], den[8][4], all[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) num[i][j] = den[i][j] = 0;
    ld_tile(a.S, a.Kp, r0, a.R, 0, vr);
    ld_tile(a.Kt, a.Kp, n0, a.N, 0, vk);
    for (int kb = 0; kb < nk; ++kb) {
      float *s = sS[kb & 1], *t = sK[kb & 1];
      int out = 0;  // a rotation of the tile with a pixel outside
      st_tile_t(s, vr, [&](float v) {
        const bool in = v >= 1e-10f;
        out |= !in;
        return in ? v : 0.0f;
      });
      st_tile_t(t, vk, [](float v) { return v; });
      if (__syncthreads_or(out) == 0) {
        if (kb + 1 < nk) {
          ld_tile(a.S, a.Kp, r0, a.R, (kb + 1) * BK, vr);
          ld_tile(a.Kt, a.Kp, n0, a.N, (kb + 1) * BK, vk);
        }
#pragma unroll 8
        for (int k = 0; k < BK; ++k) {
          f32x2 rs[8], pk[4];
          ld_twice(s, k, ty4, rs);
          ld_pairs(t, k, tx4, pk);
#pragma unroll
          for (int j = 0; j < 4; ++j) all[j] = ptx::add2(all[j], ptx::mul2(pk[j], pk[j]));
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) den[i][j] = ptx::fma2(pk[j], rs[i], den[i][j]);
        }
      } else {
        if (kb + 1 < nk) {
          ld_tile(a.S, a.Kp, r0, a.R, (kb + 1) * BK, vr);
          ld_tile(a.Kt, a.Kp, n0, a.N, (kb + 1) * BK, vk);
        }
#pragma unroll 4
        for (int k = 0; k < BK; ++k) {
          f32x2 rs[8], pk[4], p2[4];
          ld_twice(s, k, ty4, rs);
          ld_pairs(t, k, tx4, pk);
#pragma unroll
          for (int j = 0; j < 4; ++j) p2[j] = ptx::mul2(pk[j], pk[j]);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float m = ptx::unpack2(rs[i]).x > 0.0f ? 1.0f : 0.0f;
            const f32x2 mm = ptx::pack2(m, m);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              num[i][j] = ptx::fma2(p2[j], mm, num[i][j]);
              den[i][j] = ptx::fma2(pk[j], rs[i], den[i][j]);
            }
          }
        }
      }
    }
    float phi[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 u = ptx::unpack2(ptx::add2(num[i][j], all[j]));
        const float2 d = ptx::unpack2(den[i][j]);
        // phi = 1 where undefined; 1/phi = -1 marks it
        const bool ox = u.x > 0.0f && d.x > 0.0f, oy = u.y > 0.0f && d.y > 0.0f;
        phi[i][2 * j] = ox ? __fdiv_rn(u.x, d.x) : 1.0f;
        phi[i][2 * j + 1] = oy ? __fdiv_rn(u.y, d.y) : 1.0f;
        iphi[i][j] = ptx::pack2(ox ? __fdiv_rn(d.x, u.x) : -1.0f, oy ? __fdiv_rn(d.y, u.y) : -1.0f);
      }
    store_tile(a, a.PHI, phi);
    __syncthreads();  // the last stage has been read
  } else {
    float phi[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        phi[i][j] = 1.0f;
        iphi[i][j >> 1] = ptx::pack2(1.0f, 1.0f);
      }
    store_tile(a, a.PHI, phi);
  }
  // ---- pass 2: acc = sum (s - k/phi)^2 / (s + c) over s > 0
  f32x2 acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
  ld_tile(a.S, a.Kp, r0, a.R, 0, vr);
  ld_tile(a.Kraw, a.Kp, n0, a.N, 0, vk);
  for (int kb = 0; kb < nk; ++kb) {
    float *s = sS[kb & 1], *g = sG[kb & 1], *t = sK[kb & 1];
    st_tile_t(s, vr, [](float v) { return v; });
    st_tile_t(g, vr, [](float v) { return v > 0.0f ? __frcp_rn(v + kPoisC) : 0.0f; });
    st_tile_t(t, vk, [](float v) { return -v; });
    __syncthreads();
    if (kb + 1 < nk) {
      ld_tile(a.S, a.Kp, r0, a.R, (kb + 1) * BK, vr);
      ld_tile(a.Kraw, a.Kp, n0, a.N, (kb + 1) * BK, vk);
    }
#pragma unroll 4
    for (int k = 0; k < BK; ++k) {
      f32x2 rs[8], rg[8], pk[4];
      ld_twice(s, k, ty4, rs);
      ld_twice(g, k, ty4, rg);
      ld_pairs(t, k, tx4, pk);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const f32x2 d = ptx::fma2(pk[j], iphi[i][j], rs[i]);
          acc[i][j] = ptx::fma2(ptx::mul2(d, rg[i]), d, acc[i][j]);
        }
    }
  }
  __syncthreads();  // sS and sK are free
  // ---- epilogue
  float Lv[8][8];
  const float sg = *a.sigma;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = r0 + micro_idx(ty4, i);
    const bool rok = r < a.R;
    const float cnt = rok ? __ldg(a.rot_cnt + r) : 0.0f;
    const float lw = rok ? logf(__ldg(a.rotw + r)) : 0.0f;
    const float scale = cnt > 0.0f ? (1.0f / (2.0f * sg * sg)) / cnt : 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float2 e = ptx::unpack2(acc[i][j >> 1]), f = ptx::unpack2(iphi[i][j >> 1]);
      const int n = n0 + micro_idx(tx4, j);
      const bool ok = rok && n < a.N && cnt > 0.0f && ((j & 1) ? f.y : f.x) > 0.0f;
      if (rok && n < a.N && !ok) nbad++;
      Lv[i][j] = ok ? lw - ((j & 1) ? e.y : e.x) * scale : -INFINITY;
    }
  }
  if (nbad) atomicAdd(a.bad, nbad);
  estep_epilogue(a, Lv, &sS[0][0], &sK[0][0]);
}

// True-Poisson likelihood: L = log w + sum k log s + K log(K/S_r) - K.
__global__ void __launch_bounds__(TPB, 1) estep_pois_fp32_kernel(EstepArgs a) {
  __shared__ __align__(16) float sS[2][STG], sK[2][STG];
  const int ty4 = (threadIdx.x >> 4) * 4, tx4 = (threadIdx.x & 15) * 4;
  const int r0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  f32x2 acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
  float4 vr[2], vk[2];
  const int nk = a.Kp / BK;
  ld_tile(a.S, a.Kp, r0, a.R, 0, vr);
  ld_tile(a.Kraw, a.Kp, n0, a.N, 0, vk);
  for (int kb = 0; kb < nk; ++kb) {
    float *s = sS[kb & 1], *t = sK[kb & 1];
    st_tile_t(s, vr, [](float v) { return logf(fmaxf(v, kSliceFloor)); });
    st_tile_t(t, vk, [](float v) { return v; });
    __syncthreads();
    if (kb + 1 < nk) {
      ld_tile(a.S, a.Kp, r0, a.R, (kb + 1) * BK, vr);
      ld_tile(a.Kraw, a.Kp, n0, a.N, (kb + 1) * BK, vk);
    }
#pragma unroll 8
    for (int k = 0; k < BK; ++k) {
      f32x2 rl[8], pk[4];
      ld_twice(s, k, ty4, rl);
      ld_pairs(t, k, tx4, pk);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = ptx::fma2(pk[j], rl[i], acc[i][j]);
    }
  }
  __syncthreads();  // sS and sK are free
  float Lv[8][8], phi[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = r0 + micro_idx(ty4, i);
    const bool rok = r < a.R;
    const float lw = rok ? logf(__ldg(a.rotw + r)) : 0.0f;
    const float Sr = rok ? __ldg(a.rot_ssum + r) : 1.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float2 e2 = ptx::unpack2(acc[i][j >> 1]);
      const float e = (j & 1) ? e2.y : e2.x;
      const int n = n0 + micro_idx(tx4, j);
      const float Ki = n < a.N ? __ldg(a.Ksum + n) : 0.0f;
      float l, f;
      if (a.known_intensity) {
        f = 1.0f;
        l = lw + e - Sr;
      } else if (Ki > 0.0f) {
        f = Ki / Sr;
        l = lw + e + Ki * logf(f) - Ki;
      } else {
        f = 0.0f;
        l = lw;
      }
      Lv[i][j] = rok && n < a.N ? l : -INFINITY;
      phi[i][j] = f;
    }
  }
  store_tile(a, a.PHI, phi);
  estep_epilogue(a, Lv, &sS[0][0], &sK[0][0]);
}

// ------------------------------------------------------- normalise -------
constexpr float kLog2E = 1.4426950408889634f;

// Per pattern, over the rotation tiles' (max, sum exp) pairs: M = the largest max
// and s = sum_t s_t exp(m_t - M), FP64.  A block takes 32 patterns; its eight
// warps share the tiles (one thread per pattern left a small problem on a few
// SMs, and its two serial walks over the tiles took 22 to 44 us there), and their
// sums are added in warp order.  Results in warp 0, lane = pattern.
constexpr int kLseWarps = 8;
__device__ __forceinline__ void lse_tiles(const float2* __restrict__ part, int n_rt, int N, int n,
                                          float& M, double& s) {
  __shared__ float sm[kLseWarps][32];
  __shared__ double ss[kLseWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float m = -INFINITY;
  if (n < N)
    for (int t = warp; t < n_rt; t += kLseWarps) m = fmaxf(m, part[(size_t)t * N + n].x);
  sm[warp][lane] = m;
  __syncthreads();
  M = -INFINITY;
#pragma unroll
  for (int w = 0; w < kLseWarps; ++w) M = fmaxf(M, sm[w][lane]);
  double a = 0.0;
  if (n < N && M > -INFINITY)
    for (int t = warp; t < n_rt; t += kLseWarps) {
      const float2 v = part[(size_t)t * N + n];
      // v.y <= 128, so tiles 50 below the largest add less than 2^-65 of the sum; the
      // FP64 exponentials are the kernel's time
      if (v.x - M > -50.0f) a += (double)v.y * exp((double)v.x - (double)M);
    }
  ss[warp][lane] = a;
  __syncthreads();
  s = 0.0;
  if (warp == 0)
#pragma unroll
    for (int w = 0; w < kLseWarps; ++w) s += ss[w][lane];
}

// A pattern's lse in the forms its consumers read: FP64; two floats hi + lo (hi =
// fl(lse), lo = fl(lse - hi)), so that L - lse is formed in FP32 to the same accuracy;
// and in four copies, copy h from pattern h on, hi and -lo log2(e) in arrays of their
// own: the rows [R][N] of the likelihood start at any 4-byte boundary, and reading
// them by 16 bytes, mprep_hi_kernel finds their lse by 16 bytes as well.
struct LseOut {
  double* lse;
  float2* lse2;
  float* shifted;  // [4][2][ld]
  int ld;
  __device__ __forceinline__ void store(int n, double l) const {
    const bool ok = isfinite(l);
    const float hi = (float)l, lo = ok ? (float)(l - (double)hi) : 0.0f;
    lse[n] = l;
    lse2[n] = make_float2(hi, lo);
#pragma unroll
    for (int h = 0; h < 4; ++h)
      if (n >= h) {
        shifted[(size_t)(2 * h) * ld + n - h] = ok ? hi : INFINITY;  // P = 0
        shifted[(size_t)(2 * h + 1) * ld + n - h] = -lo * kLog2E;
      }
  }
};

// lse_i = M + log(s), FP64.
// Patterns with no valid pair get lse = +inf (all responsibilities 0).
// ll_part[block] = the sum of the block's finite lse.
__global__ void __launch_bounds__(32 * kLseWarps) lse_combine_kernel(
    const float2* __restrict__ part, int n_rt, int N, LseOut out, double* __restrict__ ll_part) {
  const int n = blockIdx.x * 32 + (threadIdx.x & 31);
  float M;
  double s;
  lse_tiles(part, n_rt, N, n, M, s);
  if (threadIdx.x >= 32) return;
  double l = INFINITY;
  if (n < N) {
    if (M > -INFINITY) l = (double)M + log(s);
    out.store(n, l);
  }
  double t = isfinite(l) ? l : 0.0;
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  if (threadIdx.x == 0) ll_part[blockIdx.x] = t;
}

__global__ void fill_part_kernel(float2* __restrict__ part, size_t n) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride)
    part[e] = make_float2(-INFINITY, 0.0f);
}

// ---- responsibilities -> M-step operand --------------------------------
// One block per rotation row: P = exp(L - lse), Q = P / phi, T_r = sum_i P, the
// row's captured mass and the inserted-mass bound sum_i Q_ri K_i.  Element math is
// FP32 (L - lse with lse as float hi + lo, since FP64 arithmetic is scarce on this
// GPU); per-thread sums are FP32 and the block sums FP64.

// Row sums (t, b, m) and maximum over the block, in thread 0 (mx in every thread):
// FP32 warp shuffles over the threads' FP32 partials, then the warps' sums in FP64
// on warp 0 (FP64 runs at a small fraction of the FP32 rate).
__device__ __forceinline__ void row_sums(float t, float b, float m, float& mx, double& st,
                                         double& sb, double& sm) {
  __shared__ double wsum[3][32];
  __shared__ float wmax[32];
  __shared__ float row_max;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    t += __shfl_down_sync(0xffffffffu, t, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
    m += __shfl_down_sync(0xffffffffu, m, o);
    mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
  }
  if (lane == 0) {
    wsum[0][warp] = (double)t;
    wsum[1][warp] = (double)b;
    wsum[2][warp] = (double)m;
    wmax[warp] = mx;
  }
  __syncthreads();
  if (warp == 0) {
    st = lane < nw ? wsum[0][lane] : 0.0;
    sb = lane < nw ? wsum[1][lane] : 0.0;
    sm = lane < nw ? wsum[2][lane] : 0.0;
    mx = lane < nw ? wmax[lane] : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      st += __shfl_down_sync(0xffffffffu, st, o);
      sb += __shfl_down_sync(0xffffffffu, sb, o);
      sm += __shfl_down_sync(0xffffffffu, sm, o);
      mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
    }
    if (lane == 0) row_max = mx;
  }
  __syncthreads();
  mx = row_max;
}

// The power of two that brings a row whose largest entry is mx near 2^14.
__device__ __forceinline__ int row_exponent(float mx) {
  const int ex = mx > 0.0f ? 14 - ilogbf(mx) - 1 : 0;
  return max(-100, min(100, ex));
}

struct MprepArgs {
  float* L;
  const float* PHI;
  const float2* lse2;
  const float* lse_shifted;  // LseOut, ld = ldq
  const float* Ksum;   // null: no mass bound wanted
  const float* cnorm;  // null: 1
  int N, ldq, n_rt;
  float* Q;            // FP32 M-step
  __half *Qh, *Ql;     // tensor M-step
  float* qscale;
  float* T;
  double *row_mass, *row_bound, *row_margin;
  const unsigned char* tstate;  // pruned iteration: [pattern tile][rotation tile] = 0 not
                                // evaluated (P = 0), 1 evaluated, 2 evaluated margin tile
                                // (its mass is summed); null: all evaluated
  int chunk;    // patterns per CTA of a row's cluster (mprep_hi_kernel)
  int stage;    // the row's P c_i / phi is kept in shared memory between the passes
  int write_p;  // P over L
};

// The tensor M-step's operand as FP16 hi only: Q' = P c_i / phi (phi holds c_i
// num/den, the M-step multiplies raw counts), [R][ldq], each row scaled by 2^e_r so
// that its largest entry sits near 2^14 (qscale_r = 2^-e_r).  Taking P through an
// 11-bit rounding, it is served by the hardware exponential and reciprocal, both to a
// unit or two in the last place; P = 2^x also takes the rounding of x, which is
// relative 2^-25 |x| at most (2^-18 where P nears 2^-126, below which it is 0).  Bound by HBM and by issue: 8 bytes read and 2
// written per pair, and phi only where P is not 0.  A row is kept in shared memory
// between the two passes, shared by a cluster of 1 to 8 CTAs of `chunk` patterns, so
// that four CTAs fit an SM and one's reads overlap another's writes; a row too long
// for that is formed again.  With 50 to 90 instructions per pair instead of 30, of
// which phi's load waited for L's, 10,860 x 50,000 pairs took 2,988 us (1,531 now),
// 25,680 x 20,000 1,537 (1,000), 10,860 x 10,000 376 (197), 10,860 x 4,999 377 (166).
constexpr int kMprepChunk = 14208;     // patterns per CTA, 55.5 KB
constexpr int kMprepChunkMax = 56832;  // where eight CTAs per row do not suffice, 222 KB
constexpr int kMprepStageLo = 30720;   // of mprep_kernel, two blocks per SM (120 KB)

template <bool PLAIN>
__global__ void __launch_bounds__(512, 2) mprep_hi_kernel(MprepArgs a) {
  extern __shared__ __align__(16) float smem_row[];  // [chunk + 4] when stage
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int ctas = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int r = (int)blockIdx.x / ctas, bd = (int)blockDim.x;
  const int i0 = rank * a.chunk;                               // this CTA's patterns
  const int n = max(0, min(a.N - i0, a.chunk));                // of the row,
  const int n_out = max(0, min(a.ldq - i0, a.chunk));          // and of the operand
  const unsigned char* ts =
      !PLAIN && a.tstate ? a.tstate + (size_t)(i0 >> 7) * a.n_rt + (r >> 7) : nullptr;
  float* Lr = a.L + (size_t)r * a.N + i0;
  const float* Fr = a.PHI + (size_t)r * a.N + i0;
  const float* hi0 = a.lse_shifted + i0;
  // patterns before the first 16-byte boundary of the row; the row in shared memory
  // has the same alignment
  const int head = min(n, (int)(((4 - (((size_t)r * a.N + i0) & 3)) & 3)));
  float* qrow = smem_row + ((4 - head) & 3);
  float t = 0.0f, b = 0.0f, qmax = 0.0f, mg = 0.0f;
  auto state = [&](int i) { return ts ? (int)ts[(size_t)(i >> 7) * a.n_rt] : 1; };
  auto prob = [](float l, float hi, float lo) {  // exp(l - lse), 0 for a NaN
    float p;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p) : "f"(__fmaf_rn(l - hi, kLog2E, lo)));
    return fmaxf(p, 0.0f);
  };
  auto over = [](float P, float f) {
    float rf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(f));
    return P * rf;
  };
  auto weigh = [&](int i, float q) {  // P / phi: its part of the mass bound, times c_i
    if (PLAIN) return q;
    if (a.Ksum) b = __fmaf_rn(q, __ldg(a.Ksum + i0 + i), b);
    return a.cnorm ? __fmul_rn(q, __ldg(a.cnorm + i0 + i)) : q;
  };
  auto one = [&](int i) {
    const int st = state(i);
    const float P = st ? prob(Lr[i], hi0[i], hi0[a.ldq + i]) : 0.0f;
    if (!PLAIN && a.write_p) Lr[i] = P;
    const float f = P > 0.0f ? __ldg(Fr + i) : 0.0f;
    const float q = weigh(i, f > 0.0f ? over(P, f) : 0.0f);
    t += P;
    if (st == 2) mg += P;
    qmax = fmaxf(qmax, q);
    if (a.stage) qrow[i] = q;
  };
  if (ts && head) {  // a 4-tuple may lie in two pattern tiles
    for (int i = threadIdx.x; i < n; i += bd) one(i);
  } else {
    const int n4 = (n - head) / 4, rest = n - 4 * n4;
    if ((int)threadIdx.x < rest) one((int)threadIdx.x < head ? threadIdx.x : 4 * n4 + threadIdx.x);
    float4* L4 = reinterpret_cast<float4*>(Lr + head);
    const float4* F4 = reinterpret_cast<const float4*>(Fr + head);
    const float* sh = hi0 + (size_t)(2 * head) * a.ldq;  // from pattern i0 + head on
    const float4* H4 = reinterpret_cast<const float4*>(sh);
    const float4* O4 = reinterpret_cast<const float4*>(sh + a.ldq);
    float4* Q4 = reinterpret_cast<float4*>(qrow + head);
    // two 4-tuples per thread and turn, their loads in flight together; phi is not
    // waited for where the last turn needed it
    const float4 none = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f), ones = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    bool eager = true;
    for (int j0 = threadIdx.x; j0 < n4; j0 += 2 * bd) {
      float4 l[2], hi[2], lo[2], f[2];
      int st[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = j0 + h * bd;
        st[h] = j < n4 ? state(head + 4 * j) : 0;
        l[h] = none;
        hi[h] = lo[h] = zero;
        f[h] = ones;
        if (st[h]) {
          l[h] = L4[j];
          if (eager) f[h] = __ldg(F4 + j);
          hi[h] = __ldg(H4 + j);
          lo[h] = __ldg(O4 + j);
        }
      }
      bool any[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        l[h].x = prob(l[h].x, hi[h].x, lo[h].x);
        l[h].y = prob(l[h].y, hi[h].y, lo[h].y);
        l[h].z = prob(l[h].z, hi[h].z, lo[h].z);
        l[h].w = prob(l[h].w, hi[h].w, lo[h].w);
        const float sum = (l[h].x + l[h].y) + (l[h].z + l[h].w);
        any[h] = sum > 0.0f;
        t += sum;
        if (!PLAIN && st[h] == 2) mg += sum;
        if (any[h] && !eager) f[h] = __ldg(F4 + j0 + h * bd);
      }
      eager = any[0] || any[1];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = j0 + h * bd, i = head + 4 * j;
        if (j >= n4) break;
        if (!PLAIN && a.write_p) L4[j] = l[h];
        float4 q = zero;
        if (any[h]) {
          q = make_float4(over(l[h].x, f[h].x), over(l[h].y, f[h].y), over(l[h].z, f[h].z),
                          over(l[h].w, f[h].w));
          if (!(fminf(fminf(f[h].x, f[h].y), fminf(f[h].z, f[h].w)) > 0.0f)) {
            // patterns without counts (true Poisson: phi = 0)
            q.x = f[h].x > 0.0f ? q.x : 0.0f;
            q.y = f[h].y > 0.0f ? q.y : 0.0f;
            q.z = f[h].z > 0.0f ? q.z : 0.0f;
            q.w = f[h].w > 0.0f ? q.w : 0.0f;
          }
          if (!PLAIN) {
            q.x = weigh(i, q.x);
            q.y = weigh(i + 1, q.y);
            q.z = weigh(i + 2, q.z);
            q.w = weigh(i + 3, q.w);
          }
          qmax = fmaxf(fmaxf(qmax, fmaxf(q.x, q.y)), fmaxf(q.z, q.w));
        }
        if (a.stage) Q4[j] = q;
      }
    }
  }
  if (a.stage)
    for (int i = n + threadIdx.x; i < n_out; i += bd) qrow[i] = 0.0f;
  double r0s = 0.0, r1s = 0.0, r2s = 0.0;
  row_sums(t, b, mg, qmax, r0s, r1s, r2s);
  __shared__ double part[3];
  __shared__ float part_max;
  if (ctas > 1) {  // the other CTAs' parts, in rank order
    if (threadIdx.x == 0) {
      part[0] = r0s;
      part[1] = r1s;
      part[2] = r2s;
      part_max = qmax;
    }
    cluster.sync();
    for (int k = 0; k < ctas; ++k) qmax = fmaxf(qmax, *cluster.map_shared_rank(&part_max, k));
    if (threadIdx.x == 0 && rank == 0)
      for (int k = 1; k < ctas; ++k) {
        const double* o = cluster.map_shared_rank(part, k);
        r0s += o[0];
        r1s += o[1];
        r2s += o[2];
      }
  }
  const int ex = row_exponent(qmax);
  if (threadIdx.x == 0 && rank == 0) {
    a.T[r] = (float)r0s;
    a.row_mass[r] = r0s;
    a.row_bound[r] = r1s;
    if (a.row_margin) a.row_margin[r] = r2s;
    a.qscale[r] = ldexpf(1.0f, -ex);
  }
  const float up = ldexpf(1.0f, ex);
  auto again = [&](int i) -> float {  // the row's entry, formed once more
    if (i >= n || !state(i)) return 0.0f;
    const float P = a.write_p ? Lr[i] : prob(Lr[i], hi0[i], hi0[a.ldq + i]);
    const float f = P > 0.0f ? __ldg(Fr + i) : 0.0f;
    return weigh(i, f > 0.0f ? over(P, f) : 0.0f);
  };
  // ldq and chunk are multiples of 128
  __half* out = a.Qh + (size_t)r * a.ldq + i0;
  if (a.stage && !head) {  // eight FP16 values (16 bytes) per store
    for (int j = threadIdx.x; j < n_out / 8; j += bd) {
      const float4 x = *reinterpret_cast<const float4*>(qrow + 8 * j);
      const float4 y = *reinterpret_cast<const float4*>(qrow + 8 * j + 4);
      union {
        __half2 h[4];
        uint4 u;
      } p;
      p.h[0] = __floats2half2_rn(__fmul_rn(x.x, up), __fmul_rn(x.y, up));
      p.h[1] = __floats2half2_rn(__fmul_rn(x.z, up), __fmul_rn(x.w, up));
      p.h[2] = __floats2half2_rn(__fmul_rn(y.x, up), __fmul_rn(y.y, up));
      p.h[3] = __floats2half2_rn(__fmul_rn(y.z, up), __fmul_rn(y.w, up));
      reinterpret_cast<uint4*>(out)[j] = p.u;
    }
  } else {
    for (int j = threadIdx.x; j < n_out / 2; j += bd) {
      const float x = a.stage ? qrow[2 * j] : again(2 * j);
      const float y = a.stage ? qrow[2 * j + 1] : again(2 * j + 1);
      reinterpret_cast<__half2*>(out)[j] = __floats2half2_rn(__fmul_rn(x, up), __fmul_rn(y, up));
    }
  }
  if (ctas > 1) cluster.sync();  // no CTA leaves while another reads its part
}

// The general form: Q in FP32 (FP32 M-step, [R][ldq], zero padded) or as FP16 hi +
// lo, with the correctly rounded exponential and quotient.  Bound by the bytes in
// flight: two 4-tuples per thread and turn where rows start at 16-byte boundaries, four
// pairs elsewhere.  One pair at a time took 649 us for 10,860 x 10,000 pairs, 1,746 for
// 10,860 x 20,000 and 647 for 10,860 x 9,999 (hi + lo), now 371, 646 and 463; 3,240 x
// 2,000 (FP32) 54, now 42.
__global__ void __launch_bounds__(512, 2) mprep_kernel(MprepArgs a) {
  extern __shared__ __align__(16) float qrow[];
  const int r = blockIdx.x, N = a.N, bd = (int)blockDim.x;
  const unsigned char* ts = a.tstate ? a.tstate + (r >> 7) : nullptr;
  auto state = [&](int i) { return ts ? (int)ts[(size_t)(i >> 7) * a.n_rt] : 1; };
  float t = 0.0f, b = 0.0f, qmax = 0.0f, mg = 0.0f;
  float* const Lr = a.L + (size_t)r * N;
  const float* const Fr = a.PHI + (size_t)r * N;
  // P of pattern i; q becomes its entry of the operand (f: phi, 0 where not evaluated)
  auto pair = [&](int i, int st, float l, float f, float2 li, float& q) {
    float P = 0.0f;
    if (st && isfinite(li.x) && l > -INFINITY) P = expf((l - li.x) - li.y);
    if (st == 2) mg += P;
    q = f > 0.0f ? __fdiv_rn(P, f) : 0.0f;
    t += P;
    if (a.Ksum) b = __fmaf_rn(q, __ldg(a.Ksum + i), b);
    if (a.Qh && a.cnorm) q = __fmul_rn(q, __ldg(a.cnorm + i));
    qmax = fmaxf(qmax, q);
    return P;
  };
  if ((N & 3) == 0) {  // (a 4-tuple lies in one pattern tile)
    float4* L4 = reinterpret_cast<float4*>(Lr);
    const float4* F4 = reinterpret_cast<const float4*>(Fr);
    const float4* S4 = reinterpret_cast<const float4*>(a.lse2);
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int j0 = threadIdx.x; j0 < N / 4; j0 += 2 * bd) {
      float4 l[2], f[2];
      int st[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = j0 + h * bd;
        st[h] = j < N / 4 ? state(4 * j) : 0;
        l[h] = st[h] ? L4[j] : zero;
        f[h] = st[h] ? __ldg(F4 + j) : zero;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = j0 + h * bd, i = 4 * j;
        if (j >= N / 4) break;
        const float4 s01 = __ldg(S4 + 2 * j), s23 = __ldg(S4 + 2 * j + 1);
        float4 P, q;
        P.x = pair(i, st[h], l[h].x, f[h].x, make_float2(s01.x, s01.y), q.x);
        P.y = pair(i + 1, st[h], l[h].y, f[h].y, make_float2(s01.z, s01.w), q.y);
        P.z = pair(i + 2, st[h], l[h].z, f[h].z, make_float2(s23.x, s23.y), q.z);
        P.w = pair(i + 3, st[h], l[h].w, f[h].w, make_float2(s23.z, s23.w), q.w);
        if (a.write_p) L4[j] = P;
        if (a.Q) *reinterpret_cast<float4*>(a.Q + (size_t)r * a.ldq + i) = q;
        if (a.stage) *reinterpret_cast<float4*>(qrow + i) = q;
      }
    }
  } else {
    for (int i0 = threadIdx.x; i0 < N; i0 += 4 * bd) {  // four loads in flight
      float l[4], f[4];
      float2 li[4];
      int st[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int i = i0 + h * bd;
        st[h] = i < N ? state(i) : 0;
        l[h] = st[h] ? Lr[i] : 0.0f;
        f[h] = st[h] ? __ldg(Fr + i) : 0.0f;
        li[h] = st[h] ? __ldg(a.lse2 + i) : make_float2(0.0f, 0.0f);
      }
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int i = i0 + h * bd;
        if (i >= N) break;
        float q;
        const float P = pair(i, st[h], l[h], f[h], li[h], q);
        if (a.write_p) Lr[i] = P;
        if (a.Q) a.Q[(size_t)r * a.ldq + i] = q;
        if (a.stage) qrow[i] = q;
      }
    }
  }
  if (a.Q)
    for (int i = N + threadIdx.x; i < a.ldq; i += blockDim.x) a.Q[(size_t)r * a.ldq + i] = 0.0f;
  double r0s = 0.0, r1s = 0.0, r2s = 0.0;
  row_sums(t, b, mg, qmax, r0s, r1s, r2s);
  if (threadIdx.x == 0) {
    a.T[r] = (float)r0s;
    a.row_mass[r] = r0s;
    a.row_bound[r] = r1s;
    if (a.row_margin) a.row_margin[r] = r2s;
  }
  if (!a.Qh) return;
  const int ex = row_exponent(qmax);
  const float up = ldexpf(1.0f, ex);
  auto qval = [&](int i) -> float {
    if (i >= N) return 0.0f;
    if (a.stage) return __fmul_rn(qrow[i], up);
    // re-read the row (L now holds P)
    const size_t e = (size_t)r * N + i;
    const float f = a.PHI[e];
    const float q = f > 0.0f ? __fdiv_rn(a.L[e], f) : 0.0f;
    return __fmul_rn(a.cnorm ? __fmul_rn(q, __ldg(a.cnorm + i)) : q, up);
  };
  // ldq is a multiple of 128: four FP16 values (8 bytes) per store
  for (int j = threadIdx.x; j < a.ldq / 4; j += blockDim.x) {
    const int i = 4 * j;
    union Pack4 {
      __half h[4];
      uint2 u;
    } hi, lo;
    for (int c = 0; c < 4; ++c) {
      const float q = qval(i + c);
      hi.h[c] = __float2half_rn(q);
      lo.h[c] = __float2half_rn(q - __half2float(hi.h[c]));
    }
    *reinterpret_cast<uint2*>(a.Qh + (size_t)r * a.ldq + i) = hi.u;
    *reinterpret_cast<uint2*>(a.Ql + (size_t)r * a.ldq + i) = lo.u;
  }
  if (threadIdx.x == 0) a.qscale[r] = ldexpf(1.0f, -ex);
}

// P = exp(L - lse) in place over the plan's [R][N] rows, with mprep_kernel's
// expression for an evaluated pair.  (mprep_hi_kernel, which writes P itself where
// pruning reads it, takes the hardware exponential: see its bound.)
__global__ void respons_from_loglik_kernel(float* __restrict__ L, const float2* __restrict__ lse2,
                                           int N, long long total) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += stride) {
    const int i = (int)(e % N);
    const float l = L[e];
    const float2 li = lse2[i];
    float P = 0.0f;
    if (isfinite(li.x) && l > -INFINITY) P = expf((l - li.x) - li.y);
    L[e] = P;
  }
}

int plan_respons_ready(emc_plan* p) {
  if (p->p_written) return EMC_OK;
  emc_ctx* ctx = p->ctx;
  const long long total = (long long)p->d.n_rot * p->d.n_images;
  respons_from_loglik_kernel<<<ctx->sm_count * 8, 256, 0, ctx->stream>>>(p->L, p->lse2,
                                                                        p->d.n_images, total);
  const int rc = after_launch(ctx, "respons_from_loglik_kernel");
  if (!rc) p->p_written = true;
  return rc;
}

// ---------------------------------------------------------- insert -------
struct InsertCtx {
  float* model;
  float* weight;
  ulonglong2* fix2;         // interleaved fixed-point (model, weight) sums
  float2* acc2;             // interleaved (model, weight) sums: one 8-byte atomic per point
  const float2* fix_scale;  // {model, weight} fixed-point scales (deterministic mode)
  float* u;              // sorted mode: pair values [P_eff][ldu] instead of insertion
  int ldu;
  int side;
  int interp;
  int deterministic;
};

__device__ __forceinline__ void add_voxel(const InsertCtx& c, size_t v, float val, float w) {
  if (c.deterministic) {
    const float2 sc = __ldg(c.fix_scale);
    atomicAdd(&c.fix2[v].x, (unsigned long long)fixed_from_float(__fmul_rn(val, sc.x)));
    atomicAdd(&c.fix2[v].y, (unsigned long long)fixed_from_float(__fmul_rn(w, sc.y)));
  } else {
    atomicAdd(c.acc2 + v, make_float2(val, w));
  }
}

// The voxel nearest to the detector point (x, y, z) rotated by R, -1 outside the
// reference's insertion bounds (>= 0, emc_atomic.cu:67-69).
__device__ __forceinline__ long long nearest_voxel(const InsertCtx& c, const RotMat& R, float x,
                                                   float y, float z) {
  const int side = c.side;
  const long ix = voxel_round(voxel_coord(side, rotate_row(R, 0, x, y, z)));
  const long iy = voxel_round(voxel_coord(side, rotate_row(R, 1, x, y, z)));
  const long iz = voxel_round(voxel_coord(side, rotate_row(R, 2, x, y, z)));
  if (ix < 0 || ix >= side || iy < 0 || iy >= side || iz < 0 || iz >= side) return -1;
  return ((long long)iz * side + iy) * side + ix;
}

// Trilinear splat of value `val` with weight `w` at the rotated point.
__device__ __forceinline__ void splat_point(const InsertCtx& c, const RotMat& R, float x, float y,
                                            float z, float val, float w) {
  const int side = c.side;
  const float cx = voxel_coord(side, rotate_row(R, 0, x, y, z));
  const float cy = voxel_coord(side, rotate_row(R, 1, x, y, z));
  const float cz = voxel_coord(side, rotate_row(R, 2, x, y, z));
  const float fx0 = floorf(cx), fy0 = floorf(cy), fz0 = floorf(cz);
  const int x0 = (int)fx0, y0 = (int)fy0, z0 = (int)fz0;
  const float tx = cx - fx0, ty = cy - fy0, tz = cz - fz0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int xi = x0 + (k & 1), yi = y0 + ((k >> 1) & 1), zi = z0 + (k >> 2);
    if (xi < 0 || xi >= side || yi < 0 || yi >= side || zi < 0 || zi >= side) continue;
    const float f = ((k & 1) ? tx : 1.0f - tx) * (((k >> 1) & 1) ? ty : 1.0f - ty) *
                    ((k >> 2) ? tz : 1.0f - tz);
    if (f <= 0.0f) continue;
    add_voxel(c, ((size_t)zi * side + yi) * side + xi, val * f, w * f);
  }
}

// ---------------------------------------------------- FP32 M-step --------
struct MstepArgs {
  const float* Q;     // [R][ldq]
  const float* Kraw;  // [N][Kp]
  const float* T;     // [R]
  const float* rot;   // [4R]
  const float *cx, *cy, *cz;  // [Kp]
  int R, N, Kp, ldq, P_eff;
  InsertCtx ins;
};

// U = Q K for a 128-rotation x 128-pixel tile, inserted in the epilogue (slice =
// U / T_r with weight T_r: U itself goes to the model sum).
__global__ void __launch_bounds__(TPB, 2) mstep_fp32_kernel(MstepArgs a) {
  __shared__ __align__(16) float sq[2][STG], sk[2][STG];
  __shared__ RotMat sR[BM];
  const int ty4 = (threadIdx.x >> 4) * 4, tx4 = (threadIdx.x & 15) * 4;
  const int r0 = blockIdx.y * BM, q0 = blockIdx.x * BN;
  if (threadIdx.x < BM) {
    const int r = r0 + threadIdx.x;
    if (r < a.R) sR[threadIdx.x] = quat_to_matrix(a.rot + 4 * (size_t)r);
  }
  f32x2 acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
  float4 vq[2], vk[2];
  const int nk = (a.N + BK - 1) / BK;
  auto ld_k = [&](int kb) {
    // [16 pattern rows][128 pixels]: 512 float4, thread t: f = t, t + 256
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int f = threadIdx.x + u * TPB;
      const int row = f >> 5, c4 = f & 31;
      const int i = kb * BK + row;
      vk[u] = i < a.N ? __ldg(reinterpret_cast<const float4*>(a.Kraw + (size_t)i * a.Kp + q0) + c4)
                      : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto st_k = [&](float* dst) {  // with the columns' bits flipped as in st_tile_t
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int f = threadIdx.x + u * TPB;
      const int row = f >> 5, c = (f & 31) * 4;
      *reinterpret_cast<float4*>(dst + row * BN + (c ^ ((row >> 2) << 3))) = vk[u];
    }
  };
  ld_tile(a.Q, a.ldq, r0, a.R, 0, vq);
  ld_k(0);
  for (int kb = 0; kb < nk; ++kb) {
    float *s = sq[kb & 1], *t = sk[kb & 1];
    st_tile_t(s, vq, [](float v) { return v; });
    st_k(t);
    __syncthreads();
    if (kb + 1 < nk) {
      ld_tile(a.Q, a.ldq, r0, a.R, (kb + 1) * BK, vq);
      ld_k(kb + 1);
    }
#pragma unroll 4
    for (int k = 0; k < BK; ++k) {
      f32x2 rq[8], pk[4];
      ld_twice(s, k, ty4, rq);
      ld_pairs(t, k, tx4, pk);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = ptx::fma2(pk[j], rq[i], acc[i][j]);
    }
  }
  // ---- epilogue
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int rl = micro_idx(ty4, i);
    const int r = r0 + rl;
    if (r >= a.R) continue;
    const float t = __ldg(a.T + r);
    const bool live = t > 1e-10f;
    float u[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 v = ptx::unpack2(acc[i][j]);
      u[2 * j] = v.x;
      u[2 * j + 1] = v.y;
    }
    if (a.ins.u) {  // sorted mode: the pair values, 0 where the rotation inserts nothing
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int q = q0 + micro_idx(tx4, j);
        if (q < a.P_eff) a.ins.u[(size_t)q * a.ins.ldu + r] = live ? u[j] : 0.0f;
      }
      continue;
    }
    if (!live) continue;
    const RotMat R = sR[rl];
    if (a.ins.interp == EMC_INTERP_NEAREST) {
      long long v[8];  // all voxels before the first atomic
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int q = q0 + micro_idx(tx4, j);
        v[j] = q < a.P_eff ? nearest_voxel(a.ins, R, __ldg(a.cx + q), __ldg(a.cy + q), __ldg(a.cz + q))
                           : -1;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (v[j] >= 0) add_voxel(a.ins, (size_t)v[j], u[j], t);
      continue;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int q = q0 + micro_idx(tx4, j);
      if (q < a.P_eff)
        splat_point(a.ins, R, __ldg(a.cx + q), __ldg(a.cy + q), __ldg(a.cz + q), u[j], t);
    }
  }
}

// ------------------------------------------------------- finishing -------
// Upper bounds of the inserted model and weight mass (deterministic mode):
// 1.25 * sum_r sum_i Q_ri K_i and 1.25 * P_eff * sum_r T_r, FP64, fixed order,
// and the fixed-point scales they give.
__global__ void insert_bounds_kernel(const double* __restrict__ row_mass,
                                     const double* __restrict__ row_bound, int R, int P_eff,
                                     double* __restrict__ out, float2* __restrict__ scale) {
  __shared__ double sm[256], sw[256];
  double m = 0.0, w = 0.0;
  for (int r = threadIdx.x; r < R; r += blockDim.x) {
    m += row_bound[r];
    w += row_mass[r];
  }
  sm[threadIdx.x] = m;
  sw[threadIdx.x] = w;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      sm[threadIdx.x] += sm[threadIdx.x + o];
      sw[threadIdx.x] += sw[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = 1.25 * sm[0] + 1e-30;
    out[1] = 1.25 * sw[0] * (double)P_eff + 1e-30;
    *scale = make_float2(fix_scale_pow2(out[0]), fix_scale_pow2(out[1]));
  }
}

// Inserted sums -> weight and model / weight (-1 where the weight is 0,
// emc_cuda.cu:758-768), from the fixed-point (deterministic) or the
// interleaved float accumulators; part: the blocks' {sum, count} of its positive
// voxels, for the normalisation.
__global__ void finish_insert_kernel(const ulonglong2* __restrict__ fx,
                                     const float2* __restrict__ fix_scale,
                                     const float2* __restrict__ acc2, float* __restrict__ model,
                                     float* __restrict__ weight, long long n,
                                     double* __restrict__ part) {
  const float2 sc = fx ? *fix_scale : make_float2(1.0f, 1.0f);
  const double inv_m = 1.0 / (double)sc.x, inv_w = 1.0 / (double)sc.y;  // powers of two
  double s = 0.0, c = 0.0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    float m, w;
    if (fx) {
      const ulonglong2 u = fx[v];
      m = (float)((double)(long long)u.x * inv_m);
      w = (float)((double)(long long)u.y * inv_w);
    } else {
      const float2 a = acc2[v];
      m = a.x;
      w = a.y;
    }
    weight[v] = w;
    const float q = w > 0.0f ? __fdiv_rn(m, w) : -1.0f;
    model[v] = q;
    if (q > 0.0f) {
      s += (double)q;
      c += 1.0;
    }
  }
  block_sum2(s, c);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = s;
    part[2 * blockIdx.x + 1] = c;
  }
}

// ---- one rank of a rotation split --------------------------------------
// Per pattern, over this plan's rotations: the largest log-likelihood and the
// sum of exp(L - max) (FP64), from the per-tile partials.
__global__ void __launch_bounds__(32 * kLseWarps) rank_partial_kernel(
    const float2* __restrict__ part, int n_rt, int N, float* __restrict__ out_max,
    double* __restrict__ out_sum) {
  const int n = blockIdx.x * 32 + (threadIdx.x & 31);
  float M;
  double s;
  lse_tiles(part, n_rt, N, n, M, s);
  if (threadIdx.x >= 32 || n >= N) return;
  out_max[n] = M;
  out_sum[n] = s;
}

// The normaliser combined over all ranks, in the plan's own form (FP64 and
// float hi + lo).
__global__ void lse_from_global_kernel(const double* __restrict__ lse_in, int N,
                                       LseOut out) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n < N) out.store(n, lse_in[n]);
}

// The inserted sums as floats (model sum of T_r x slice, weight sum of T_r),
// exactly as finish_insert_kernel reads them.
__global__ void sums_out_kernel(const ulonglong2* __restrict__ fx,
                                const float2* __restrict__ fix_scale,
                                const float2* __restrict__ acc2,
                                float* __restrict__ msum, float* __restrict__ wsum, long long n) {
  const float2 sc = fx ? *fix_scale : make_float2(1.0f, 1.0f);
  const double inv_m = 1.0 / (double)sc.x, inv_w = 1.0 / (double)sc.y;  // powers of two
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    if (fx) {
      const ulonglong2 u = fx[v];
      msum[v] = (float)((double)(long long)u.x * inv_m);
      wsum[v] = (float)((double)(long long)u.y * inv_w);
    } else {
      const float2 a = acc2[v];
      msum[v] = a.x;
      wsum[v] = a.y;
    }
  }
}

// main.cpp:467-476 after the all-reduce: both sums divided by the number of
// ranks (devide_part), then model / weight (-1 where the weight is 0).
__global__ void model_from_sums_kernel(const float* __restrict__ msum,
                                       const float* __restrict__ wsum, float n_ranks,
                                       float* __restrict__ model, float* __restrict__ weight,
                                       long long n, double* __restrict__ part) {
  double s = 0.0, c = 0.0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    const float m = __fdiv_rn(msum[v], n_ranks), w = __fdiv_rn(wsum[v], n_ranks);
    weight[v] = w;
    const float q = w > 0.0f ? __fdiv_rn(m, w) : -1.0f;
    model[v] = q;
    if (q > 0.0f) {
      s += (double)q;
      c += 1.0;
    }
  }
  block_sum2(s, c);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = s;
    part[2 * blockIdx.x + 1] = c;
  }
}

}  // namespace emc

using namespace emc;

// ======================================================= C ABI ===========
extern "C" int emc_plan_create(emc_ctx* ctx, const emc_plan_desc* desc, emc_plan** out) {
  EMC_CHECK_CTX(ctx);
  EMC_REQUIRE(ctx, desc && out, "plan_create: null argument");
  *out = nullptr;
  const emc_plan_desc& d = *desc;
  EMC_REQUIRE(ctx, d.side > 1 && d.side <= 1024, "plan_create: side %d out of range", d.side);
  EMC_REQUIRE(ctx, d.n_images > 0 && d.n_rot > 0, "plan_create: empty problem");
  EMC_REQUIRE(ctx, d.n_rot <= 65535 * EMC_RT && (long long)d.n_rot * d.n_images < (1LL << 40),
              "plan_create: problem too large");
  EMC_REQUIRE(ctx, d.diff == EMC_DIFF_POISSON || d.diff == EMC_DIFF_TRUE_POISSON,
              "plan_create: diff %d not supported by the fused path", d.diff);
  EMC_REQUIRE(ctx, d.interp == EMC_INTERP_NEAREST || d.interp == EMC_INTERP_TRILINEAR,
              "plan_create: bad interp");
  EMC_REQUIRE(ctx, d.precision == EMC_PREC_FP32 || d.precision == EMC_PREC_MIXED,
              "plan_create: bad precision");
  EMC_REQUIRE(ctx,
              d.insert_mode == EMC_INSERT_ATOMIC || d.insert_mode == EMC_INSERT_DETERMINISTIC ||
                  d.insert_mode == EMC_INSERT_SORTED,
              "plan_create: bad insert mode");
  EMC_REQUIRE(ctx, d.blur_sigma >= 0.0f && std::isfinite(d.blur_sigma), "plan_create: bad blur");
  emc_plan* p = new emc_plan();
  p->ctx = ctx;
  p->d = d;
  p->n2 = d.side * d.side;
  p->Np = ceil_div(d.n_images, 128) * 128;  // whole 128-pattern tiles (and 64-pattern k-blocks)
  p->Rp = ceil_div(d.n_rot, 128) * 128;
  p->n_rt = ceil_div(d.n_rot, EMC_RT);
  const size_t RN = (size_t)d.n_rot * d.n_images;
  const size_t n3 = (size_t)d.side * d.side * d.side;
  int rc = EMC_OK;
  if (!rc) rc = alloc_n(p, &p->L, RN);
  if (!rc) rc = alloc_n(p, &p->PHI, RN);
  if (!rc) rc = alloc_n(p, &p->part, (size_t)p->n_rt * d.n_images);
  if (!rc) rc = alloc_n(p, &p->lse, d.n_images);
  if (!rc) rc = alloc_n(p, &p->lse2, d.n_images);
  if (!rc) rc = alloc_n(p, &p->lse_shifted, (size_t)8 * p->Np);
  if (!rc) rc = alloc_n(p, &p->ll_part, ceil_div(d.n_images, 32));
  if (!rc) {
    cudaError_t e = cudaFuncSetAttribute(mprep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(sizeof(float) * kMprepStageLo));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(mprep_hi_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(sizeof(float) * (kMprepChunkMax + 4)));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(mprep_hi_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(sizeof(float) * (kMprepChunkMax + 4)));
    if (e != cudaSuccess) rc = cuda_fail(ctx, e, "plan_create: mprep smem");
  }
  if (!rc) {
    cudaError_t e = cudaFuncSetAttribute(pattern_row_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, kRowSmemMax);
    if (e != cudaSuccess) rc = cuda_fail(ctx, e, "plan_create: pattern row smem");
  }
  if (!rc) rc = alloc_n(p, &p->T, p->Rp);
  if (!rc) rc = alloc_n(p, &p->rot_cnt, p->Rp);
  if (!rc) rc = alloc_n(p, &p->rot_A, p->Rp);
  if (!rc) rc = alloc_n(p, &p->rot_ssum, p->Rp);
  if (!rc) rc = alloc_n(p, &p->red, (size_t)kRedSlots + 2 * (size_t)p->Rp + 2 * 1024 + 2);
  if (!rc) rc = alloc_n(p, &p->cnorm, d.n_images);
  if (!rc) rc = alloc_n(p, &p->Ksum, d.n_images);
  if (!rc) rc = alloc_n(p, &p->flags, 16);
  if (!rc) rc = alloc_n(p, &p->sigma_dev, 1);
  if (!rc && d.blur_sigma > 0.0f) {
    const size_t n3b = (size_t)d.side * d.side * d.side;
    float *ba = nullptr, *bb = nullptr, *bg = nullptr;
    unsigned char* bk = nullptr;
    rc = alloc_n(p, &ba, n3b);
    if (!rc) rc = alloc_n(p, &bb, n3b);
    if (!rc) rc = alloc_n(p, &bg, (size_t)d.side);
    if (!rc) rc = plan_alloc(p, (void**)&bk, n3b);
    if (!rc) rc = blur_prepare(ctx, d.side, d.blur_sigma, ba, bb, bg, bk, &p->blur);
  }
  if (!rc) {
    cudaError_t e = cudaHostAlloc((void**)&p->report, sizeof(IterReport), cudaHostAllocDefault);
    if (e == cudaSuccess) e = cudaMemsetAsync(p->flags, 0, 16 * sizeof(int), ctx->stream);
    if (e != cudaSuccess) rc = cuda_fail(ctx, e, "plan_create");
  }
  if (!rc && d.precision == EMC_PREC_FP32) rc = alloc_n(p, &p->Q, (size_t)d.n_rot * p->Np);
  if (!rc && d.insert_mode == EMC_INSERT_DETERMINISTIC) {
    rc = alloc_n(p, &p->fix2, n3);
  }
  if (!rc && d.insert_mode != EMC_INSERT_DETERMINISTIC) rc = alloc_n(p, &p->acc2, n3);
  if (rc) {
    emc_plan_destroy(p);
    return rc;
  }
  *out = p;
  return EMC_OK;
}

extern "C" int emc_plan_destroy(emc_plan* p) {
  if (!p) return EMC_OK;
  if (p->ctx) cudaStreamSynchronize(p->ctx->stream);
  prune_free(p);
  sorted_free(p);
  if (p->graph_exec) cudaGraphExecDestroy(p->graph_exec);
  if (p->graph) cudaGraphDestroy(p->graph);
  for (auto& e : p->ev)
    if (e) cudaEventDestroy(e);
  if (p->tc) tc_free(p);
  for (void* a : p->allocs) cudaFree(a);
  if (p->report) cudaFreeHost(p->report);
  delete p;
  return EMC_OK;
}

extern "C" size_t emc_plan_workspace_bytes(const emc_plan* p) { return p ? p->bytes : 0; }

// The pattern-side operands (per-pattern factor, compacted counts, their
// sums, and the tensor-core forms once those exist) for the pattern order
// perm (device [N]: position -> input pattern; nullptr: input order).
int emc::pattern_side(emc_plan* p, const int* d_perm, bool with_tc) {
  emc_ctx* ctx = p->ctx;
  const int n2 = p->n2, N = p->d.n_images;
  int rc;
  pattern_norm_kernel<<<ceil_div(N, 128), 128, 0, ctx->stream>>>(
      p->images, p->mask, n2, N, p->d.normalize_images, p->cnorm, d_perm);
  if ((rc = after_launch(ctx, "pattern_norm_kernel"))) return rc;
  // Kt exists only for the FP32 path (null: not written).
  const int nqb = ceil_div(p->Kp, 256);
  // once the tensor-core operands exist, their FP16 counts come from the same
  // pass at the current scale (bind re-runs them if the new counts need
  // another scale)
  const bool fused = p->tc != nullptr && p->Kh != nullptr;
  p->fused_scale = fused ? p->count_scale : 0.0f;
  const size_t row_smem = pattern_row_smem(n2, p->Kp);
  if (row_smem <= (size_t)kRowSmemMax) {
    pattern_row_kernel<<<N, kRowThreads, row_smem, ctx->stream>>>(
        p->images, p->pix, p->cnorm, n2, N, p->Kp, p->Kraw, p->Kt, p->flags, d_perm,
        p->Ksum, fused ? p->Kh : nullptr, p->count_scale);
    if ((rc = after_launch(ctx, "pattern_row_kernel"))) return rc;
    if (with_tc && p->tc) return tc_pattern_side(p, d_perm, fused);
    return EMC_OK;
  }
  pattern_ops_kernel<<<(unsigned)N * (unsigned)nqb, 256, 0, ctx->stream>>>(
      p->images, p->pix, p->cnorm, n2, N, p->Kp, p->Kraw, p->Kt, p->flags, d_perm,
      p->ksum_part, fused ? p->Kh : nullptr, p->count_scale);
  if ((rc = after_launch(ctx, "pattern_ops_kernel"))) return rc;
  pattern_sums_kernel<<<ceil_div(N, 256), 256, 0, ctx->stream>>>(p->ksum_part, N, nqb, p->Ksum);
  if ((rc = after_launch(ctx, "pattern_sums_kernel"))) return rc;
  if (with_tc && p->tc) return tc_pattern_side(p, d_perm, fused);
  return EMC_OK;
}

extern "C" int emc_plan_bind(emc_plan* p, const float* d_images, const int* d_mask,
                             const float* d_x, const float* d_y, const float* d_z,
                             const float* d_rot, const float* d_rot_weights) {
  if (!p) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  EMC_REQUIRE(ctx, d_images && d_mask && d_x && d_y && d_z && d_rot && d_rot_weights,
              "plan_bind: null pointer");
  const int n2 = p->n2, N = p->d.n_images;
  const int prev_P = p->P_eff;
  // Mask -> compacted pixel list (host; once per plan).
  std::vector<int> hmask(n2);
  EMC_CUDA(ctx, cudaMemcpyAsync(hmask.data(), d_mask, sizeof(int) * n2, cudaMemcpyDeviceToHost,
                                ctx->stream));
  EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  // a re-bind with the same mask keeps the compacted pixel list
  const bool same_mask = prev_P != 0 && hmask == p->h_mask;
  std::vector<int> pix;
  if (same_mask) {
    pix = p->h_pix;
  } else {
    for (int q = 0; q < n2; ++q) {
      EMC_REQUIRE(ctx, hmask[q] == 0 || hmask[q] == 1, "plan_bind: mask values must be 0 or 1");
      if (hmask[q]) pix.push_back(q);
    }
    EMC_REQUIRE(ctx, !pix.empty(), "plan_bind: mask is empty");
    // Compacted pixels in one-pixel bands of detector radius, each band in
    // order of angle.  By radius: the bright low-q pixels, the only ones whose
    // k^2 needs a second FP16 term, share a few k-blocks of the tensor-core
    // E-step, and the dim outer blocks form the count tail where the H lo
    // term is dropped.  By angle within a band: the 32 pixels of a warp are
    // neighbours on the ring, so the expand's model gathers of a warp touch
    // neighbouring voxels.  (The order is otherwise free: every compacted
    // array uses it consistently.)
    const int side = p->d.side;
    std::vector<std::pair<long long, double>> key(n2);
    for (int q : pix) {
      const double dx = (double)(q % side) - side / 2 + 0.5, dy = (double)(q / side) - side / 2 + 0.5;
      key[q] = {(long long)std::floor(std::sqrt(dx * dx + dy * dy)), std::atan2(dy, dx)};
    }
    std::stable_sort(pix.begin(), pix.end(), [&](int a, int b) { return key[a] < key[b]; });
  }
  EMC_REQUIRE(ctx, prev_P == 0 || prev_P == (int)pix.size(),
              "plan_bind: a re-bind must keep the mask's pixel count (%d != %d)", (int)pix.size(),
              prev_P);
  p->bound = false;
  p->P_eff = (int)pix.size();
  p->Kp = ceil_div(p->P_eff, 128) * 128;  // whole 128-pixel M-step tiles
  pix.resize(p->Kp, -1);
  int rc = EMC_OK;
  if (prev_P == 0) {
  if (!rc) rc = alloc_n(p, &p->pix, p->Kp);
  if (!rc) rc = alloc_n(p, &p->cx, p->Kp);
  if (!rc) rc = alloc_n(p, &p->cy, p->Kp);
  if (!rc) rc = alloc_n(p, &p->cz, p->Kp);
  if (!rc) rc = alloc_n(p, &p->ksum_part, (size_t)N * ceil_div(p->Kp, 256));
  if (!rc && p->d.precision == EMC_PREC_FP32) rc = alloc_n(p, &p->Kraw, (size_t)N * p->Kp);
  if (!rc && p->d.precision == EMC_PREC_FP32) rc = alloc_n(p, &p->S, (size_t)p->Rp * p->Kp);
  if (!rc && p->d.precision == EMC_PREC_FP32) {
    rc = alloc_n(p, &p->Kt, (size_t)N * p->Kp);
  }
  // rows R..Rp of the slices stay zero: the expand writes rows < R only
  if (!rc && p->S) {
    const cudaError_t e =
        cudaMemsetAsync(p->S, 0, sizeof(float) * (size_t)p->Rp * p->Kp, ctx->stream);
    if (e != cudaSuccess) rc = cuda_fail(ctx, e, "plan_bind");
  }
  }
  if (rc) return rc;
  if (!same_mask) {
    p->h_mask = hmask;
    p->h_pix.assign(pix.begin(), pix.begin() + p->P_eff);
    // pageable source: staged before the call returns
    EMC_CUDA(ctx, cudaMemcpyAsync(p->pix, pix.data(), sizeof(int) * p->Kp,
                                  cudaMemcpyHostToDevice, ctx->stream));
  }
  EMC_CUDA(ctx, cudaMemsetAsync(p->flags, 0, 16 * sizeof(int), ctx->stream));
  gather_coords_kernel<<<ceil_div(p->Kp, 256), 256, 0, ctx->stream>>>(p->pix, d_x, d_y, d_z, p->cx,
                                                                      p->cy, p->cz, p->Kp);
  if ((rc = after_launch(ctx, "gather_coords_kernel"))) return rc;
  p->images = d_images;
  p->mask = d_mask;
  if ((rc = pattern_side(p, nullptr, false))) return rc;
  int hflags[16];
  EMC_CUDA(ctx, cudaMemcpyAsync(hflags, p->flags, sizeof(hflags), cudaMemcpyDeviceToHost, ctx->stream));
  EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (hflags[0] & 1) return fail(ctx, EMC_ERR_NONFINITE, "plan_bind: images contain NaN/Inf");
  p->counts_fp16_exact = !(hflags[0] & 2) && !(hflags[0] & 8);
  p->counts_integer = !(hflags[0] & 2);
  p->count_max = hflags[8];
  p->images = d_images;
  p->mask = d_mask;
  p->x = d_x;
  p->y = d_y;
  p->z = d_z;
  p->rot = d_rot;
  p->rotw = d_rot_weights;
  if (p->d.precision == EMC_PREC_MIXED) {
    if ((rc = tc_bind(p))) return rc;
  }
  // with pruning on, a new binding starts from the input pattern order, the
  // coherent order of its own rotations and a full scan
  if ((rc = prune_reset(p))) return rc;
  p->bound = true;
  // sorted insertion: the voxel map of this binding's rotations and pixels
  if ((rc = sorted_ensure(p))) {
    p->bound = false;
    return rc;
  }
  return EMC_OK;
}

template <int INTERP>
static int expand_launch(emc_plan* p, const float* model, const RotOps& ops) {
  emc_ctx* ctx = p->ctx;
  // the block size that leaves the fewest threads without pixels in the last turn
  // (64^3: 160 of 800 quads, 50 -> 42 us); with S_r summed always 256: the
  // true-Poisson likelihood holds K log S_r, and another order of that sum moves it by
  // more than all its other rounding
  const int n4 = p->Kp / 4;
  int threads = 256;
  for (int t = 224; t >= 128 && ops.live && !ops.Lh; t -= 32)
    if (ceil_div(n4, t) * t < ceil_div(n4, threads) * threads) threads = t;
  auto kernel = !ops.live    ? slice_rows_kernel<INTERP, kSliceFp32>
                : ops.Lh     ? slice_rows_kernel<INTERP, kSliceTcPois>
                : ops.bright ? (ops.MSl ? slice_rows_kernel<INTERP, kSliceTcBrightLo>
                                        : slice_rows_kernel<INTERP, kSliceTcBright>)
                : ops.MSl    ? slice_rows_kernel<INTERP, kSliceTcLo>
                             : slice_rows_kernel<INTERP, kSliceTc>;
  kernel<<<ceil_div(p->d.n_rot, slice_rows_per_block<INTERP>()), threads, 0, ctx->stream>>>(
      model, p->d.side, p->rot, p->pix, p->cx, p->cy, p->cz, p->d.n_rot, p->Kp, p->S, p->rot_cnt,
      p->rot_A, p->rot_ssum, ops);
  int rc = after_launch(ctx, "slice_rows_kernel");
  if (rc || !ops.tiny) return rc;
  tiny_plane_kernel<INTERP><<<dim3(p->n_rt, kTinyBlocks), 256, 0, ctx->stream>>>(
      model, p->d.side, p->rot, p->pix, p->cx, p->cy, p->cz, p->d.n_rot, p->Kp, ops.tiny, ops.nkb,
      tc_tiny_plane(p));
  return after_launch(ctx, "tiny_plane_kernel");
}

static int plan_expand(emc_plan* p, const float* model) {
  emc_ctx* ctx = p->ctx;
  const RotOps ops = tc_rot_ops(p);
  return p->d.interp == EMC_INTERP_NEAREST ? expand_launch<EMC_INTERP_NEAREST>(p, model, ops)
                                           : expand_launch<EMC_INTERP_TRILINEAR>(p, model, ops);
}

static int plan_estep_fp32(emc_plan* p) {
  emc_ctx* ctx = p->ctx;
  EstepArgs a;
  a.S = p->S;
  a.Kraw = p->Kraw;
  a.Kt = p->Kt;
  a.Ksum = p->Ksum;
  a.rot_cnt = p->rot_cnt;
  a.rot_ssum = p->rot_ssum;
  a.rotw = p->rotw;
  a.L = p->L;
  a.PHI = p->PHI;
  a.part = p->part;
  a.bad = p->flags + 4;
  a.R = p->d.n_rot;
  a.N = p->d.n_images;
  a.Kp = p->Kp;
  a.sigma = p->sigma_dev;
  a.known_intensity = p->d.known_intensity;
  dim3 grid(ceil_div(a.N, BN), ceil_div(a.R, BM));
  if (p->d.diff == EMC_DIFF_POISSON)
    estep_fp32_kernel<<<grid, TPB, 0, ctx->stream>>>(a);
  else
    estep_pois_fp32_kernel<<<grid, TPB, 0, ctx->stream>>>(a);
  return after_launch(ctx, "estep_fp32_kernel");
}

static InsertCtx make_insert_ctx(emc_plan* p, float* model, float* weight) {
  InsertCtx c;
  c.model = model;
  c.weight = weight;
  c.fix2 = p->fix2;
  c.acc2 = p->acc2;
  c.fix_scale = reinterpret_cast<const float2*>(p->red + kRedFixScale);
  c.u = p->d.insert_mode == EMC_INSERT_SORTED ? p->ins_u : nullptr;
  c.ldu = p->ins_ldu;
  c.side = p->d.side;
  c.interp = p->d.interp;
  c.deterministic = p->d.insert_mode == EMC_INSERT_DETERMINISTIC;
  return c;
}


static int plan_mstep_fp32(emc_plan* p, float* model, float* weight, const InsertCtx& ins) {
  emc_ctx* ctx = p->ctx;
  MstepArgs a;
  a.Q = p->Q;
  a.Kraw = p->Kraw;
  a.T = p->T;
  a.rot = p->rot;
  a.cx = p->cx;
  a.cy = p->cy;
  a.cz = p->cz;
  a.R = p->d.n_rot;
  a.N = p->d.n_images;
  a.Kp = p->Kp;
  a.ldq = p->Np;
  a.P_eff = p->P_eff;
  a.ins = ins;
  (void)model;
  (void)weight;
  dim3 grid(ceil_div(p->P_eff, BN), ceil_div(a.R, BM));
  mstep_fp32_kernel<<<grid, TPB, 0, ctx->stream>>>(a);
  return after_launch(ctx, "mstep_fp32_kernel");
}

// The stages of one iteration, each enqueued on the context stream: kernels,
// device-to-device copies and memsets only (no allocation, no host copy, no
// synchronisation), so the sequence can be captured in a CUDA graph.  The
// E-step reads sigma from p->sigma_dev.  A full iteration runs them in order;
// one rank of a rotation split (emc_rank_*) runs the E-step, exports its
// per-pattern partials, and resumes at the M-step with the global normaliser.
static int enqueue_normalise(emc_plan* p, float* d_model, int nb);

// Blocks of a pass over the model that leaves mean partials behind, and where
// they go (the reduction buffer's tail).
static int mean_blocks(const emc_plan* p, long long n) {
  return (int)std::min<long long>(ceil_div(n, 1024), std::min(kMeanBlocks, p->ctx->sm_count * 4));
}
static double* mean_parts(const emc_plan* p) { return p->red + kRedSlots + 2 * (size_t)p->Rp + 2; }

static int mark_phase(emc_plan* p, int i) {
  emc_ctx* ctx = p->ctx;
  if (p->profiling) EMC_CUDA(ctx, cudaEventRecord(p->ev[i], ctx->stream));
  return EMC_OK;
}

// expand + scaling + likelihood + per-tile (max, sum exp) partials
static int enqueue_estep(emc_plan* p, float* d_model) {
  emc_ctx* ctx = p->ctx;
  const int N = p->d.n_images;
  int rc;
  if ((rc = mark_phase(p, 0))) return rc;
  if (p->prune_tiles) {  // skipped tiles contribute (max, sum exp) = (-inf, 0)
    fill_part_kernel<<<ctx->sm_count * 4, 256, 0, ctx->stream>>>(p->part,
                                                                (size_t)p->n_rt * N);
    if ((rc = after_launch(ctx, "fill_part_kernel"))) return rc;
  }
  if ((rc = plan_expand(p, d_model))) return rc;
  if ((rc = mark_phase(p, 1))) return rc;
  if (p->d.precision == EMC_PREC_MIXED)
    rc = tc_estep(p);
  else
    rc = plan_estep_fp32(p);
  if (rc) return rc;
  return mark_phase(p, 2);
}

static LseOut lse_out(emc_plan* p) { return {p->lse, p->lse2, p->lse_shifted, p->Np}; }

// The terms of the total log-likelihood that plan_wait adds: the partials of
// lse_combine_kernel (or, after a rank's M-step, every pattern's lse).
static void own_loglik(emc_plan* p) {
  p->ll_src = p->ll_part;
  p->ll_n = ceil_div(p->d.n_images, 32);
}

// the normaliser lse_i from the per-tile partials, and the terms of the total
// log-likelihood
static int enqueue_lse(emc_plan* p) {
  emc_ctx* ctx = p->ctx;
  const int N = p->d.n_images;
  int rc;
  const int nb = ceil_div(N, 32);
  lse_combine_kernel<<<nb, 32 * kLseWarps, 0, ctx->stream>>>(p->part, p->n_rt, N, lse_out(p),
                                                             p->ll_part);
  if ((rc = after_launch(ctx, "lse_combine_kernel"))) return rc;
  own_loglik(p);
  return mark_phase(p, 3);
}

// Rows of mprep_hi_kernel: the fewest CTAs that keep `chunk` at kMprepChunk.
static int launch_mprep_hi(emc_plan* p, MprepArgs a) {
  emc_ctx* ctx = p->ctx;
  const int N = p->d.n_images;
  int ctas = 1;
  while (ctas < 8 && N > ctas * kMprepChunk) ctas *= 2;
  for (;; ctas = 1) {
    a.chunk = ceil_div(ceil_div(N, ctas), 128) * 128;
    a.stage = a.chunk <= kMprepChunkMax;
    // a thread for eight pairs of a short row
    const int threads = a.chunk <= 1024 ? 128 : a.chunk <= kMprepChunk ? 256 : 512;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p->d.n_rot * (unsigned)ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = a.stage ? sizeof(float) * (a.chunk + 4) : 0;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const bool plain = !a.Ksum && !a.cnorm && !a.tstate && !a.write_p;
    const cudaError_t e =
        cudaLaunchKernelEx(&cfg, plain ? mprep_hi_kernel<true> : mprep_hi_kernel<false>, a);
    if (e == cudaSuccess) break;
    if (ctas == 1) return cuda_fail(ctx, e, "mprep_hi_kernel launch");
    (void)cudaGetLastError();  // a device that cannot co-schedule the cluster
  }
  return after_launch(ctx, "mprep_hi_kernel");
}

// responsibilities (mprep) and the M-step with insertion into the zeroed
// accumulators (acc2, or fix2 when deterministic); model / weight
// are the buffers the insertion context names (not written here)
static int enqueue_mstep(emc_plan* p, float* d_model, float* d_weight) {
  emc_ctx* ctx = p->ctx;
  const int R = p->d.n_rot, N = p->d.n_images;
  const long long n3 = (long long)p->d.side * p->d.side * p->d.side;
  int rc;
  double* row_mass = p->red + kRedSlots;
  double* row_bound = row_mass + p->Rp;
  const bool tcm = p->d.precision == EMC_PREC_MIXED;
  const bool hi_only = tcm && !p->mstep_q_lo;
  const int stage = tcm && N <= (hi_only ? 8 * kMprepChunkMax : kMprepStageLo);
  // P is written over L only where it is read back: by the pruning of the
  // next iteration, or by mprep_kernel's own second pass when the row of Q does
  // not fit shared memory.  Otherwise the responsibilities are formed on request
  // (emc_plan_results, emc_plan_best_quaternions: plan_respons_ready).
  const int write_p = (p->prune != nullptr || (tcm && !hi_only && !stage)) ? 1 : 0;
  MprepArgs ma;
  ma.L = p->L;
  ma.PHI = p->PHI;
  ma.lse2 = p->lse2;
  ma.lse_shifted = p->lse_shifted;
  ma.Ksum = p->d.insert_mode == EMC_INSERT_DETERMINISTIC ? p->Ksum : nullptr;
  ma.cnorm = p->d.normalize_images ? p->cnorm : nullptr;
  ma.N = N;
  ma.ldq = p->Np;
  ma.n_rt = p->n_rt;
  ma.Q = tcm ? nullptr : p->Q;
  ma.Qh = tcm ? p->Qh : nullptr;
  ma.Ql = tcm && p->mstep_q_lo ? p->Ql : nullptr;
  ma.qscale = p->qscale;
  ma.T = p->T;
  ma.row_mass = row_mass;
  ma.row_bound = row_bound;
  ma.row_margin = p->prune_margin;
  ma.tstate = p->prune_tiles ? p->prune_state : nullptr;
  ma.stage = stage;
  ma.write_p = write_p;
  if (hi_only) {
    if ((rc = launch_mprep_hi(p, ma))) return rc;
  } else {
    mprep_kernel<<<R, 512, stage ? sizeof(float) * N : 0, ctx->stream>>>(ma);
  }
  p->p_written = write_p != 0;
  if ((rc = after_launch(ctx, "mprep_kernel"))) return rc;
  if ((rc = mark_phase(p, 4))) return rc;
  const bool det = p->d.insert_mode == EMC_INSERT_DETERMINISTIC;
  if (det) {
    insert_bounds_kernel<<<1, 256, 0, ctx->stream>>>(
        row_mass, row_bound, R, p->P_eff, p->red + kRedBoundM,
        reinterpret_cast<float2*>(p->red + kRedFixScale));
    if ((rc = after_launch(ctx, "insert_bounds_kernel"))) return rc;
    EMC_CUDA(ctx, cudaMemsetAsync(p->fix2, 0, sizeof(ulonglong2) * n3, ctx->stream));
  } else if (p->d.insert_mode == EMC_INSERT_ATOMIC) {
    EMC_CUDA(ctx, cudaMemsetAsync(p->acc2, 0, sizeof(float2) * n3, ctx->stream));
  }  // sorted: the reduction writes every voxel of acc2
  InsertCtx ins = make_insert_ctx(p, d_model, d_weight);
  if (tcm)
    rc = tc_mstep(p, d_model, d_weight);
  else
    rc = plan_mstep_fp32(p, d_model, d_weight, ins);
  if (!rc && p->d.insert_mode == EMC_INSERT_SORTED) rc = sorted_reduce(p);
  return rc;
}

// model = inserted sums / weight, normalised to a positive mean of 1, blurred
static int enqueue_finish(emc_plan* p, float* d_model, float* d_weight) {
  emc_ctx* ctx = p->ctx;
  const long long n3 = (long long)p->d.side * p->d.side * p->d.side;
  const bool det = p->d.insert_mode == EMC_INSERT_DETERMINISTIC;
  int rc;
  const int nb = mean_blocks(p, n3);
  finish_insert_kernel<<<nb, 256, 0, ctx->stream>>>(
      det ? p->fix2 : nullptr, reinterpret_cast<const float2*>(p->red + kRedFixScale),
      p->acc2, d_model, d_weight, n3, mean_parts(p));
  if ((rc = after_launch(ctx, "finish_insert_kernel"))) return rc;
  if ((rc = mark_phase(p, 5))) return rc;
  return enqueue_normalise(p, d_model, nb);
}

// model / positive mean (the reference's normalize_model) from the nb mean
// partials of the pass that formed the model, then the blur
static int enqueue_normalise(emc_plan* p, float* d_model, int nb) {
  emc_ctx* ctx = p->ctx;
  const long long n3 = (long long)p->d.side * p->d.side * p->d.side;
  int rc;
  if ((rc = launch_scale_by_partials(ctx, d_model, n3, mean_parts(p), nb, p->red + kRedMean)))
    return rc;
  if (p->d.blur_sigma > 0.0f) {
    if ((rc = blur_run(ctx, d_model, p->blur))) return rc;
  }
  return mark_phase(p, 6);
}

static int iterate_enqueue(emc_plan* p, float* d_model, float* d_weight) {
  int rc;
  if ((rc = enqueue_estep(p, d_model))) return rc;
  if ((rc = enqueue_lse(p))) return rc;
  if ((rc = enqueue_mstep(p, d_model, d_weight))) return rc;
  return enqueue_finish(p, d_model, d_weight);
}

// Start of an iteration, before its graph or its first kernel: the annealing width,
// and zeros in the invalid-pair counter and the expand's block flags.  The width is
// written by a kernel rather than a host-to-device copy: a copy would queue on the
// copy engine behind any bulk host copy that another stream has issued (the next
// patterns, uploaded while this iteration runs) and hold the iteration back until
// that copy ends.
__global__ void begin_kernel(float* __restrict__ sigma, float v, int* __restrict__ bad,
                             uint4* __restrict__ flags, int n16) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e == 0) {
    *sigma = v;
    *bad = 0;
  }
  if (e < n16) flags[e] = make_uint4(0, 0, 0, 0);
}

static int begin_iteration(emc_plan* p, float sigma, cudaStream_t stream) {
  const size_t bytes = p->rot_flags ? 2 * (size_t)p->n_rt * (p->Kp / 64) : 0;
  const int n16 = (int)((bytes + 15) / 16);  // rot_flags is allocated in whole 16 bytes
  begin_kernel<<<std::max(1, ceil_div(n16, 256)), 256, 0, stream>>>(
      p->sigma_dev, sigma, p->flags + 4, reinterpret_cast<uint4*>(p->rot_flags), n16);
  return after_launch(p->ctx, "begin_kernel");
}

static int set_sigma(emc_plan* p, float sigma) {
  emc_ctx* ctx = p->ctx;
  EMC_REQUIRE(ctx, sigma > 0.0f && std::isfinite(sigma), "iterate: bad sigma");
  return begin_iteration(p, sigma, ctx->stream);
}

extern "C" int emc_iterate_async(emc_plan* p, float* d_model, float* d_weight, float sigma) {
  if (!p) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  EMC_REQUIRE(ctx, p->bound, "iterate: plan not bound");
  EMC_REQUIRE(ctx, d_model && d_weight, "iterate: null model/weight");
  int rc = set_sigma(p, sigma);
  if (rc) return rc;
  return iterate_enqueue(p, d_model, d_weight);
}

// What plan_wait reads, in one launch and one write to host memory.
__global__ void __launch_bounds__(1024) report_kernel(const int* __restrict__ flags,
                                                      const int* __restrict__ status,
                                                      const double* __restrict__ red,
                                                      const double* __restrict__ row_mass,
                                                      const double* __restrict__ margin, int R,
                                                      const double* __restrict__ ll, int n_ll,
                                                      IterReport* __restrict__ out) {
  double m = 0.0, g = 0.0;
  for (int r = threadIdx.x; r < R; r += blockDim.x) {
    m += row_mass[r];
    if (margin) g += margin[r];
  }
  block_sum2(m, g);
  double l = 0.0, none = 0.0;  // the finite entries
  for (int i = threadIdx.x; i < n_ll; i += blockDim.x)
    if (isfinite(ll[i])) l += ll[i];
  __syncthreads();
  block_sum2(l, none);
  if (threadIdx.x == 0) {
    out->mass = m;
    out->margin = g;
    out->loglik = l;
    out->status = status ? *status : 0;
  }
  if (threadIdx.x < 8) out->flags[threadIdx.x] = flags[threadIdx.x];
  if (threadIdx.x < kRedSlots) out->red[threadIdx.x] = red[threadIdx.x];
  __threadfence_system();
}

// Synchronises, then reports what the device recorded since the last wait:
// a pipeline wait that timed out, slice values outside the FP16 operand
// range; fills stats (of the last iteration) and clears the status words.
// margin: per-rotation masses whose sum goes to *margin_sum (may both be null).
int emc::plan_wait(emc_plan* p, emc_iter_stats* stats, const double* margin, double* margin_sum) {
  emc_ctx* ctx = p->ctx;
  int* dtc = tc_status(p);
  report_kernel<<<1, 1024, 0, ctx->stream>>>(p->flags, dtc, p->red, p->red + kRedSlots, margin,
                                             stats || margin ? p->d.n_rot : 0, p->ll_src,
                                             stats ? p->ll_n : 0, p->report);
  const int rc = after_launch(ctx, "report_kernel");
  if (rc) return rc;
  EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const IterReport h = *p->report;
  if (h.status) EMC_CUDA(ctx, cudaMemsetAsync(dtc, 0, sizeof(int), ctx->stream));
  if (h.flags[0] & 4) EMC_CUDA(ctx, cudaMemsetAsync(p->flags, 0, sizeof(int), ctx->stream));
  if (h.status)
    return fail(ctx, EMC_ERR_TIMEOUT, "iterate: tensor-core pipeline wait timed out (status 0x%x)",
                h.status);
  if (h.flags[0] & 4)
    return fail(ctx, EMC_ERR_UNSUPPORTED, "iterate: slice values exceed the FP16 operand range");
  if (stats) {
    stats->total_loglik = h.loglik;
    stats->model_mean_before = h.red[kRedMean + 1] > 0 ? h.red[kRedMean] / h.red[kRedMean + 1] : 0.0;
    stats->captured_mass = h.mass / (double)p->d.n_images;
    stats->bad_pairs = h.flags[4];
    stats->reserved = 0;
  }
  if (margin_sum) *margin_sum = h.margin;
  return EMC_OK;
}

extern "C" int emc_plan_wait(emc_plan* p, emc_iter_stats* stats) {
  return p ? plan_wait(p, stats, nullptr, nullptr) : EMC_ERR_INVALID;
}

extern "C" int emc_iterate(emc_plan* p, float* d_model, float* d_weight, float sigma,
                           emc_iter_stats* stats) {
  if (p && p->prune) {
    bool handled = false;
    const int prc = prune_iterate(p, d_model, d_weight, sigma, stats, &handled);
    if (handled || prc) return prc;
  }
  int rc = emc_iterate_async(p, d_model, d_weight, sigma);
  if (rc) return rc;
  return emc_plan_wait(p, stats);
}

extern "C" int emc_plan_capture(emc_plan* p, float* d_model, float* d_weight) {
  if (!p) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  EMC_REQUIRE(ctx, p->bound, "plan_capture: plan not bound");
  EMC_REQUIRE(ctx, d_model && d_weight, "plan_capture: null model/weight");
  EMC_REQUIRE(ctx, ctx->stream != nullptr,
              "plan_capture: the legacy default stream cannot be captured; use emc_set_stream");
  if (p->graph_exec) {
    EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    cudaGraphExecDestroy(p->graph_exec);
    p->graph_exec = nullptr;
  }
  if (p->graph) {
    cudaGraphDestroy(p->graph);
    p->graph = nullptr;
  }
  const bool prof = p->profiling;
  EMC_CUDA(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
  p->profiling = false;  // no event records inside the graph
  // recording runs nothing: what the last iteration left stays described as it was
  const bool p_written = p->p_written;
  const double* const ll_src = p->ll_src;
  const int ll_n = p->ll_n;
  const int rc = iterate_enqueue(p, d_model, d_weight);
  const bool graph_p_written = p->p_written;
  p->p_written = p_written;
  p->ll_src = ll_src;
  p->ll_n = ll_n;
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(ctx->stream, &g);
  p->profiling = prof;
  if (rc) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  if (e != cudaSuccess) return cuda_fail(ctx, e, "plan_capture: end capture");
  const cudaError_t ei = cudaGraphInstantiate(&p->graph_exec, g, 0);
  if (ei != cudaSuccess) {
    cudaGraphDestroy(g);
    return cuda_fail(ctx, ei, "plan_capture: instantiate");
  }
  p->graph = g;
  p->graph_p_written = graph_p_written;
  return EMC_OK;
}

extern "C" int emc_plan_replay(emc_plan* p, float sigma) {
  if (!p) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  EMC_REQUIRE(ctx, p->graph_exec, "plan_replay: no captured iteration");
  int rc = set_sigma(p, sigma);
  if (rc) return rc;
  EMC_CUDA(ctx, cudaGraphLaunch(p->graph_exec, ctx->stream));
  own_loglik(p);
  p->p_written = p->graph_p_written;
  return EMC_OK;
}

// ---------------------------------------------------------------- batch --
// Several independent reconstructions in one graph launch: each plan's
// captured iteration becomes a child graph of one parent graph with no edges
// between them, so the GPU runs them concurrently.
struct emc_batch {
  std::vector<emc_plan*> plans;
  std::vector<bool> p_written;  // each plan's, after a run
  emc_ctx* ctx = nullptr;  // stream of the launches (the first plan's context)
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

extern "C" int emc_batch_create(emc_plan** plans, float** d_models, float** d_weights, int n,
                                emc_batch** out) {
  if (!plans || !d_models || !d_weights || n <= 0 || !out || !plans[0]) return EMC_ERR_INVALID;
  emc_ctx* ctx = plans[0]->ctx;
  for (int k = 0; k < n; ++k) {
    EMC_REQUIRE(ctx, plans[k] && d_models[k] && d_weights[k], "batch_create: null entry %d", k);
    EMC_REQUIRE(ctx, plans[k]->ctx->device == ctx->device, "batch_create: plans on two devices");
    const int rc = emc_plan_capture(plans[k], d_models[k], d_weights[k]);
    if (rc) return fail(ctx, rc, "batch_create: plan %d: %s", k, emc_last_error(plans[k]->ctx));
  }
  emc_batch* b = new emc_batch();
  b->plans.assign(plans, plans + n);
  for (emc_plan* p : b->plans) b->p_written.push_back(p->graph_p_written);
  b->ctx = ctx;
  cudaError_t e = cudaGraphCreate(&b->graph, 0);
  for (int k = 0; k < n && e == cudaSuccess; ++k) {
    cudaGraphNode_t node;
    e = cudaGraphAddChildGraphNode(&node, b->graph, nullptr, 0, plans[k]->graph);
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&b->exec, b->graph, 0);
  if (e != cudaSuccess) {
    emc_batch_destroy(b);
    return cuda_fail(ctx, e, "batch_create");
  }
  *out = b;
  return EMC_OK;
}

extern "C" int emc_batch_run(emc_batch* b, const float* sigmas) {
  if (!b || !sigmas) return EMC_ERR_INVALID;
  emc_ctx* ctx = b->ctx;
  for (size_t k = 0; k < b->plans.size(); ++k) {
    const float sg = sigmas[k];
    EMC_REQUIRE(ctx, sg > 0.0f && std::isfinite(sg), "batch_run: bad sigma %zu", k);
    const int rc = begin_iteration(b->plans[k], sg, ctx->stream);
    if (rc) return rc;
  }
  EMC_CUDA(ctx, cudaGraphLaunch(b->exec, ctx->stream));
  for (size_t k = 0; k < b->plans.size(); ++k) {
    own_loglik(b->plans[k]);
    b->plans[k]->p_written = b->p_written[k];
  }
  return EMC_OK;
}

extern "C" int emc_batch_wait(emc_batch* b, emc_iter_stats* stats) {
  if (!b) return EMC_ERR_INVALID;
  emc_ctx* ctx = b->ctx;
  EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  int first = EMC_OK;
  for (size_t k = 0; k < b->plans.size(); ++k) {
    emc_plan* p = b->plans[k];
    const int rc = emc_plan_wait(p, stats ? stats + k : nullptr);
    if (rc && !first) first = fail(ctx, rc, "batch: plan %zu: %s", k, emc_last_error(p->ctx));
    // the status resets of emc_plan_wait run on the plan's own stream
    cudaStreamSynchronize(p->ctx->stream);
  }
  return first;
}

extern "C" int emc_batch_destroy(emc_batch* b) {
  if (!b) return EMC_OK;
  if (b->ctx) cudaStreamSynchronize(b->ctx->stream);
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  delete b;
  return EMC_OK;
}

extern "C" int emc_plan_get_option(const emc_plan* p, int option, int* value) {
  if (!p || !value) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  switch (option) {
    case EMC_OPT_MSTEP_QLO: *value = p->mstep_q_lo; return EMC_OK;
    case EMC_OPT_ESTEP_GHLO: *value = p->estep_gh_lo; return EMC_OK;
    case EMC_OPT_MSTEP_AGGREGATE: *value = p->mstep_aggregate; return EMC_OK;
    case EMC_OPT_COUNTS_ROUND: *value = p->counts_round; return EMC_OK;
    case EMC_OPT_ESTEP_RASTER: *value = p->estep_raster; return EMC_OK;
    case EMC_OPT_ESTEP_PAIR: *value = p->estep_pair; return EMC_OK;
    case EMC_OPT_MSTEP_RASTER: *value = p->mstep_raster; return EMC_OK;
    case EMC_OPT_DEBUG_SPIN: *value = (int)p->debug_spin; return EMC_OK;
    case EMC_OPT_MSTEP_PAIR: *value = p->mstep_pair; return EMC_OK;
    case EMC_OPT_GLO_TAIL: *value = p->glo_tail_ppm; return EMC_OK;
    case EMC_OPT_HLO_TAIL: *value = p->hlo_tail_ppm; return EMC_OK;
    default: return fail(ctx, EMC_ERR_INVALID, "plan_get_option: unknown option %d", option);
  }
}

extern "C" int emc_plan_set_option(emc_plan* p, int option, int value) {
  if (!p) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  if (option == EMC_OPT_ESTEP_GHLO) {
    EMC_REQUIRE(ctx, value >= -1 && value <= 3, "plan_set_option: gh_lo %d", value);
    p->estep_gh_lo = value;
    return tc_ensure_mslo(p);
  }
  if (option == EMC_OPT_ESTEP_RASTER) {
    EMC_REQUIRE(ctx, value != 0 && value >= -4096 && value <= 4096,
                "plan_set_option: raster %d", value);
    p->estep_raster = value;
    return EMC_OK;
  }
  if (option == EMC_OPT_MSTEP_RASTER) {
    EMC_REQUIRE(ctx, value != 0 && value >= -4096 && value <= 4096,
                "plan_set_option: M-step raster %d", value);
    p->mstep_raster = value;
    return EMC_OK;
  }
  if (option == EMC_OPT_ESTEP_PAIR) {
    EMC_REQUIRE(ctx, value == 0 || value == 1, "plan_set_option: pair %d", value);
    p->estep_pair = value;
    return EMC_OK;
  }
  if (option == EMC_OPT_MSTEP_PAIR) {
    EMC_REQUIRE(ctx, value == 0 || value == 1, "plan_set_option: M-step pair %d", value);
    p->mstep_pair = value;
    return EMC_OK;
  }
  if (option == EMC_OPT_DEBUG_SPIN) {
    EMC_REQUIRE(ctx, value >= 0, "plan_set_option: debug spin %d", value);
    p->debug_spin = (unsigned)value;
    return EMC_OK;
  }
  if (option == EMC_OPT_MSTEP_AGGREGATE) {
    EMC_REQUIRE(ctx, value == 0 || value == 1, "plan_set_option: aggregate %d", value);
    p->mstep_aggregate = value;
    return EMC_OK;
  }
  if (option == EMC_OPT_COUNTS_ROUND) {
    EMC_REQUIRE(ctx, value == 0 || value == 1, "plan_set_option: counts_round %d", value);
    EMC_REQUIRE(ctx, !p->tc, "plan_set_option: set EMC_OPT_COUNTS_ROUND before bind");
    p->counts_round = value;
    return EMC_OK;
  }
  if (option == EMC_OPT_GLO_TAIL || option == EMC_OPT_HLO_TAIL) {
    EMC_REQUIRE(ctx, value >= 0 && value <= 1000000, "plan_set_option: lo tail %d", value);
    p->hlo_tail_ppm = value;
    if (option == EMC_OPT_GLO_TAIL) p->glo_tail_ppm = value;
    return p->tc ? tc_block_lists(p) : EMC_OK;
  }
  if (option == EMC_OPT_MSTEP_QLO) {
    EMC_REQUIRE(ctx, value == 0 || value == 1, "plan_set_option: q_lo %d", value);
    p->mstep_q_lo = value;
    return value ? tc_ensure_qlo(p) : EMC_OK;
  }
  return fail(ctx, EMC_ERR_INVALID, "plan_set_option: unknown option %d", option);
}

extern "C" int emc_plan_autotune(emc_plan* p, const float* d_model, float sigma, int* h_raster,
                                 float* h_ms) {
  if (!p) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  EMC_REQUIRE(ctx, p->bound, "autotune: plan not bound");
  EMC_REQUIRE(ctx, d_model, "autotune: null model");
  if (p->d.precision != EMC_PREC_MIXED) {  // the FP32 path has no tile order to tune
    if (h_raster) *h_raster = 0;
    if (h_ms) *h_ms = 0.0f;
    return EMC_OK;
  }
  int rc = set_sigma(p, sigma);
  if (!rc) rc = plan_expand(p, d_model);
  if (!rc) rc = tc_autotune(p, 256, h_raster, h_ms);
  // the timed launches count non-finite pairs of partial grids: not an iteration's
  if (!rc) EMC_CUDA(ctx, cudaMemsetAsync(p->flags + 4, 0, sizeof(int), ctx->stream));
  if (!rc) EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return rc;
}

extern "C" int emc_plan_time_likelihood(emc_plan* p, const float* d_model, float sigma,
                                        int raster, int first_tile, int n_tiles, float* h_ms,
                                        int* h_total_tiles) {
  if (!p) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  EMC_REQUIRE(ctx, p->bound, "time_likelihood: plan not bound");
  EMC_REQUIRE(ctx, p->d.precision == EMC_PREC_MIXED, "time_likelihood: tensor-core plans only");
  EMC_REQUIRE(ctx, raster != 0 && raster >= -4096 && raster <= 4096 && first_tile >= 0 &&
                       n_tiles > 0 && h_ms, "time_likelihood: bad arguments");
  int rc = EMC_OK;
  if (d_model) {
    rc = set_sigma(p, sigma);
    if (!rc) rc = plan_expand(p, d_model);
  }
  if (!rc) rc = tc_time_estep(p, raster, first_tile, n_tiles, h_ms);
  if (!rc && h_total_tiles) *h_total_tiles = tc_estep_tiles(p);
  if (!rc) EMC_CUDA(ctx, cudaMemsetAsync(p->flags + 4, 0, sizeof(int), ctx->stream));
  return rc;
}

extern "C" int emc_plan_set_profiling(emc_plan* p, int on) {
  if (!p) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  if (on && !p->ev[0]) {
    for (auto& e : p->ev) EMC_CUDA(ctx, cudaEventCreate(&e));
  }
  p->profiling = on != 0;
  return EMC_OK;
}

extern "C" int emc_plan_phase_ms(emc_plan* p, float* ms, int n) {
  if (!p || !ms || n < 0) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  EMC_REQUIRE(ctx, p->profiling, "plan_phase_ms: profiling is off");
  EMC_CUDA(ctx, cudaEventSynchronize(p->ev[emc_plan::kPhases]));
  for (int i = 0; i < n && i < emc_plan::kPhases; ++i)
    EMC_CUDA(ctx, cudaEventElapsedTime(ms + i, p->ev[i], p->ev[i + 1]));
  return EMC_OK;
}

extern "C" int emc_plan_results(emc_plan* p, const float** d_respons, const float** d_scaling,
                                const double** d_lse) {
  if (!p) return EMC_ERR_INVALID;
  if (d_respons) {
    const int rc = plan_respons_ready(p);
    if (rc) return rc;
  }
  if (d_respons) *d_respons = p->L;
  if (d_scaling) *d_scaling = p->PHI;
  if (d_lse) *d_lse = p->lse;
  return EMC_OK;
}

// ---- one rank of the reference's rotation split (main.cpp:141-154) -------
extern "C" int emc_rank_estep(emc_plan* p, float* d_model, float sigma, float* d_max,
                              double* d_sumexp) {
  if (!p) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  EMC_REQUIRE(ctx, p->bound, "rank_estep: plan not bound");
  EMC_REQUIRE(ctx, d_model && d_max && d_sumexp, "rank_estep: null argument");
  EMC_REQUIRE(ctx, !p->prune, "rank_estep: pruning is not supported on a rotation split");
  int rc = set_sigma(p, sigma);
  if (rc) return rc;
  if ((rc = enqueue_estep(p, d_model))) return rc;
  const int N = p->d.n_images;
  rank_partial_kernel<<<ceil_div(N, 32), 32 * kLseWarps, 0, ctx->stream>>>(p->part, p->n_rt, N,
                                                                          d_max, d_sumexp);
  return after_launch(ctx, "rank_partial_kernel");
}

extern "C" int emc_rank_mstep(emc_plan* p, const double* d_lse, float* d_model_sum,
                              float* d_weight_sum) {
  if (!p) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  EMC_REQUIRE(ctx, p->bound, "rank_mstep: plan not bound");
  EMC_REQUIRE(ctx, d_lse && d_model_sum && d_weight_sum, "rank_mstep: null argument");
  EMC_REQUIRE(ctx, !p->prune, "rank_mstep: pruning is not supported on a rotation split");
  const int N = p->d.n_images;
  const long long n3 = (long long)p->d.side * p->d.side * p->d.side;
  lse_from_global_kernel<<<ceil_div(N, 256), 256, 0, ctx->stream>>>(d_lse, N, lse_out(p));
  int rc = after_launch(ctx, "lse_from_global_kernel");
  if (rc) return rc;
  p->ll_src = p->lse;
  p->ll_n = N;
  if ((rc = mark_phase(p, 3))) return rc;
  if ((rc = enqueue_mstep(p, d_model_sum, d_weight_sum))) return rc;
  const bool det = p->d.insert_mode == EMC_INSERT_DETERMINISTIC;
  const int nb = (int)std::min<long long>(ceil_div(n3, 256), (long long)ctx->sm_count * 8);
  sums_out_kernel<<<nb, 256, 0, ctx->stream>>>(det ? p->fix2 : nullptr,
                                                reinterpret_cast<const float2*>(p->red + kRedFixScale),
                                                p->acc2, d_model_sum,
                                                d_weight_sum, n3);
  return after_launch(ctx, "sums_out_kernel");
}

extern "C" int emc_model_from_sums(emc_plan* p, const float* d_model_sum,
                                   const float* d_weight_sum, int n_ranks, float* d_model,
                                   float* d_weight) {
  if (!p) return EMC_ERR_INVALID;
  emc_ctx* ctx = p->ctx;
  EMC_REQUIRE(ctx, d_model_sum && d_weight_sum && d_model && d_weight && n_ranks >= 1,
              "model_from_sums: bad argument");
  const long long n3 = (long long)p->d.side * p->d.side * p->d.side;
  const int nb = mean_blocks(p, n3);
  model_from_sums_kernel<<<nb, 256, 0, ctx->stream>>>(d_model_sum, d_weight_sum, (float)n_ranks,
                                                       d_model, d_weight, n3, mean_parts(p));
  int rc = after_launch(ctx, "model_from_sums_kernel");
  if (rc) return rc;
  if ((rc = mark_phase(p, 5))) return rc;
  return enqueue_normalise(p, d_model, nb);
}
