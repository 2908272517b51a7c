// Scaling (row A5) and likelihood (row A6) with the reference's arithmetic.
//
// Reference: update_scaling_full_kernel + calculate_scaling_absolute
// (emc_cuda.cu:438-454, 516-539) and calculate_responsabilities_kernel with
// its per-diff device functions (emc_cuda.cu:159-295).  The reference runs one
// 512-thread block per (image, rotation) pair.  Its result depends on the
// order of the float additions: thread t sums pixels t, t+512, ... and the 512
// partials are then folded by a halving tree.  These kernels keep exactly that
// per-pair order (so the host oracle can check them to the last bit where no
// transcendental function is involved) but give each block a few images and
// four rotations, so that what depends on one side only is loaded, or computed,
// once for all of them.  They are the drop-in (quirk-exact) path; the fused
// iteration uses the tiled kernels of the plan instead.
//
// Quirks kept on purpose:
//  * the scaling denominator accumulates in an int: every partial add is
//    truncated toward zero (emc_cuda.cu:439, 446);
//  * the scaling masks compare against the double literal 1e-10;
//  * the POISSON term is evaluated in FP64 per pixel (double literal 0.02,
//    emc_cuda.cu:205) and rounded into a float running sum;
//  * count == 0 or den == 0 give the reference's NaN / Inf.
//
// What bounds them: FP32 issue.  FP64, conversions and divisions per pair and
// pixel (an FP64 square root and division, an FP32 division, two int/float
// conversions) took 59 ms for the likelihood and 2.9 ms for the scaling of 2,000
// patterns x 180 rotations of 64 x 64; the forms below give the same roundings
// from FP32 multiply-adds.
#include <algorithm>

#include "common.cuh"

namespace emc {

constexpr int kVT = 512;       // virtual threads per pair (the reference's TNUM)
constexpr int kRotPerCta = 4;  // rotations of a block
constexpr int kImgScal = 4;    // images of a scaling block
constexpr int kImgResp = 8;    // images of a likelihood block
constexpr int kPairsPerFold = kVT / 32;
// Rotations per launch (the grid's second dimension ends at 65,535), and per call.
constexpr int kChunkLaunch = 65535 * kRotPerCta, kChunkMax = 65535 * 8;

// Folds 16 pairs' 512-wide partials with the reference's tree, data[t] +=
// data[t + s] for s = 256, 128, ..., 1: the partials go through shared memory to
// one warp per pair, whose lane l holds t = l, l + 32, ...: the steps from 256 to
// 32 add inside the lane, the rest are shuffles, the same pairs in the same
// order.  Returns pair `warp`'s sum in every warp's lane 0.
template <typename T>
__device__ __forceinline__ T fold16(const T (&v)[kPairsPerFold], T* smem) {
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kPairsPerFold; ++j) smem[j * kVT + threadIdx.x] = v[j];
  __syncthreads();
  const T* src = smem + (threadIdx.x >> 5) * kVT + (threadIdx.x & 31);
  T x[kVT / 32];
#pragma unroll
  for (int j = 0; j < kVT / 32; ++j) x[j] = src[32 * j];
#pragma unroll
  for (int h = kVT / 64; h >= 1; h >>= 1)
#pragma unroll
    for (int j = 0; j < h; ++j) x[j] = x[j] + x[j + h];
  T r = x[0];
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) r = r + __shfl_down_sync(0xffffffffu, r, s);
  return r;
}

// den + k s truncated toward zero into an int, kept as the float of that int
// (the reference converts it back before the next addition, exactly where the
// int came from a float).  Below 2^23 adding 2^23 toward zero drops the
// fraction; from there on a float has none, and the int saturates at 2^31 - 1,
// which converts back to 2^31.
__device__ __forceinline__ float trunc_add(float den, float k, float s) {
  const float f = __fmaf_rn(k, s, den);
  const float t = __fsub_rn(__fadd_rz(f, 8388608.0f), 8388608.0f);
  return f < 8388608.0f ? t : fminf(f, 2147483648.0f);
}

// One block: kImgScal images x kRotPerCta rotations.
__global__ void __launch_bounds__(kVT) scaling_ref_kernel(
    const float* __restrict__ images, const float* __restrict__ slices,
    const int* __restrict__ mask, float* __restrict__ scaling, int n_2d, int n_images,
    int slice_start, int chunk) {
  __shared__ float s_fold[kPairsPerFold * kVT];
  static_assert(kRotPerCta * kImgScal == kPairsPerFold, "one fold per block");
  const int i0 = blockIdx.x * kImgScal, r0 = blockIdx.y * kRotPerCta;
  const float* img[kImgScal];
  const float* sl[kRotPerCta];
#pragma unroll
  for (int i = 0; i < kImgScal; ++i)
    img[i] = images + (size_t)min(i0 + i, n_images - 1) * n_2d;
#pragma unroll
  for (int j = 0; j < kRotPerCta; ++j) sl[j] = slices + (size_t)min(r0 + j, chunk - 1) * n_2d;
  float num[kPairsPerFold], den[kPairsPerFold];
#pragma unroll
  for (int e = 0; e < kPairsPerFold; ++e) num[e] = den[e] = 0.0f;
  for (int p = threadIdx.x; p < n_2d; p += kVT) {
    if (__ldg(mask + p) <= 0) continue;
    float k[kImgScal], s[kRotPerCta];
#pragma unroll
    for (int i = 0; i < kImgScal; ++i) k[i] = __ldg(img[i] + p);
#pragma unroll
    for (int j = 0; j < kRotPerCta; ++j) s[j] = __ldg(sl[j] + p);
    // x >= 1e-10f is (double)x > 1e-10 for every float x
#pragma unroll
    for (int i = 0; i < kImgScal; ++i) {
      if (!(k[i] >= 1e-10f)) continue;
#pragma unroll
      for (int j = 0; j < kRotPerCta; ++j)
        if (s[j] >= 1e-10f) {
          const int e = i * kRotPerCta + j;
          num[e] = __fmaf_rn(k[i], k[i], num[e]);
          den[e] = trunc_add(den[e], k[i], s[j]);
        }
    }
  }
  const float n = fold16(num, s_fold);
  int di[kPairsPerFold];
#pragma unroll
  for (int e = 0; e < kPairsPerFold; ++e) di[e] = __float2int_rz(den[e]);
  const int d = fold16(di, reinterpret_cast<int*>(s_fold));
  const int e = threadIdx.x >> 5, i = i0 + e / kRotPerCta, r = r0 + e % kRotPerCta;
  if ((threadIdx.x & 31) == 0 && i < n_images && r < chunk)
    scaling[(size_t)(slice_start + r) * n_images + i] = __fdiv_rn(n, __int2float_rn(d));
}

// k / phi correctly rounded from the correctly rounded reciprocal r of phi
// (Markstein 1990): the quotient by r and one exact residual.  For operands and
// a quotient well inside the normal range.
__device__ __forceinline__ float div_by(float k, float phi, float r) {
  const float y = __fmul_rn(k, r);
  return __fmaf_rn(__fmaf_rn(-y, phi, k), r, y);
}

// |x| in [lo, hi] (false for NaN).
__device__ __forceinline__ bool in_range(float x, float lo, float hi) {
  return fabsf(x) >= lo && fabsf(x) <= hi;
}

// One block: kImgResp images x kRotPerCta rotations.  The reference rounds
// (double)sum + ((double)d / sqrt((double)s + 0.02))^2 to float; d^2 / (s + 0.02)
// and the sum are formed here in pairs of floats (48 bits: 1 / (s + 0.02) once
// per rotation and pixel, the square, product and sum exact to their low
// halves), which rounds to the same float except where the FP64 result lies
// within 2^-21 of an ulp of a tie.  Pixels outside the range where the pairs
// hold (checked) take the reference's own operations: a term stays below (2^51)^2 x 50
// < 2^108, so that a thread's sum (2^20 terms for 2^29 pixels) does not reach infinity,
// where a pair's low half would be NaN.
template <int DIFF>
__global__ void __launch_bounds__(kVT, 1) respons_ref_kernel(
    const float* __restrict__ slices, const float* __restrict__ images,
    const int* __restrict__ mask, float sigma, const float* __restrict__ scaling,
    float* __restrict__ respons, const float* __restrict__ weights, int n_2d, int n_images,
    int slice_start, int chunk) {
  constexpr int PAIRS = kImgResp * kRotPerCta;
  __shared__ float s_fold[kPairsPerFold * kVT];
  __shared__ float2 s_phi[PAIRS];  // phi and its reciprocal, as div_by takes them
  __shared__ float s_raw[PAIRS];   // phi
  __shared__ int s_cnt[kRotPerCta];
  const int i0 = blockIdx.x * kImgResp, r0 = blockIdx.y * kRotPerCta;
  const float* img[kImgResp];
  const float* sl[kRotPerCta];
#pragma unroll
  for (int i = 0; i < kImgResp; ++i)
    img[i] = images + (size_t)min(i0 + i, n_images - 1) * n_2d;
#pragma unroll
  for (int j = 0; j < kRotPerCta; ++j) sl[j] = slices + (size_t)min(r0 + j, chunk - 1) * n_2d;
  int bad = 0;
  if (threadIdx.x < PAIRS) {
    const int i = min(i0 + (int)threadIdx.x / kRotPerCta, n_images - 1);
    const int r = min(r0 + (int)threadIdx.x % kRotPerCta, chunk - 1);
    const float phi = __ldg(scaling + (size_t)(slice_start + r) * n_images + i);
    s_raw[threadIdx.x] = phi;
    // k / inf = 0 (a denominator truncated to 0 everywhere) is k (1 / inf) with residual k * 0
    const bool inf = isinf(phi);
    s_phi[threadIdx.x] = inf ? make_float2(1.0f, 0.0f) : make_float2(phi, __frcp_rn(phi));
    bad = !inf && !in_range(phi, 0x1p-25f, 0x1p60f);
  }
  if (threadIdx.x < kRotPerCta) s_cnt[threadIdx.x] = 0;
  const bool phi_ok = !__syncthreads_or(bad);
  float sum[PAIRS];
  int cnt[kRotPerCta];
#pragma unroll
  for (int e = 0; e < PAIRS; ++e) sum[e] = 0.0f;
#pragma unroll
  for (int j = 0; j < kRotPerCta; ++j) cnt[j] = 0;
  for (int p = threadIdx.x; p < n_2d; p += kVT) {
    if (__ldg(mask + p) == 0) continue;
    float k[kImgResp], s[kRotPerCta];
    bool ok = phi_ok;
#pragma unroll
    for (int i = 0; i < kImgResp; ++i) {
      k[i] = __ldg(img[i] + p);
      ok = ok && (k[i] == 0.0f || in_range(k[i], 0x1p-60f, 0x1p25f));
    }
#pragma unroll
    for (int j = 0; j < kRotPerCta; ++j) {
      s[j] = __ldg(sl[j] + p);
      cnt[j] += s[j] > 0.0f;
      ok = ok && (!(s[j] > 0.0f) || in_range(s[j], 0x1p-50f, 0x1p50f));
    }
    if (ok) {
#pragma unroll
      for (int j = 0; j < kRotPerCta; ++j) {
        if (!(s[j] > 0.0f)) continue;
        float wh = 0.0f, wl = 0.0f;
        if (DIFF == EMC_DIFF_POISSON) {
          // a = s + 0.02 as a pair (0.02 = 0.02f + (0.02 - 0.02f)), w = 1 / a
          constexpr float ch = 0.02f, cl = (float)(0.02 - (double)0.02f);
          const float h = __fadd_rn(s[j], ch), b = __fsub_rn(h, s[j]);
          const float l = __fadd_rn(__fadd_rn(__fsub_rn(s[j], __fsub_rn(h, b)), __fsub_rn(ch, b)), cl);
          wh = __frcp_rn(h);
          wl = __fmul_rn(wh, __fmaf_rn(-wh, l, __fmaf_rn(-wh, h, 1.0f)));
        }
#pragma unroll
        for (int i = 0; i < kImgResp; ++i) {
          const int e = i * kRotPerCta + j;
          const float2 f = s_phi[e];
          const float d = __fsub_rn(s[j], div_by(k[i], f.x, f.y));
          if (DIFF == EMC_DIFF_POISSON) {
            const float q = __fmul_rn(d, d), ql = __fmaf_rn(d, d, -q);
            const float x = __fmul_rn(q, wh);
            const float xl = __fmaf_rn(q, wl, __fmaf_rn(ql, wh, __fmaf_rn(q, wh, -x)));
            const float t = __fadd_rn(sum[e], x), b = __fsub_rn(t, sum[e]);
            const float tl = __fadd_rn(__fsub_rn(sum[e], __fsub_rn(t, b)), __fsub_rn(x, b));
            sum[e] = __fadd_rn(t, __fadd_rn(tl, xl));
          } else if (DIFF == EMC_DIFF_ABSOLUTE) {
            sum[e] = __fmaf_rn(d, d, sum[e]);
          } else {  // EMC_DIFF_RELATIVE
            const float q = __fdiv_rn(d, s[j]);
            sum[e] = __fmaf_rn(q, q, sum[e]);
          }
        }
      }
    } else {
#pragma unroll 1
      for (int e0 = 0; e0 < PAIRS; ++e0) {
        // (one pair at a time: register arrays are indexed by constants only)
#pragma unroll
        for (int e = 0; e < PAIRS; ++e) {
          if (e != e0) continue;
          const int i = e / kRotPerCta, j = e % kRotPerCta;
          if (!(s[j] > 0.0f)) continue;
          const float d = __fsub_rn(s[j], __fdiv_rn(k[i], s_raw[e]));
          if (DIFF == EMC_DIFF_POISSON) {
            const double t = (double)d / sqrt((double)s[j] + 0.02);
            sum[e] = (float)((double)sum[e] + t * t);
          } else if (DIFF == EMC_DIFF_ABSOLUTE) {
            sum[e] = __fmaf_rn(d, d, sum[e]);
          } else {
            const float q = __fdiv_rn(d, s[j]);
            sum[e] = __fmaf_rn(q, q, sum[e]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kRotPerCta; ++j) {
    const int c = (int)__reduce_add_sync(0xffffffffu, (unsigned)cnt[j]);
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_cnt[j], c);
  }
#pragma unroll
  for (int h = 0; h < PAIRS / kPairsPerFold; ++h) {
    float part[kPairsPerFold];
#pragma unroll
    for (int e = 0; e < kPairsPerFold; ++e) part[e] = sum[h * kPairsPerFold + e];
    const float total = fold16(part, s_fold);
    const int e = h * kPairsPerFold + (int)(threadIdx.x >> 5);
    const int i = i0 + e / kRotPerCta, jr = e % kRotPerCta, r = slice_start + r0 + jr;
    if ((threadIdx.x & 31) == 0 && i < n_images && r0 + jr < chunk) {
      const double sig2 = (double)__fmul_rn(sigma, sigma);
      const double lw = (double)logf(__ldg(weights + r));
      const double v = (double)total / 2.0 / (double)__int2float_rn(s_cnt[jr]) / sig2;
      respons[(size_t)r * n_images + i] = (float)(lw - v);
    }
  }
}

}  // namespace emc

extern "C" int emc_update_scaling_full(emc_ctx* ctx, const float* d_images,
                                       const float* d_slices, const int* d_mask,
                                       float* d_scaling, int N_2d, int N_images,
                                       int slice_start, int slice_chunk, int diff) {
  EMC_CHECK_CTX(ctx);
  (void)diff;  // the reference ignores diff here and always uses the absolute form
  EMC_REQUIRE(ctx, d_images && d_slices && d_mask && d_scaling, "update_scaling_full: null pointer");
  EMC_REQUIRE(ctx, N_2d > 0 && N_images >= 0 && slice_start >= 0 && slice_chunk >= 0,
              "update_scaling_full: bad sizes");
  if (N_images == 0 || slice_chunk == 0) return EMC_OK;
  EMC_REQUIRE(ctx, slice_chunk <= emc::kChunkMax, "update_scaling_full: chunk too large");
  for (int r0 = 0; r0 < slice_chunk; r0 += emc::kChunkLaunch) {
    const int n = std::min(slice_chunk - r0, emc::kChunkLaunch);
    dim3 grid(emc::ceil_div(N_images, emc::kImgScal), emc::ceil_div(n, emc::kRotPerCta));
    emc::scaling_ref_kernel<<<grid, emc::kVT, 0, ctx->stream>>>(
        d_images, d_slices + (size_t)r0 * N_2d, d_mask, d_scaling, N_2d, N_images,
        slice_start + r0, n);
    const int rc = emc::after_launch(ctx, "scaling_ref_kernel");
    if (rc) return rc;
  }
  return EMC_OK;
}

extern "C" int emc_calculate_responsabilities(emc_ctx* ctx, const float* d_slices,
                                              const float* d_images, const int* d_mask,
                                              float sigma, const float* d_scaling,
                                              float* d_respons, const float* d_weights, int N_2d,
                                              int N_images, int slice_start, int slice_chunk,
                                              int diff) {
  EMC_CHECK_CTX(ctx);
  EMC_REQUIRE(ctx, d_images && d_slices && d_mask && d_scaling && d_respons && d_weights,
              "calculate_responsabilities: null pointer");
  EMC_REQUIRE(ctx, N_2d > 0 && N_images >= 0 && slice_start >= 0 && slice_chunk >= 0,
              "calculate_responsabilities: bad sizes");
  EMC_REQUIRE(ctx, diff == EMC_DIFF_ABSOLUTE || diff == EMC_DIFF_POISSON || diff == EMC_DIFF_RELATIVE,
              "calculate_responsabilities: diff %d is not a reference diff type", diff);
  if (N_images == 0 || slice_chunk == 0) return EMC_OK;
  EMC_REQUIRE(ctx, slice_chunk <= emc::kChunkMax, "calculate_responsabilities: chunk too large");
  auto* kernel = diff == EMC_DIFF_POISSON    ? emc::respons_ref_kernel<EMC_DIFF_POISSON>
                 : diff == EMC_DIFF_ABSOLUTE ? emc::respons_ref_kernel<EMC_DIFF_ABSOLUTE>
                                             : emc::respons_ref_kernel<EMC_DIFF_RELATIVE>;
  for (int r0 = 0; r0 < slice_chunk; r0 += emc::kChunkLaunch) {
    const int n = std::min(slice_chunk - r0, emc::kChunkLaunch);
    dim3 grid(emc::ceil_div(N_images, emc::kImgResp), emc::ceil_div(n, emc::kRotPerCta));
    kernel<<<grid, emc::kVT, 0, ctx->stream>>>(d_slices + (size_t)r0 * N_2d, d_images, d_mask,
                                               sigma, d_scaling, d_respons, d_weights, N_2d,
                                               N_images, slice_start + r0, n);
    const int rc = emc::after_launch(ctx, "respons_ref_kernel");
    if (rc) return rc;
  }
  return EMC_OK;
}
