// Learned rotation proposal: a small convolutional network that maps a
// diffraction pattern to a rotation, trained on the GPU (forward, backward
// and Adam kernels below) on the most probable rotations of EMC's own
// responsibilities, and used to seed pruned iterations
// (emc_plan_set_proposals) for patterns that have no responsibilities yet.
// The reference has no counterpart; the network follows the
// rotation-proposal design of the EMC iteration's pruning: 4 convolutions
// (3x3, stride 2, 64 channels, ReLU) over the pattern binned to 64 x 64
// pixels, one linear layer to a 6D rotation (the first two columns of the
// rotation matrix, made orthonormal by Gram-Schmidt).
//
// Friedel symmetry makes a pattern at rotation M nearly identical to the one
// at M diag(-1, -1, 1) (a half turn about the beam axis; they differ only
// through the Ewald sphere's curvature), whose 6D form is exactly the
// negative.  The loss is therefore min(|o - t|^2, |o + t|^2) per pattern,
// and a prediction proposes both rotations.
//
// Arithmetic is FP32 SIMT: one forward pass is 26 MFLOP per pattern,
// under 1 % of a 128^3 iteration's E-step per pattern, so the tensor cores
// stay with the iteration's contractions.  Every reduction has a fixed order
// (no atomics), so training is reproducible for a given seed.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "emc_gb300.h"
#include "geometry.cuh"
#include "plan.cuh"
#include "ptx.cuh"

namespace emc {
namespace pn {
constexpr int D = 64;              // input side
constexpr int CH = 64;             // channels of every convolution
constexpr int NCONV = 4;
constexpr int FC_IN = CH * 4 * 4;  // 1024
constexpr int OUT = 6;
constexpr int CC = 8;              // channels per reduction chunk of the convolution kernels
constexpr int WS = CH + 4;         // padded row of 64 channels in shared memory
constexpr int WG_BLOCKS = 304;     // blocks of a weight-gradient launch, two per SM
constexpr int FC_ROWS = 16;        // samples per block of the linear head's backward pass

__host__ __device__ constexpr int cin(int l) { return l == 0 ? 1 : CH; }
__host__ __device__ constexpr int hin(int l) { return D >> l; }  // 64, 32, 16, 8
}  // namespace pn

struct ProposalNet {
  emc_ctx* ctx = nullptr;
  size_t off_w[pn::NCONV], off_b[pn::NCONV], off_fw = 0, off_fb = 0, n_params = 0;
  float *params = nullptr, *grads = nullptr, *adam_m = nullptr, *adam_v = nullptr;
  long long adam_t = 0;
  // inputs
  float* X = nullptr;  // [n][64*64]
  int n_data = 0;
  float* stats = nullptr;  // [2][4096]: per-input-pixel mean and 1 / spread of the training data
  bool have_stats = false;
  // per-batch workspace (capacity cap samples)
  int cap = 0;
  float* act[pn::NCONV + 1] = {};  // act[0] = gathered inputs, act[l+1] = output of conv l
  float* out = nullptr;            // [cap][6]
  float *g0 = nullptr, *g1 = nullptr;  // ping-pong activation gradients (largest layer)
  float* gout = nullptr;               // [cap][6]
  float* wpart = nullptr;              // weight- and bias-gradient partials
  size_t wpart_cap = 0;
  float* loss = nullptr;               // [cap]
  int* idx = nullptr;                  // [cap] sample -> data row
  int* quarter = nullptr;              // [cap] in-plane quarter turns of the sample
  float* labels6 = nullptr;            // [cap][6]
};

// ------------------------------------------------------------ inputs -----
// X[j] = log1p(v * 4096 / max(sum v, 1)), v = the pattern's counts summed
// over b x b pixel blocks (b = side / 64) inside the mask (negative counts,
// the per-pattern masked pixels, count 0); then standardised per input pixel
// with the training data's mean and spread (the radial falloff that every
// pattern shares carries no orientation).
__global__ void proposal_inputs_kernel(const float* __restrict__ images,
                                       const int* __restrict__ mask, int side, int n,
                                       float* __restrict__ X) {
  const int i = blockIdx.x;
  if (i >= n) return;
  const int b = side / pn::D;
  const float* im = images + (size_t)i * side * side;
  float v[16];
  float s = 0.0f;
  for (int u = 0; u < 16; ++u) {
    const int o = threadIdx.x + u * 256;  // output pixel 0..4095
    const int oy = o / pn::D, ox = o % pn::D;
    float a = 0.0f;
    for (int dy = 0; dy < b; ++dy)
      for (int dx = 0; dx < b; ++dx) {
        const int p = (oy * b + dy) * side + ox * b + dx;
        const float k = im[p];
        if (mask[p] > 0 && k > 0.0f) a += k;
      }
    v[u] = a;
    s += a;
  }
  __shared__ float red[256];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
    __syncthreads();
  }
  const float scale = 4096.0f / fmaxf(red[0], 1.0f);
  for (int u = 0; u < 16; ++u)
    X[(size_t)i * 4096 + threadIdx.x + u * 256] = log1pf(v[u] * scale);
}

// Batch inputs: row idx[j] of X turned in-plane by quarter[j] x 90 degrees
// (nullptr: not turned).  A turn by +90 degrees, X'(u, v) = X(v, -u) in
// centred coordinates, is the pattern of rotation M Rz(-90 deg): exact on
// the 64 x 64 grid, whose mask and pixel heights are symmetric under it.
// stats[0][c] = mean over rows of X[.][c], stats[1][c] = 1 / sqrt(var + 1e-4)
// (FP64 sums in row order); one thread per input pixel.
__global__ void input_stats_kernel(const float* __restrict__ X, int n, float* __restrict__ stats) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= 4096) return;
  double s = 0.0, s2 = 0.0;
  for (int i = 0; i < n; ++i) {
    const double v = X[(size_t)i * 4096 + c];
    s += v;
    s2 += v * v;
  }
  const double m = s / n;
  const double var = fmax(s2 / n - m * m, 0.0);
  stats[c] = (float)m;
  stats[4096 + c] = (float)(1.0 / sqrt(var + 1e-4));
}

// X[i][c] = (X[i][c] - mean[c]) * inv[c].
__global__ void standardize_kernel(float* __restrict__ X, size_t n, const float* __restrict__ stats) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n * 4096) return;
  const int c = (int)(e % 4096);
  X[e] = (X[e] - stats[c]) * stats[4096 + c];
}

__global__ void gather_rows_kernel(const float* __restrict__ X, const int* __restrict__ idx,
                                   const int* __restrict__ quarter, int rows,
                                   float* __restrict__ out) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (size_t)rows * 4096) return;
  const int j = (int)(e / 4096), c = (int)(e % 4096);
  int oy = c / pn::D, ox = c % pn::D;
  const int k = quarter ? (quarter[j] & 3) : 0;
  for (int t = 0; t < k; ++t) {  // source of one +90 degree turn: (63 - ox, oy) as (row, col)
    const int ny = pn::D - 1 - ox, nx = oy;
    oy = ny;
    ox = nx;
  }
  out[e] = X[(size_t)idx[j] * 4096 + oy * pn::D + ox];
}

// ------------------------------------------------------- convolutions ----
// All of them keep a patch of the input (or of the output gradient) and eight
// channels' weights in shared memory and 64 to 72 sums per thread in registers,
// so that a value from shared memory serves eight multiply-adds; what bounds them
// is FP32 issue.  The GEMM form before, with 4 x 4 sums per thread and every
// element of the implicit column matrix addressed by divisions, reached 14 TFLOP/s
// forward: 4,107 us for 2,250 patterns, now 1,406 (49 TFLOP/s in the layer with 16 x
// 16 outputs); the gradients of 250 patterns took 3,271 us, now 560.

// A stride-2 row of the input in shared memory: the even columns 0, 2, .. at 0,
// the odd ones -1, 1, 3, .. at HO, so that the eight outputs of a thread read
// neighbours.  Rows -1 .. 2 HO - 1 at 0 .. 2 HO; what lies outside is zero.
template <int HO>
struct ConvPatch {
  static constexpr int HI = 2 * HO, ROWS = HI + 1, RS = 2 * HO + 4, SIZE = ROWS * RS;
  static __device__ __forceinline__ int at(int y, int x) {
    return (y + 1) * RS + ((x & 1) ? HO + (x + 1) / 2 : x / 2);
  }
  // pixels 4 q .. 4 q + 3 of an image into its patch
  static __device__ __forceinline__ void put4(float* patch, int q, float4 v) {
    const int y = q / (HI / 4), x = (q % (HI / 4)) * 4;
    float* row = patch + (y + 1) * RS + x / 2;
    *reinterpret_cast<float2*>(row) = make_float2(v.x, v.z);
    row[HO + 1] = v.y;
    row[HO + 2] = v.w;
  }
};

// Channel i of the eight that channel group cg of a block's eight takes: four and
// four, so that the groups' 16-byte loads meet all banks once.
__device__ __forceinline__ int own_channel(int cg, int i) {
  return (i & 4) * 8 + cg * 4 + (i & 3);
}

using ptx::f32x2;

__device__ __forceinline__ f32x2 twice(float x) { return ptx::pack2(x, x); }

__device__ __forceinline__ float4 relu_grad(float4 out, float4 g) {
  return make_float4(out.x > 0.0f ? g.x : 0.0f, out.y > 0.0f ? g.y : 0.0f,
                     out.z > 0.0f ? g.z : 0.0f, out.w > 0.0f ? g.w : 0.0f);
}

__device__ __forceinline__ float4 ldg4(const float* p) {
  return __ldg(reinterpret_cast<const float4*>(p));
}

// First convolution (one input channel, 64 -> 32 pixels): one thread per output
// pixel, all 64 channels.
__global__ void __launch_bounds__(256) conv0_fwd_kernel(const float* __restrict__ in,
                                                        const float* __restrict__ W,
                                                        const float* __restrict__ bias,
                                                        float* __restrict__ out) {
  constexpr int HI = pn::D, HO = HI / 2, NPX = HO * HO;
  __shared__ __align__(16) float sW[9][pn::CH], sB[pn::CH];
  for (int e = threadIdx.x; e < 9 * pn::CH; e += 256) sW[e % 9][e / 9] = W[e];
  if (threadIdx.x < pn::CH) sB[threadIdx.x] = bias[threadIdx.x];
  __syncthreads();
  const int b = blockIdx.x / (NPX / 256), p = (blockIdx.x % (NPX / 256)) * 256 + threadIdx.x;
  const int oy = p / HO, ox = p % HO;
  const float* src = in + (size_t)b * HI * HI;
  float v[9];
#pragma unroll
  for (int t = 0; t < 9; ++t) {
    const int y = 2 * oy + t / 3 - 1, x = 2 * ox + t % 3 - 1;
    v[t] = y >= 0 && x >= 0 ? src[y * HI + x] : 0.0f;  // never past the other edge
  }
  float* dst = out + (size_t)b * pn::CH * NPX + p;
#pragma unroll 4
  for (int c = 0; c < pn::CH; c += 4) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int t = 0; t < 9; ++t) {
      const float4 w = *reinterpret_cast<const float4*>(&sW[t][c]);
      a.x = fmaf(w.x, v[t], a.x);
      a.y = fmaf(w.y, v[t], a.y);
      a.z = fmaf(w.z, v[t], a.z);
      a.w = fmaf(w.w, v[t], a.w);
    }
    const float o[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int u = 0; u < 4; ++u) dst[(size_t)(c + u) * NPX] = fmaxf(o[u] + sB[c + u], 0.0f);
  }
}

// out[b][co][p] = relu(bias[co] + sum_{ci,t} W[co][ci*9+t] in[b][ci][tap(p,t)]),
// 64 input channels, in the order of (ci, t).  256 threads: 8 groups of 8 output
// channels x 32 groups of PX neighbouring outputs, over SPB samples.
template <int HO>
struct ConvFwd {
  using Patch = ConvPatch<HO>;
  static constexpr int PX = HO >= 8 ? 8 : 4;
  static constexpr int GROUPS = HO * HO / PX, SPB = 32 / GROUPS;
  static constexpr int X = pn::CC * SPB * Patch::SIZE, W = pn::CC * 9 * pn::WS;
  static constexpr int SMEM = (X + W) * 4;
};

template <int HO>
__global__ void __launch_bounds__(256, 2) conv_fwd_kernel(const float* __restrict__ in,
                                                          const float* __restrict__ W,
                                                          const float* __restrict__ bias,
                                                          float* __restrict__ out, int B) {
  using F = ConvFwd<HO>;
  using Patch = typename F::Patch;
  constexpr int PX = F::PX, HI = Patch::HI, K = pn::CH * 9;
  extern __shared__ __align__(16) float sm[];
  float *sX = sm, *sW = sm + F::X;
  const int cg = threadIdx.x & 7, pg = threadIdx.x >> 3;
  const int smp = pg / F::GROUPS, g = pg % F::GROUPS;
  const int oy = g / (HO / PX), ox = (g % (HO / PX)) * PX;
  const int b0 = blockIdx.x * F::SPB;
  for (int e = threadIdx.x; e < F::X; e += 256) sX[e] = 0.0f;  // the borders stay zero
  f32x2 acc[4][PX];  // pairs of output channels
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < PX; ++j) acc[i][j] = 0;
  for (int c0 = 0; c0 < pn::CH; c0 += pn::CC) {
    __syncthreads();
    constexpr int Q = HI * HI / 4;
#pragma unroll 8
    for (int e = threadIdx.x; e < pn::CC * F::SPB * Q; e += 256) {
      const int q = e % Q, u = e / Q, c = u % pn::CC, sp = u / pn::CC;
      if (b0 + sp < B)
        Patch::put4(sX + (c * F::SPB + sp) * Patch::SIZE, q,
                    ldg4(in + ((size_t)(b0 + sp) * pn::CH + c0 + c) * (HI * HI) + 4 * q));
    }
#pragma unroll 5
    for (int e = threadIdx.x; e < pn::CH * pn::CC * 9 / 4; e += 256) {
      const int co = e % pn::CH, k = e / pn::CH * 4;
      const float4 w = ldg4(W + (size_t)co * K + c0 * 9 + k);
      float* dst = sW + k * pn::WS + co;
      dst[0] = w.x;
      dst[pn::WS] = w.y;
      dst[2 * pn::WS] = w.z;
      dst[3 * pn::WS] = w.w;
    }
    __syncthreads();
#pragma unroll 1
    for (int c = 0; c < pn::CC; ++c) {
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) {
        const float* row = sX + (c * F::SPB + smp) * Patch::SIZE + (2 * oy + ky) * Patch::RS + ox;
        f32x2 ev[PX], od[PX + 1];
#pragma unroll
        for (int j = 0; j < PX; j += 4) {
          const float4 a = *reinterpret_cast<const float4*>(row + j);
          const float4 o = *reinterpret_cast<const float4*>(row + HO + j);
          ev[j] = twice(a.x); ev[j + 1] = twice(a.y); ev[j + 2] = twice(a.z); ev[j + 3] = twice(a.w);
          od[j] = twice(o.x); od[j + 1] = twice(o.y); od[j + 2] = twice(o.z); od[j + 3] = twice(o.w);
        }
        od[PX] = twice(row[HO + PX]);
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) {
          const float* wp = sW + (c * 9 + ky * 3 + kx) * pn::WS + cg * 4;
          const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(wp);
          const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(wp + 32);
          const f32x2 w[4] = {w0.x, w0.y, w1.x, w1.y};
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < PX; ++j)
              acc[i][j] = ptx::fma2(w[i], kx == 1 ? ev[j] : od[j + (kx >> 1)], acc[i][j]);
        }
      }
    }
  }
  const int b = b0 + smp;
  if (b >= B) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int co = own_channel(cg, i);
    const float bi = bias[co];
    float* dst = out + (((size_t)b * pn::CH + co) * HO + oy) * HO + ox;
    auto value = [&](int j) {
      const float2 v = ptx::unpack2(acc[i >> 1][j]);
      return fmaxf(((i & 1) ? v.y : v.x) + bi, 0.0f);
    };
#pragma unroll
    for (int j = 0; j < PX; j += 4)
      *reinterpret_cast<float4*>(dst + j) =
          make_float4(value(j), value(j + 1), value(j + 2), value(j + 3));
  }
}

// Backward through ReLU and the convolution to its input:
// gin[b][ci][q] = sum_{co,t} W[co][ci*9+t] d[b][co][p(q,t)], d = gout * (out > 0),
// over the output pixels p whose tap t reads input pixel q, in the order of
// (co, t).  Of the nine taps an input pixel meets one, two, two or four, by the
// parity of its row and column: a thread takes the 2 x 2 input pixels of four
// neighbouring output positions for 4 input channels, 9 products per position,
// channel and co.  256 threads: 16 channel groups x 16 position groups.
template <int HO>
struct ConvBwd {
  static constexpr int ROWS = HO == 16 ? 4 : HO;  // output rows per block and sample
  static constexpr int SPB = 64 / (ROWS * HO), PARTS = HO / ROWS;
  static constexpr int RS = HO + 4, SIZE = (ROWS + 1) * RS;  // one row and column more
  static constexpr int DSZ = pn::CC * SPB * SIZE, W = pn::CC * 9 * pn::WS;
  static constexpr int SMEM = (DSZ + W) * 4;
};

template <int HO>
__global__ void __launch_bounds__(256, 2) conv_bwd_data_kernel(const float* __restrict__ gout,
                                                               const float* __restrict__ out,
                                                               const float* __restrict__ W,
                                                               float* __restrict__ gin, int B) {
  using F = ConvBwd<HO>;
  constexpr int HI = 2 * HO, K = pn::CH * 9;
  extern __shared__ __align__(16) float sm[];
  float *sD = sm, *sW = sm + F::DSZ;
  const int cg = threadIdx.x & 15, pp = threadIdx.x >> 4;
  constexpr int GROUPS = F::ROWS * HO / 4;
  const int smp = pp / GROUPS, g = pp % GROUPS;
  const int ry = g / (HO / 4), px = (g % (HO / 4)) * 4;
  const int b0 = (blockIdx.x / F::PARTS) * F::SPB, y0 = (blockIdx.x % F::PARTS) * F::ROWS;
  for (int e = threadIdx.x; e < F::DSZ; e += 256) sD[e] = 0.0f;  // the borders stay zero
  // pairs of input channels; pixel (2 y, 2 x), (2 y, 2 x + 1), (2 y + 1, 2 x), ..
  f32x2 acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[i][j][u] = 0;
  for (int c0 = 0; c0 < pn::CH; c0 += pn::CC) {
    __syncthreads();
    for (int e = threadIdx.x; e < pn::CC * F::SPB * (F::ROWS + 1) * (HO / 4); e += 256) {
      const int x = e % (HO / 4) * 4, u = e / (HO / 4), r = u % (F::ROWS + 1), v = u / (F::ROWS + 1);
      const int c = v % pn::CC, sp = v / pn::CC;
      if (b0 + sp < B && y0 + r < HO) {
        const size_t o = (((size_t)(b0 + sp) * pn::CH + c0 + c) * HO + y0 + r) * HO + x;
        *reinterpret_cast<float4*>(sD + (c * F::SPB + sp) * F::SIZE + r * F::RS + x) =
            relu_grad(ldg4(out + o), ldg4(gout + o));
      }
    }
#pragma unroll 6
    for (int e = threadIdx.x; e < pn::CC * K; e += 256) {
      const int c = e / K, k = e % K;  // k = ci * 9 + t
      sW[(c * 9 + k % 9) * pn::WS + k / 9] = W[(size_t)(c0 + c) * K + k];
    }
    __syncthreads();
#pragma unroll 1
    for (int c = 0; c < pn::CC; ++c) {
      const float* r0 = sD + (c * F::SPB + smp) * F::SIZE + ry * F::RS + px;
      const float* r1 = r0 + F::RS;
      const float4 e0 = *reinterpret_cast<const float4*>(r0);
      const float4 e1 = *reinterpret_cast<const float4*>(r1);
      const f32x2 d0[5] = {twice(e0.x), twice(e0.y), twice(e0.z), twice(e0.w), twice(r0[4])};
      const f32x2 d1[5] = {twice(e1.x), twice(e1.y), twice(e1.z), twice(e1.w), twice(r1[4])};
#pragma unroll
      for (int t = 0; t < 9; ++t) {
        const ulonglong2 w0 =
            *reinterpret_cast<const ulonglong2*>(sW + (c * 9 + t) * pn::WS + cg * 4);
        const f32x2 w[2] = {w0.x, w0.y};
        const int ky = t / 3, kx = t % 3;
        const int cls = (ky != 1 ? 2 : 0) + (kx != 1 ? 1 : 0);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            acc[i][j][cls] =
                ptx::fma2(w[i], (ky == 0 ? d1 : d0)[j + (kx == 0 ? 1 : 0)], acc[i][j][cls]);
      }
    }
  }
  const int b = b0 + smp;
  if (b >= B) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float* dst = gin + (((size_t)b * pn::CH + cg * 4 + i) * HI + 2 * (y0 + ry)) * HI + 2 * px;
    auto value = [&](int j, int u) {
      const float2 v = ptx::unpack2(acc[i >> 1][j][u]);
      return (i & 1) ? v.y : v.x;
    };
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
      *reinterpret_cast<float4*>(dst + 2 * j) =
          make_float4(value(j, 0), value(j, 1), value(j + 1, 0), value(j + 1, 1));
      *reinterpret_cast<float4*>(dst + HI + 2 * j) =
          make_float4(value(j, 2), value(j, 3), value(j + 1, 2), value(j + 1, 3));
    }
  }
}

// Weight and bias gradient partials of one block's samples: part[s][co][k] = sum
// over them and the output pixels of d[co] in[tap], bpart[s][co] = sum of d.  A
// block takes 8 input channels (72 of the k); 256 threads: 8 groups of 8 output
// channels x 8 input channels x 4 splits of the output rows, each with 8 x 9
// sums; the splits are added in order at the end.
template <int HO>
struct ConvWgrad {
  using Patch = ConvPatch<HO>;
  static constexpr int X = pn::CC * Patch::SIZE, DSZ = HO * HO * pn::WS;
  static constexpr int RED = 3 * 64 * 72;
  static constexpr int SMEM = 4 * (X + DSZ > RED ? X + DSZ : RED);
};

template <int HO>
__global__ void __launch_bounds__(256, 2) conv_wgrad_kernel(const float* __restrict__ gout,
                                                            const float* __restrict__ out,
                                                            const float* __restrict__ in,
                                                            float* __restrict__ part,
                                                            float* __restrict__ bpart, int B,
                                                            int per) {
  using F = ConvWgrad<HO>;
  using Patch = typename F::Patch;
  constexpr int HI = Patch::HI, NPX = HO * HO, K = pn::CH * 9;
  extern __shared__ __align__(16) float sm[];
  float *sX = sm, *sD = sm + F::X;
  const int cg = threadIdx.x & 7, ci = (threadIdx.x >> 3) & 7, sp = threadIdx.x >> 6;
  const int c0 = blockIdx.x * pn::CC, s = blockIdx.y;
  const int bend = min(B, (s + 1) * per);
  f32x2 acc[4][9];  // pairs of output channels
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int t = 0; t < 9; ++t) acc[i][t] = 0;
  float bsum = 0.0f;  // block 0: channel threadIdx.x & 63, split sp of the pixels
  for (int e = threadIdx.x; e < F::X; e += 256) sX[e] = 0.0f;
  for (int b = s * per; b < bend; ++b) {
    __syncthreads();
    constexpr int Q = HI * HI / 4;
#pragma unroll 4
    for (int e = threadIdx.x; e < pn::CC * Q; e += 256)
      Patch::put4(sX + e / Q * Patch::SIZE, e % Q,
                  ldg4(in + ((size_t)b * pn::CH + c0) * (HI * HI) + 4 * e));
#pragma unroll 4
    for (int e = threadIdx.x; e < pn::CH * NPX / 4; e += 256) {
      const int co = e % pn::CH, px = e / pn::CH * 4;
      const size_t o = ((size_t)b * pn::CH + co) * NPX + px;
      const float4 d = relu_grad(ldg4(out + o), ldg4(gout + o));
      float* dst = sD + px * pn::WS + co;
      dst[0] = d.x;
      dst[pn::WS] = d.y;
      dst[2 * pn::WS] = d.z;
      dst[3 * pn::WS] = d.w;
    }
    __syncthreads();
    for (int oy = sp; oy < HO; oy += 4) {
      const float* row = sX + ci * Patch::SIZE + 2 * oy * Patch::RS;
      f32x2 lft[3];
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) lft[ky] = twice(row[ky * Patch::RS + HO]);
#pragma unroll 2
      for (int ox = 0; ox < HO; ++ox) {
        const float* dp = sD + (oy * HO + ox) * pn::WS + cg * 4;
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(dp);
        const ulonglong2 c = *reinterpret_cast<const ulonglong2*>(dp + 32);
        const f32x2 d[4] = {a.x, a.y, c.x, c.y};
        f32x2 x[9];
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
          x[3 * ky] = lft[ky];
          x[3 * ky + 1] = twice(row[ky * Patch::RS + ox]);
          x[3 * ky + 2] = lft[ky] = twice(row[ky * Patch::RS + HO + ox + 1]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int t = 0; t < 9; ++t) acc[i][t] = ptx::fma2(d[i], x[t], acc[i][t]);
      }
    }
    if (blockIdx.x == 0)
      for (int p = sp; p < NPX; p += 4) bsum += sD[p * pn::WS + (threadIdx.x & 63)];
  }
  __syncthreads();
  const int lane64 = threadIdx.x & 63;
  auto value = [&](int i, int t) {
    const float2 v = ptx::unpack2(acc[i >> 1][t]);
    return (i & 1) ? v.y : v.x;
  };
  if (sp > 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int t = 0; t < 9; ++t) sm[((sp - 1) * 72 + i * 9 + t) * 64 + lane64] = value(i, t);
  }
  __syncthreads();
  if (sp == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int t = 0; t < 9; ++t) {
        float v = value(i, t);
#pragma unroll
        for (int u = 0; u < 3; ++u) v += sm[(u * 72 + i * 9 + t) * 64 + lane64];
        part[((size_t)s * pn::CH + own_channel(cg, i)) * K + (c0 + ci) * 9 + t] = v;
      }
  }
  if (blockIdx.x == 0) {
    __syncthreads();
    sm[threadIdx.x] = bsum;
    __syncthreads();
    if (threadIdx.x < 64) {
      float v = 0.0f;
#pragma unroll
      for (int u = 0; u < 4; ++u) v += sm[u * 64 + threadIdx.x];
      bpart[(size_t)s * pn::CH + threadIdx.x] = v;
    }
  }
}

// The same for the first convolution (one input channel): a warp takes 8 output
// channels, its lanes neighbouring pixels; the lanes' sums are added at the end.
__global__ void __launch_bounds__(256) conv0_wgrad_kernel(const float* __restrict__ gout,
                                                          const float* __restrict__ out,
                                                          const float* __restrict__ in,
                                                          float* __restrict__ part,
                                                          float* __restrict__ bpart, int B,
                                                          int per) {
  constexpr int HI = pn::D, HO = HI / 2, NPX = HO * HO;
  using Patch = ConvPatch<HO>;
  __shared__ float sX[Patch::SIZE];
  const int lane = threadIdx.x & 31, cw = (threadIdx.x >> 5) * 8, s = blockIdx.x;
  const int bend = min(B, (s + 1) * per);
  float acc[8][10];  // nine taps and the bias
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int t = 0; t < 10; ++t) acc[i][t] = 0.0f;
  for (int e = threadIdx.x; e < Patch::SIZE; e += 256) sX[e] = 0.0f;
  for (int b = s * per; b < bend; ++b) {
    __syncthreads();
    for (int e = threadIdx.x; e < HI * HI; e += 256)
      sX[Patch::at(e / HI, e % HI)] = in[(size_t)b * HI * HI + e];
    __syncthreads();
    for (int oy = 0; oy < HO; ++oy) {  // 32 pixels: one row
      float x[9];
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) {
        const float* row = sX + (2 * oy + ky) * Patch::RS;
        x[3 * ky] = row[HO + lane];
        x[3 * ky + 1] = row[lane];
        x[3 * ky + 2] = row[HO + lane + 1];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const size_t o = ((size_t)b * pn::CH + cw + i) * NPX + oy * HO + lane;
        const float d = out[o] > 0.0f ? gout[o] : 0.0f;
#pragma unroll
        for (int t = 0; t < 9; ++t) acc[i][t] = fmaf(d, x[t], acc[i][t]);
        acc[i][9] += d;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int t = 0; t < 10; ++t) {
      float v = acc[i][t];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) {
        if (t < 9)
          part[((size_t)s * pn::CH + cw + i) * 9 + t] = v;
        else
          bpart[(size_t)s * pn::CH + cw + i] = v;
      }
    }
}

// grad[e] = sum_s part[s][e] (fixed order), e < n; then the n2 of part2 the same.
__global__ void sum_parts_kernel(const float* __restrict__ part, const float* __restrict__ part2,
                                 int S, int n, int n2, float* __restrict__ grad,
                                 float* __restrict__ grad2) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n + n2) return;
  const float* src = e < n ? part + e : part2 + (e - n);
  const int m = e < n ? n : n2;
  float a = 0.0f;
#pragma unroll 16
  for (int s = 0; s < S; ++s) a += src[(size_t)s * m];
  if (e < n)
    grad[e] = a;
  else
    grad2[e - n] = a;
}

// ---------------------------------------------------------- linear head --
// o[b][j] = fb[j] + sum_k fw[j][k] h[b][k]; one block per sample.
__global__ void fc_fwd_kernel(const float* __restrict__ h, const float* __restrict__ fw,
                              const float* __restrict__ fb, float* __restrict__ o) {
  const int b = blockIdx.x;
  __shared__ float red[pn::OUT][256];
  for (int j = 0; j < pn::OUT; ++j) {
    float a = 0.0f;
    for (int k = threadIdx.x; k < pn::FC_IN; k += 256)
      a = fmaf(fw[j * pn::FC_IN + k], h[(size_t)b * pn::FC_IN + k], a);
    red[j][threadIdx.x] = a;
  }
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      for (int j = 0; j < pn::OUT; ++j) red[j][threadIdx.x] += red[j][threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x < pn::OUT) o[b * pn::OUT + threadIdx.x] = red[threadIdx.x][0] + fb[threadIdx.x];
}

// gh[b][k] = sum_j fw[j][k] go[b][j]; part[s][j][k] = sum_b go[b][j] h[b][k] and
// bpart[s][j] = sum_b go[b][j] over the FC_ROWS samples of block row s.
__global__ void __launch_bounds__(256) fc_bwd_kernel(const float* __restrict__ h,
                                                     const float* __restrict__ fw,
                                                     const float* __restrict__ go, int B,
                                                     float* __restrict__ gh,
                                                     float* __restrict__ part,
                                                     float* __restrict__ bpart) {
  const int k = blockIdx.x * 256 + threadIdx.x, s = blockIdx.y;
  const int b0 = s * pn::FC_ROWS, b1 = min(B, b0 + pn::FC_ROWS);
  float w[pn::OUT], g[pn::OUT] = {};
#pragma unroll
  for (int j = 0; j < pn::OUT; ++j) w[j] = fw[j * pn::FC_IN + k];
#pragma unroll 4
  for (int b = b0; b < b1; ++b) {
    const float hv = h[(size_t)b * pn::FC_IN + k];
    float a = 0.0f;
#pragma unroll
    for (int j = 0; j < pn::OUT; ++j) {
      const float gj = __ldg(go + b * pn::OUT + j);
      g[j] = fmaf(gj, hv, g[j]);
      a = fmaf(w[j], gj, a);
    }
    gh[(size_t)b * pn::FC_IN + k] = a;
  }
#pragma unroll
  for (int j = 0; j < pn::OUT; ++j) part[((size_t)s * pn::OUT + j) * pn::FC_IN + k] = g[j];
  if (blockIdx.x == 0 && threadIdx.x < pn::OUT) {
    float a = 0.0f;
    for (int b = b0; b < b1; ++b) a += go[b * pn::OUT + threadIdx.x];
    bpart[s * pn::OUT + threadIdx.x] = a;
  }
}

// ------------------------------------------------------------ rotations --
// 6D form of a rotation: the first two columns of its matrix (as used by the
// slicing kernels: rotated = M p).
__device__ __forceinline__ void quat_to_6d(const float* q, float* t) {
  const RotMat m = quat_to_matrix(q);
  t[0] = m.m[0]; t[1] = m.m[3]; t[2] = m.m[6];
  t[3] = m.m[1]; t[4] = m.m[4]; t[5] = m.m[7];
}

// labels6[j] = 6D form of quats[idx[j]] composed with Rz(-90 deg) quarter[j]
// times: (c1, c2) -> (-c2, c1) per turn.
__global__ void labels_kernel(const float* __restrict__ quats, const int* __restrict__ idx,
                              const int* __restrict__ quarter, int B,
                              float* __restrict__ labels6) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= B) return;
  float t[6];
  quat_to_6d(quats + 4 * (size_t)idx[j], t);
  const int k = quarter ? (quarter[j] & 3) : 0;
  for (int u = 0; u < k; ++u) {
    const float a0 = t[0], a1 = t[1], a2 = t[2];
    t[0] = -t[3]; t[1] = -t[4]; t[2] = -t[5];
    t[3] = a0; t[4] = a1; t[5] = a2;
  }
  for (int c = 0; c < 6; ++c) labels6[6 * j + c] = t[c];
}

// loss[j] = min(|o - t|^2, |o + t|^2); go = (2 / B)(o -+ t) of the smaller.
__global__ void loss_kernel(const float* __restrict__ o, const float* __restrict__ t, int B,
                            float* __restrict__ loss, float* __restrict__ go) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= B) return;
  float dp = 0.0f, dm = 0.0f;
  for (int c = 0; c < pn::OUT; ++c) {
    const float a = o[6 * j + c], b = t[6 * j + c];
    dp += (a - b) * (a - b);
    dm += (a + b) * (a + b);
  }
  const float s = dp <= dm ? 1.0f : -1.0f;
  loss[j] = fminf(dp, dm);
  const float f = 2.0f / (float)B;
  for (int c = 0; c < pn::OUT; ++c) go[6 * j + c] = f * (o[6 * j + c] - s * t[6 * j + c]);
}

// Gram-Schmidt of the 6D output to a rotation matrix, then its quaternion
// (Shepperd's method: the largest of 1 + trace and the 1 + 2 m_ii - trace
// picks the stable formula), canonical with w >= 0.
__device__ void six_d_to_quat(const float* o, float* q) {
  float a[3] = {o[0], o[1], o[2]}, b[3] = {o[3], o[4], o[5]};
  float na = sqrtf(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
  if (!(na > 1e-20f)) {
    a[0] = 1.0f; a[1] = 0.0f; a[2] = 0.0f;
    na = 1.0f;
  }
  for (int c = 0; c < 3; ++c) a[c] /= na;
  const float d = a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
  for (int c = 0; c < 3; ++c) b[c] -= d * a[c];
  float nb = sqrtf(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
  if (!(nb > 1e-20f)) {  // any unit vector orthogonal to a
    const int ax = fabsf(a[0]) < 0.9f ? 0 : 1;
    float e[3] = {0.0f, 0.0f, 0.0f};
    e[ax] = 1.0f;
    const float de = a[ax];
    for (int c = 0; c < 3; ++c) b[c] = e[c] - de * a[c];
    nb = sqrtf(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
  }
  for (int c = 0; c < 3; ++c) b[c] /= nb;
  const float r3[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2],
                       a[0] * b[1] - a[1] * b[0]};
  // row-major m with columns a, b, r3
  const float m0 = a[0], m1 = b[0], m2 = r3[0];
  const float m3 = a[1], m4 = b[1], m5 = r3[1];
  const float m6 = a[2], m7 = b[2], m8 = r3[2];
  const float tr = m0 + m4 + m8;
  float w, x, y, z;
  if (tr > 0.0f) {
    const float S = sqrtf(tr + 1.0f) * 2.0f;
    w = 0.25f * S; x = (m7 - m5) / S; y = (m2 - m6) / S; z = (m3 - m1) / S;
  } else if (m0 > m4 && m0 > m8) {
    const float S = sqrtf(1.0f + m0 - m4 - m8) * 2.0f;
    w = (m7 - m5) / S; x = 0.25f * S; y = (m1 + m3) / S; z = (m2 + m6) / S;
  } else if (m4 > m8) {
    const float S = sqrtf(1.0f + m4 - m0 - m8) * 2.0f;
    w = (m2 - m6) / S; x = (m1 + m3) / S; y = 0.25f * S; z = (m5 + m7) / S;
  } else {
    const float S = sqrtf(1.0f + m8 - m0 - m4) * 2.0f;
    w = (m3 - m1) / S; x = (m2 + m6) / S; y = (m5 + m7) / S; z = 0.25f * S;
  }
  const float n = sqrtf(w * w + x * x + y * y + z * z);
  const float sg = w < 0.0f ? -1.0f / n : 1.0f / n;
  q[0] = w * sg; q[1] = x * sg; q[2] = y * sg; q[3] = z * sg;
}

// quats[row][0] = the predicted rotation, quats[row][1] = its Friedel mate
// q (x) (0, 0, 0, 1) = (-z, y, -x, w), both with w >= 0.
__global__ void predict_quats_kernel(const float* __restrict__ o, const int* __restrict__ idx,
                                     int B, float* __restrict__ quats) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= B) return;
  float q[4];
  six_d_to_quat(o + 6 * j, q);
  float* d = quats + 8 * (size_t)idx[j];
  for (int c = 0; c < 4; ++c) d[c] = q[c];
  float m[4] = {-q[3], q[2], -q[1], q[0]};
  const float sg = m[0] < 0.0f ? -1.0f : 1.0f;
  for (int c = 0; c < 4; ++c) d[4 + c] = sg * m[c];
}

__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v, size_t n, float lr_t,
                            float b1, float b2, float eps) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const float ge = g[e];
  const float me = b1 * m[e] + (1.0f - b1) * ge;
  const float ve = b2 * v[e] + (1.0f - b2) * ge * ge;
  m[e] = me;
  v[e] = ve;
  p[e] -= lr_t * me / (sqrtf(ve) + eps);
}

// ------------------------------------------------------------------ host -

static int ensure_cap(ProposalNet* n, int B) {
  emc_ctx* ctx = n->ctx;
  if (B <= n->cap) return EMC_OK;
  for (float** a : {&n->out, &n->g0, &n->g1, &n->gout, &n->loss, &n->labels6}) {
    cudaFree(*a);
    *a = nullptr;
  }
  cudaFree(n->idx);
  n->idx = nullptr;
  cudaFree(n->quarter);
  n->quarter = nullptr;
  for (auto& a : n->act) {
    cudaFree(a);
    a = nullptr;
  }
  n->cap = 0;
  size_t biggest = 0;
  for (int l = 0; l <= pn::NCONV; ++l) {
    const size_t sz = l == 0 ? (size_t)pn::D * pn::D
                             : (size_t)pn::CH * (pn::hin(l - 1) / 2) * (pn::hin(l - 1) / 2);
    EMC_CUDA(ctx, cudaMalloc(&n->act[l], sizeof(float) * sz * B));
    biggest = std::max(biggest, sz);
  }
  EMC_CUDA(ctx, cudaMalloc(&n->out, sizeof(float) * pn::OUT * B));
  EMC_CUDA(ctx, cudaMalloc(&n->gout, sizeof(float) * pn::OUT * B));
  EMC_CUDA(ctx, cudaMalloc(&n->g0, sizeof(float) * biggest * B));
  EMC_CUDA(ctx, cudaMalloc(&n->g1, sizeof(float) * biggest * B));
  EMC_CUDA(ctx, cudaMalloc(&n->loss, sizeof(float) * B));
  EMC_CUDA(ctx, cudaMalloc(&n->idx, sizeof(int) * B));
  EMC_CUDA(ctx, cudaMalloc(&n->quarter, sizeof(int) * B));
  EMC_CUDA(ctx, cudaMalloc(&n->labels6, sizeof(float) * 6 * B));
  n->cap = B;
  return EMC_OK;
}

// More than 48 KB of shared memory per block has to be asked for, once per device.
template <typename Kernel>
static int big_smem(emc_ctx* ctx, Kernel k, int bytes) {
  EMC_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  return EMC_OK;
}

static int conv_smem(emc_ctx* ctx) {
  int rc = big_smem(ctx, conv_fwd_kernel<16>, ConvFwd<16>::SMEM);
  if (!rc) rc = big_smem(ctx, conv_fwd_kernel<8>, ConvFwd<8>::SMEM);
  if (!rc) rc = big_smem(ctx, conv_fwd_kernel<4>, ConvFwd<4>::SMEM);
  if (!rc) rc = big_smem(ctx, conv_bwd_data_kernel<16>, ConvBwd<16>::SMEM);
  if (!rc) rc = big_smem(ctx, conv_bwd_data_kernel<8>, ConvBwd<8>::SMEM);
  if (!rc) rc = big_smem(ctx, conv_bwd_data_kernel<4>, ConvBwd<4>::SMEM);
  if (!rc) rc = big_smem(ctx, conv_wgrad_kernel<16>, ConvWgrad<16>::SMEM);
  if (!rc) rc = big_smem(ctx, conv_wgrad_kernel<8>, ConvWgrad<8>::SMEM);
  if (!rc) rc = big_smem(ctx, conv_wgrad_kernel<4>, ConvWgrad<4>::SMEM);
  return rc;
}

// Convolution l (64 input channels) to HO x HO outputs.
template <int HO>
static int conv_fwd(ProposalNet* n, int l, int B) {
  emc_ctx* ctx = n->ctx;
  conv_fwd_kernel<HO><<<ceil_div(B, ConvFwd<HO>::SPB), 256, ConvFwd<HO>::SMEM, ctx->stream>>>(
      n->act[l], n->params + n->off_w[l], n->params + n->off_b[l], n->act[l + 1], B);
  return after_launch(ctx, "conv_fwd_kernel");
}

static int grow_parts(ProposalNet* n, size_t need) {
  emc_ctx* ctx = n->ctx;
  if (need <= n->wpart_cap) return EMC_OK;
  cudaFree(n->wpart);
  n->wpart = nullptr;
  n->wpart_cap = 0;
  EMC_CUDA(ctx, cudaMalloc(&n->wpart, sizeof(float) * need));
  n->wpart_cap = need;
  return EMC_OK;
}

static int sum_parts(ProposalNet* n, const float* bpart, int S, int nw, int nb, size_t off_w,
                     size_t off_b) {
  emc_ctx* ctx = n->ctx;
  sum_parts_kernel<<<ceil_div(nw + nb, 256), 256, 0, ctx->stream>>>(
      n->wpart, bpart, S, nw, nb, n->grads + off_w, n->grads + off_b);
  return after_launch(ctx, "sum_parts_kernel");
}

// Gradients of convolution l's weights and bias from g (d loss / d act[l + 1]), and
// with gin of its input.
template <int HO>
static int conv_bwd(ProposalNet* n, int l, int B, const float* g, float* gin) {
  emc_ctx* ctx = n->ctx;
  int rc;
  const int groups = pn::CH / pn::CC, per = ceil_div(B, pn::WG_BLOCKS / groups);
  const int S = ceil_div(B, per), K = pn::CH * 9;
  if ((rc = grow_parts(n, (size_t)S * pn::CH * (K + 1)))) return rc;
  float* bpart = n->wpart + (size_t)S * pn::CH * K;
  conv_wgrad_kernel<HO><<<dim3(groups, S), 256, ConvWgrad<HO>::SMEM, ctx->stream>>>(
      g, n->act[l + 1], n->act[l], n->wpart, bpart, B, per);
  if ((rc = after_launch(ctx, "conv_wgrad_kernel"))) return rc;
  if ((rc = sum_parts(n, bpart, S, pn::CH * K, pn::CH, n->off_w[l], n->off_b[l]))) return rc;
  using Bw = ConvBwd<HO>;
  conv_bwd_data_kernel<HO><<<ceil_div(B, Bw::SPB) * Bw::PARTS, 256, Bw::SMEM, ctx->stream>>>(
      g, n->act[l + 1], n->params + n->off_w[l], gin, B);
  return after_launch(ctx, "conv_bwd_data_kernel");
}

// Forward pass of the B samples whose data rows are in n->idx (turned by
// n->quarter when `turned`).
static int forward(ProposalNet* n, int B, bool turned) {
  emc_ctx* ctx = n->ctx;
  int rc;
  const size_t e0 = (size_t)B * 4096;
  gather_rows_kernel<<<(unsigned)((e0 + 255) / 256), 256, 0, ctx->stream>>>(
      n->X, n->idx, turned ? n->quarter : nullptr, B, n->act[0]);
  if ((rc = after_launch(ctx, "gather_rows_kernel"))) return rc;
  conv0_fwd_kernel<<<B * 4, 256, 0, ctx->stream>>>(n->act[0], n->params + n->off_w[0],
                                                  n->params + n->off_b[0], n->act[1]);
  if ((rc = after_launch(ctx, "conv0_fwd_kernel"))) return rc;
  if ((rc = conv_fwd<16>(n, 1, B)) || (rc = conv_fwd<8>(n, 2, B)) || (rc = conv_fwd<4>(n, 3, B)))
    return rc;
  fc_fwd_kernel<<<B, 256, 0, ctx->stream>>>(n->act[pn::NCONV], n->params + n->off_fw,
                                            n->params + n->off_fb, n->out);
  return after_launch(ctx, "fc_fwd_kernel");
}

// Backward pass from n->gout (d loss / d output) into n->grads.
static int backward(ProposalNet* n, int B) {
  emc_ctx* ctx = n->ctx;
  int rc;
  float* gcur = n->g0;  // gradient of act[l + 1] (post-ReLU output of conv l)
  float* gnext = n->g1;
  const int Sf = ceil_div(B, pn::FC_ROWS), nf = pn::OUT * pn::FC_IN;
  if ((rc = grow_parts(n, (size_t)Sf * (nf + pn::OUT)))) return rc;
  float* bpart = n->wpart + (size_t)Sf * nf;
  fc_bwd_kernel<<<dim3(pn::FC_IN / 256, Sf), 256, 0, ctx->stream>>>(
      n->act[pn::NCONV], n->params + n->off_fw, n->gout, B, gcur, n->wpart, bpart);
  if ((rc = after_launch(ctx, "fc_bwd_kernel"))) return rc;
  if ((rc = sum_parts(n, bpart, Sf, nf, pn::OUT, n->off_fw, n->off_fb))) return rc;
  if ((rc = conv_bwd<4>(n, 3, B, gcur, gnext)) || (rc = conv_bwd<8>(n, 2, B, gnext, gcur)) ||
      (rc = conv_bwd<16>(n, 1, B, gcur, gnext)))
    return rc;
  const int per = ceil_div(B, pn::WG_BLOCKS), S = ceil_div(B, per);
  if ((rc = grow_parts(n, (size_t)S * pn::CH * 10))) return rc;
  bpart = n->wpart + (size_t)S * pn::CH * 9;
  conv0_wgrad_kernel<<<S, 256, 0, ctx->stream>>>(gnext, n->act[1], n->act[0], n->wpart, bpart, B,
                                                 per);
  if ((rc = after_launch(ctx, "conv0_wgrad_kernel"))) return rc;
  return sum_parts(n, bpart, S, pn::CH * 9, pn::CH, n->off_w[0], n->off_b[0]);
}

// Loss of the batch in n->idx against labels (quaternions, data rows) and
// its gradient in n->grads; *h_loss = mean loss.
static int loss_and_grads(ProposalNet* n, int B, const float* d_quats, float* h_loss,
                          bool turned) {
  emc_ctx* ctx = n->ctx;
  int rc;
  if ((rc = forward(n, B, turned))) return rc;
  labels_kernel<<<ceil_div(B, 128), 128, 0, ctx->stream>>>(d_quats, n->idx,
                                                            turned ? n->quarter : nullptr, B,
                                                            n->labels6);
  if ((rc = after_launch(ctx, "labels_kernel"))) return rc;
  loss_kernel<<<ceil_div(B, 128), 128, 0, ctx->stream>>>(n->out, n->labels6, B, n->loss,
                                                          n->gout);
  if ((rc = after_launch(ctx, "loss_kernel"))) return rc;
  if ((rc = backward(n, B))) return rc;
  if (h_loss) {
    std::vector<float> l(B);
    EMC_CUDA(ctx, cudaMemcpyAsync(l.data(), n->loss, sizeof(float) * B, cudaMemcpyDeviceToHost,
                                  ctx->stream));
    EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    double s = 0.0;
    for (float v : l) s += v;
    *h_loss = (float)(s / B);
  }
  return EMC_OK;
}

// splitmix64 stream for weight initialisation and shuffles.
struct Mix64 {
  uint64_t s;
  uint64_t next() {
    uint64_t z = (s += 0x9e3779b97f4a7c15ULL);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
  }
  double uniform() { return (double)(next() >> 11) * (1.0 / 9007199254740992.0); }
};

}  // namespace emc

using namespace emc;

struct emc_proposal : ProposalNet {};

extern "C" int emc_proposal_create(emc_ctx* ctx, unsigned long long seed, emc_proposal** out) {
  if (!ctx || !out) return EMC_ERR_INVALID;
  emc_proposal* n = new emc_proposal();
  n->ctx = ctx;
  if (const int rc = conv_smem(ctx)) {
    delete n;
    return rc;
  }
  size_t o = 0;
  for (int l = 0; l < pn::NCONV; ++l) {
    n->off_w[l] = o;
    o += (size_t)pn::CH * pn::cin(l) * 9;
    n->off_b[l] = o;
    o += pn::CH;
  }
  n->off_fw = o;
  o += (size_t)pn::OUT * pn::FC_IN;
  n->off_fb = o;
  o += pn::OUT;
  n->n_params = o;
  // He-uniform weights (bound sqrt(6 / fan_in)), zero biases
  std::vector<float> h(o, 0.0f);
  Mix64 rng{seed ^ 0x5851f42d4c957f2dULL};
  for (int l = 0; l < pn::NCONV; ++l) {
    const double bound = std::sqrt(6.0 / (pn::cin(l) * 9.0));
    for (size_t e = 0; e < (size_t)pn::CH * pn::cin(l) * 9; ++e)
      h[n->off_w[l] + e] = (float)((2.0 * rng.uniform() - 1.0) * bound);
  }
  const double fb = std::sqrt(3.0 / pn::FC_IN);
  for (size_t e = 0; e < (size_t)pn::OUT * pn::FC_IN; ++e)
    h[n->off_fw + e] = (float)((2.0 * rng.uniform() - 1.0) * fb);
  cudaError_t e = cudaMalloc(&n->params, sizeof(float) * o);
  if (e == cudaSuccess) e = cudaMalloc(&n->grads, sizeof(float) * o);
  if (e == cudaSuccess) e = cudaMalloc(&n->adam_m, sizeof(float) * o);
  if (e == cudaSuccess) e = cudaMalloc(&n->adam_v, sizeof(float) * o);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(n->params, h.data(), sizeof(float) * o, cudaMemcpyHostToDevice,
                        ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(n->adam_m, 0, sizeof(float) * o, ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(n->adam_v, 0, sizeof(float) * o, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) {
    const int rc = cuda_fail(ctx, e, "proposal_create");
    emc_proposal_destroy(n);
    return rc;
  }
  *out = n;
  return EMC_OK;
}

extern "C" int emc_proposal_destroy(emc_proposal* n) {
  if (!n) return EMC_OK;
  if (n->ctx) cudaStreamSynchronize(n->ctx->stream);
  for (float* a : {n->params, n->grads, n->adam_m, n->adam_v, n->X, n->out, n->g0, n->g1,
                   n->gout, n->wpart, n->loss, n->labels6, n->stats})
    cudaFree(a);
  for (auto& a : n->act) cudaFree(a);
  cudaFree(n->idx);
  cudaFree(n->quarter);
  delete n;
  return EMC_OK;
}

extern "C" int emc_proposal_param_count(const emc_proposal* n) {
  return n ? (int)n->n_params : 0;
}

extern "C" int emc_proposal_params(emc_proposal* n, float* h_params, int get) {
  if (!n || !h_params) return EMC_ERR_INVALID;
  emc_ctx* ctx = n->ctx;
  const size_t bytes = sizeof(float) * n->n_params;
  if (get) {
    EMC_CUDA(ctx, cudaMemcpyAsync(h_params, n->params, bytes, cudaMemcpyDeviceToHost, ctx->stream));
  } else {
    EMC_CUDA(ctx, cudaMemcpyAsync(n->params, h_params, bytes, cudaMemcpyHostToDevice, ctx->stream));
    EMC_CUDA(ctx, cudaMemsetAsync(n->adam_m, 0, bytes, ctx->stream));
    EMC_CUDA(ctx, cudaMemsetAsync(n->adam_v, 0, bytes, ctx->stream));
    n->adam_t = 0;
  }
  EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return EMC_OK;
}

extern "C" int emc_proposal_set_data(emc_proposal* n, const float* d_images, const int* d_mask,
                                     int side, int n_images, int fit_stats) {
  if (!n) return EMC_ERR_INVALID;
  emc_ctx* ctx = n->ctx;
  EMC_REQUIRE(ctx, d_images && d_mask && n_images > 0, "proposal_set_data: bad arguments");
  EMC_REQUIRE(ctx, fit_stats || n->have_stats,
              "proposal_set_data: no input statistics yet (fit them on the training data)");
  EMC_REQUIRE(ctx, side >= pn::D && side % pn::D == 0,
              "proposal_set_data: side %d is not a multiple of 64", side);
  if (n_images > n->n_data) {
    cudaFree(n->X);
    n->X = nullptr;
    n->n_data = 0;
    EMC_CUDA(ctx, cudaMalloc(&n->X, sizeof(float) * 4096 * (size_t)n_images));
  }
  n->n_data = n_images;
  proposal_inputs_kernel<<<n_images, 256, 0, ctx->stream>>>(d_images, d_mask, side, n_images,
                                                             n->X);
  int rc = after_launch(ctx, "proposal_inputs_kernel");
  if (rc) return rc;
  if (!n->stats) EMC_CUDA(ctx, cudaMalloc(&n->stats, sizeof(float) * 2 * 4096));
  if (fit_stats) {
    input_stats_kernel<<<16, 256, 0, ctx->stream>>>(n->X, n_images, n->stats);
    if ((rc = after_launch(ctx, "input_stats_kernel"))) return rc;
    n->have_stats = true;
  }
  const size_t e = (size_t)n_images * 4096;
  standardize_kernel<<<(unsigned)((e + 255) / 256), 256, 0, ctx->stream>>>(n->X, n_images,
                                                                          n->stats);
  return after_launch(ctx, "standardize_kernel");
}

extern "C" int emc_proposal_stats(emc_proposal* n, float* h_stats, int get) {
  if (!n || !h_stats) return EMC_ERR_INVALID;
  emc_ctx* ctx = n->ctx;
  if (!n->stats) EMC_CUDA(ctx, cudaMalloc(&n->stats, sizeof(float) * 2 * 4096));
  if (get) {
    EMC_REQUIRE(ctx, n->have_stats, "proposal_stats: none fitted");
    EMC_CUDA(ctx, cudaMemcpyAsync(h_stats, n->stats, sizeof(float) * 8192, cudaMemcpyDeviceToHost,
                                  ctx->stream));
  } else {
    EMC_CUDA(ctx, cudaMemcpyAsync(n->stats, h_stats, sizeof(float) * 8192, cudaMemcpyHostToDevice,
                                  ctx->stream));
    n->have_stats = true;
  }
  EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return EMC_OK;
}

extern "C" int emc_proposal_inputs(emc_proposal* n, int first, int count, float* h_out) {
  if (!n || !h_out) return EMC_ERR_INVALID;
  emc_ctx* ctx = n->ctx;
  EMC_REQUIRE(ctx, first >= 0 && count >= 0 && first + count <= n->n_data,
              "proposal_inputs: rows out of range");
  EMC_CUDA(ctx, cudaMemcpyAsync(h_out, n->X + (size_t)first * 4096, sizeof(float) * 4096 * count,
                                cudaMemcpyDeviceToHost, ctx->stream));
  EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return EMC_OK;
}

extern "C" int emc_proposal_loss_grad(emc_proposal* n, const int* h_rows, int B,
                                      const float* d_quats, float* h_loss, float* h_grads) {
  if (!n) return EMC_ERR_INVALID;
  emc_ctx* ctx = n->ctx;
  EMC_REQUIRE(ctx, h_rows && B > 0 && d_quats && n->X, "proposal_loss_grad: bad arguments");
  for (int j = 0; j < B; ++j)
    EMC_REQUIRE(ctx, h_rows[j] >= 0 && h_rows[j] < n->n_data, "proposal_loss_grad: bad row");
  int rc = ensure_cap(n, B);
  if (rc) return rc;
  EMC_CUDA(ctx, cudaMemcpyAsync(n->idx, h_rows, sizeof(int) * B, cudaMemcpyHostToDevice,
                                ctx->stream));
  if ((rc = loss_and_grads(n, B, d_quats, h_loss, false))) return rc;
  if (h_grads)
    EMC_CUDA(ctx, cudaMemcpyAsync(h_grads, n->grads, sizeof(float) * n->n_params,
                                  cudaMemcpyDeviceToHost, ctx->stream));
  EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return EMC_OK;
}

extern "C" int emc_proposal_train(emc_proposal* n, const float* d_quats, const int* h_rows,
                                  int n_rows, int epochs, int batch, float lr,
                                  unsigned long long seed, int augment, float* h_epoch_loss) {
  if (!n) return EMC_ERR_INVALID;
  emc_ctx* ctx = n->ctx;
  EMC_REQUIRE(ctx, d_quats && n->X && epochs >= 0 && batch > 0 && lr > 0.0f,
              "proposal_train: bad arguments");
  std::vector<int> rows;
  if (h_rows) {
    rows.assign(h_rows, h_rows + n_rows);
    for (int r : rows)
      EMC_REQUIRE(ctx, r >= 0 && r < n->n_data, "proposal_train: row %d out of range", r);
  } else {
    rows.resize(n->n_data);
    for (int j = 0; j < n->n_data; ++j) rows[j] = j;
  }
  EMC_REQUIRE(ctx, !rows.empty(), "proposal_train: no rows");
  int rc = ensure_cap(n, batch);
  if (rc) return rc;
  Mix64 rng{seed};
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  std::vector<int> stage(batch), quarter(batch);
  const long long total_steps = (long long)epochs * (long long)ceil_div((int)rows.size(), batch);
  long long step = 0;
  for (int ep = 0; ep < epochs; ++ep) {
    for (size_t j = rows.size(); j > 1; --j) {  // Fisher-Yates
      const size_t k = (size_t)(rng.next() % j);
      std::swap(rows[j - 1], rows[k]);
    }
    double sum = 0.0;
    size_t seen = 0;
    for (size_t s0 = 0; s0 < rows.size(); s0 += batch) {
      const int B = (int)std::min<size_t>(batch, rows.size() - s0);
      std::copy(rows.begin() + s0, rows.begin() + s0 + B, stage.begin());
      for (int j = 0; j < B; ++j) quarter[j] = augment ? (int)(rng.next() >> 62) : 0;
      EMC_CUDA(ctx, cudaMemcpyAsync(n->idx, stage.data(), sizeof(int) * B, cudaMemcpyHostToDevice,
                                    ctx->stream));
      EMC_CUDA(ctx, cudaMemcpyAsync(n->quarter, quarter.data(), sizeof(int) * B,
                                    cudaMemcpyHostToDevice, ctx->stream));
      // pageable sources are staged before the calls return; the next batch
      // overwrites them only after that
      float l = 0.0f;
      if ((rc = loss_and_grads(n, B, d_quats, h_epoch_loss ? &l : nullptr, true))) return rc;
      sum += (double)l * B;
      seen += B;
      ++n->adam_t;
      const double c1 = 1.0 - std::pow((double)b1, (double)n->adam_t);
      const double c2 = 1.0 - std::pow((double)b2, (double)n->adam_t);
      // cosine decay of the step size over this call, to 5 % at its end
      const double prog = (double)(step++) / (double)std::max<long long>(1, total_steps - 1);
      const double sched = 0.05 + 0.95 * 0.5 * (1.0 + std::cos(M_PI * prog));
      const float lr_t = (float)(lr * sched * std::sqrt(c2) / c1);
      adam_kernel<<<(unsigned)((n->n_params + 255) / 256), 256, 0, ctx->stream>>>(
          n->params, n->grads, n->adam_m, n->adam_v, n->n_params, lr_t, b1, b2, eps);
      if ((rc = after_launch(ctx, "adam_kernel"))) return rc;
    }
    if (h_epoch_loss) h_epoch_loss[ep] = (float)(sum / (double)seen);
  }
  EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return EMC_OK;
}

extern "C" int emc_proposal_predict(emc_proposal* n, float* d_quats_out) {
  if (!n) return EMC_ERR_INVALID;
  emc_ctx* ctx = n->ctx;
  EMC_REQUIRE(ctx, d_quats_out && n->X, "proposal_predict: bad arguments");
  const int B = 1024;
  int rc = ensure_cap(n, B);
  if (rc) return rc;
  std::vector<int> stage(B);
  for (int s0 = 0; s0 < n->n_data; s0 += B) {
    const int cnt = std::min(B, n->n_data - s0);
    for (int j = 0; j < cnt; ++j) stage[j] = s0 + j;
    EMC_CUDA(ctx, cudaMemcpyAsync(n->idx, stage.data(), sizeof(int) * cnt, cudaMemcpyHostToDevice,
                                  ctx->stream));
    if ((rc = forward(n, cnt, false))) return rc;
    predict_quats_kernel<<<ceil_div(cnt, 128), 128, 0, ctx->stream>>>(n->out, n->idx, cnt,
                                                                      d_quats_out);
    if ((rc = after_launch(ctx, "predict_quats_kernel"))) return rc;
    EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));  // `stage` is reused
  }
  return EMC_OK;
}
