// Tensor-core (tcgen05 + TMA) E-step and M-step of the fused iteration.
//
// E-step.  For a tile of patterns (M, one TMEM lane each) x 128 rotations (N)
// the reference's "poisson" likelihood with per-pair scaling (emc_cuda.cu:
// 196-216, 438-454) is expanded into four sums over the compacted pixels,
//   num = sum k^2 [s > 1e-10]        den = sum k s [s > 1e-10]
//   B   = sum k s/(s+c) [s > 0]      C   = sum k^2 /(s+c) [s > 0]
// so that with 1/phi = den/num:  S_ri = A_r - 2 B/phi + C/phi^2  and
// L_ri = log w_r - S_ri / (2 count_r sigma^2).  They come from contractions of
// the counts (exact in FP16, with k (k - 1) as two FP16 terms) with M'S, with
// H = 1/(s+c) and, where a slice has invalid pixels, with their indicator; the
// section below says how.  The epilogue forms L and phi, stores them coalesced
// along patterns, and keeps a running (max, sum exp) per pattern over the
// tile's rotations: the per-tile LSE partials that the FP64 normaliser
// combines.
//
// M-step.  U = Q K^T over the patterns for a tile of 128 (a pair of CTAs: 256)
// rotations x 256 pixels, Q = P / phi as FP16 hi (or hi + lo) with a per-rotation
// power-of-two scale, K the exact FP16 counts; the epilogue inserts U, which is T_r
// times the slice, at the rotated pixel (nearest or trilinear) with weight T_r -- the
// slice never reaches HBM (emc_atomic.cu:88-132, 183-200).
//
// Pipeline: one warp (three in the reference likelihood) issues TMA loads into a
// ring of shared-memory stages (mbarrier full/empty handshake), the next owns TMEM
// and issues tcgen05.mma from one elected lane, sixteen run the epilogue.  Every
// wait is bounded and reports through a device status word (EMC_ERR_TIMEOUT on the
// host).
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "geometry.cuh"
#include "plan.cuh"
#include "ptx.cuh"

namespace emc {

// ------------------------------------------------------- tensor maps -----
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// Row-major FP16 matrix [rows][cols] (cols contiguous), tiles of
// box_rows x box_cols, 64B or 128B swizzle (box_cols * 2 == swizzle span).
static int make_map(emc_ctx* ctx, CUtensorMap* map, const void* base, uint64_t rows,
                    uint64_t cols, uint32_t box_rows, uint32_t box_cols) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(ctx, EMC_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  if (((uintptr_t)base & 15) || ((cols * 2) & 15))
    return fail(ctx, EMC_ERR_INTERNAL, "tensor map: misaligned base or pitch");
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * 2};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  const CUtensorMapSwizzle sw =
      box_cols * 2 == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(ctx, EMC_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return EMC_OK;
}

// ---------------------------------------------------- pattern operands ---

// Counts -> FP16 operand, rows of Kp (patterns padded to Np with zeros):
// Kh = fp16(k) (k itself up to 2048; larger counts rounded to 11 significant
// bits) times the power of two `scale`, exactly.
__global__ void tc_pattern_ops_kernel(const float* __restrict__ images, const int* __restrict__ pix,
                                      int n2, int N, int Kp, __half* __restrict__ Kh,
                                      const int* __restrict__ perm, float scale) {
  // one block per (pattern row, 256 pixels), pixel blocks the fast index
  const int nqb = (Kp + 255) / 256;
  const int i = (int)(blockIdx.x / nqb);
  const int q = (int)(blockIdx.x % nqb) * 256 + threadIdx.x;
  if (q >= Kp) return;
  float k = 0.0f;
  if (i < N) {
    const int p = pix[q];
    if (p >= 0) k = __ldg(images + (size_t)(perm ? perm[i] : i) * n2 + p);
  }
  Kh[(size_t)i * Kp + q] = __float2half_rn(__half2float(__float2half_rn(k)) * scale);
}

namespace es {  // bits of a (128-pattern tile, 64-pixel block) in blk_bits and the lists
constexpr uint32_t kJ = 1;    // a count above 1
constexpr uint32_t kJlo = 2;  // k (k - 1) has a second FP16 term
constexpr uint32_t kHlo = 4;  // lists: before the count tail, K . H takes H's lo half
constexpr uint32_t kAny = 8;  // a count
}  // namespace es

// bits[pt][kb] of the block, and in blocks with a count above 1 the operand
// j = k (k - 1) as FP16 hi (and lo where some term needs it).  One CTA per block
// of two pattern tiles: a pair of CTAs multiplies both where one needs it, so
// j is written for both.  256 rows x 128 B, eight 16-byte loads a thread.
__global__ void __launch_bounds__(256) tc_count_blocks_kernel(
    const __half* __restrict__ Kh, int Kp, int nkb, int n_pt, float scale,
    __half* __restrict__ Jh, __half* __restrict__ Jl, unsigned char* __restrict__ bits,
    unsigned char* __restrict__ sub_any) {
  const int kb = blockIdx.x, pt0 = 2 * blockIdx.y;
  const int nt = min(2, n_pt - pt0);
  const float inv = 1.0f / scale;
  union V {
    uint4 u;
    __half h[8];
  } v[2][4];
  int any[2] = {0, 0}, two[2] = {0, 0}, low[2] = {0, 0};
  int sub[2][2] = {};  // of the tile's two halves of 64 patterns
  auto at = [&](int t, int j) {
    const int e = threadIdx.x + 256 * j;
    return (size_t)((pt0 + t) * 128 + (e >> 3)) * Kp + kb * 64 + (e & 7) * 8;
  };
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    if (t >= nt) break;
#pragma unroll
    for (int j = 0; j < 4; ++j) v[t][j].u = *reinterpret_cast<const uint4*>(Kh + at(t, j));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      sub[t][j >> 1] |= (v[t][j].u.x | v[t][j].u.y | v[t][j].u.z | v[t][j].u.w) != 0;
#pragma unroll
      for (int c = 0; c < 8; ++c) two[t] |= __half2float(v[t][j].h[c]) * inv > 1.0f;
    }
  }
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    sub[t][0] = __syncthreads_or(sub[t][0]);
    sub[t][1] = __syncthreads_or(sub[t][1]);
    any[t] = sub[t][0] | sub[t][1];
    two[t] = __syncthreads_or(two[t]);
  }
  if ((two[0] | two[1]) && Jh) {
    V lo[2][4];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (t >= nt) break;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        V hi;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float k = __half2float(v[t][j].h[c]) * inv;
          const float x = k * (k - 1.0f) * scale;
          hi.h[c] = __float2half_rn(x);
          lo[t][j].h[c] = __float2half_rn(x - __half2float(hi.h[c]));
          low[t] |= __half2float(lo[t][j].h[c]) != 0.0f;
        }
        *reinterpret_cast<uint4*>(Jh + at(t, j)) = hi.u;
      }
    }
    low[0] = __syncthreads_or(low[0]);
    low[1] = __syncthreads_or(low[1]);
    if (low[0] | low[1])
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (t >= nt) break;
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(Jl + at(t, j)) = lo[t][j].u;
      }
  }
  if (threadIdx.x < 2 * nt) {
    const int t = threadIdx.x >> 1, h = threadIdx.x & 1;
    sub_any[(size_t)kb * (2 * n_pt) + 2 * pt0 + threadIdx.x] = (unsigned char)(
        (t ? (h ? sub[1][1] : sub[1][0]) : (h ? sub[0][1] : sub[0][0])) != 0);
  }
  if (threadIdx.x < nt) {
    const int t = threadIdx.x;
    bits[(size_t)(pt0 + t) * nkb + kb] = (unsigned char)(
        ((t ? any[1] : any[0]) ? es::kAny : 0u) | ((t ? two[1] : two[0]) ? es::kJ : 0u) |
        ((t ? low[1] : low[0]) ? es::kJlo : 0u));
  }
}

// One warp per pattern row n: ktot = sum k and k2tot = sum k^2 (integers, then
// rounded once), and the last 64-pixel block b whose suffix (blocks b ..) still
// holds more than eps of the row's counts: lo_kb[n / 128] (zeroed before)
// becomes the largest b + 1 over the tile's rows, lo_kb[n_pt] the largest of
// all.  bright (zeroed before) is set where k2tot is not exact in FP32 or a count's
// k (k - 1) not in two FP16 terms.  Lane l takes a contiguous run of blocks: run sums, a warp prefix scan,
// then a second walk over its run.
__global__ void __launch_bounds__(256) tc_count_rows_kernel(const __half* __restrict__ Kh, int Kp,
                                                            int nkb, int N, float scale, float eps,
                                                            float* __restrict__ ktot,
                                                            float* __restrict__ k2tot,
                                                            int* __restrict__ lo_kb,
                                                            int* __restrict__ bright) {
  const int n = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (n >= N) return;  // whole warps
  const float inv = 1.0f / scale;
  const __half* k = Kh + (size_t)n * Kp;
  const int per = (nkb + 31) / 32;
  const int b0 = min(lane * per, nkb), b1 = min(b0 + per, nkb);
  unsigned most = 0;
  auto block = [&](int b, unsigned long long& s2) {  // the block's sum of k; k^2 added to s2
    const uint4* v = reinterpret_cast<const uint4*>(k + 64 * (size_t)b);
    unsigned s = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint4 u = v[j];
      if ((u.x | u.y | u.z | u.w) == 0) continue;
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[h]));
        const unsigned x = (unsigned)(f.x * inv), y = (unsigned)(f.y * inv);
        s += x + y;
        most = max(most, max(x, y));
        s2 += (unsigned long long)x * x + (unsigned long long)y * y;
      }
    }
    return s;
  };
  unsigned long long s2 = 0, dummy = 0, c = 0;
  for (int b = b0; b < b1; ++b) c += block(b, s2);
  unsigned long long incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  most = __reduce_max_sync(0xffffffffu, most);
  const unsigned long long total = __shfl_sync(0xffffffffu, incl, 31);
  const float lim = eps * (float)total;
  unsigned long long pre = incl - c;  // the counts of the blocks before b0
  int last = -1;
  for (int b = b0; b < b1; ++b) {
    if ((float)(total - pre) > lim) last = b;  // the suffix from b
    pre += block(b, dummy);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
  if (lane == 0) {
    ktot[n] = (float)total;
    k2tot[n] = (float)s2;
    if (s2 >= 1ull << 24 || most > 2048u) *bright = 1;  // races store the same value
    if (last >= 0) {
      atomicMax(lo_kb + n / 128, last + 1);
      atomicMax(lo_kb + (N + 127) / 128, last + 1);
    }
  }
}

// First n_qt warps: the M-step's lists.  Then list i < n_pt: the blocks of pattern
// tile i; list n_pt + i: those of tiles 2 i and 2 i + 1 together.  One warp each.
// A tile without counts keeps block 0, so that its accumulators are written.  The
// last warps: live[kb].
__global__ void __launch_bounds__(32) tc_block_lists_kernel(
    const unsigned char* __restrict__ bits, int n_pt, int nkb, const int* __restrict__ lo_kb,
    uint32_t* __restrict__ pt_list, int* __restrict__ pt_n, uint32_t* __restrict__ pp_list,
    int* __restrict__ pp_n, unsigned char* __restrict__ live,
    const unsigned char* __restrict__ sub_any, int n_qt, unsigned char* __restrict__ ms_map,
    int* __restrict__ ms_list, int* __restrict__ ms_n) {
  const int lane = threadIdx.x, n_pp = (n_pt + 1) / 2;
  int i = blockIdx.x;
  if (i < n_qt) {  // the M-step's list of pixel tile i
    const int nb = 2 * n_pt;
    int n = 0;
    for (int b0 = 0; b0 < nb; b0 += 32) {
      const int b = b0 + lane;
      int any = 0;
      for (int k = 4 * i; k < min(4 * i + 4, nkb); ++k)
        any |= b < nb ? sub_any[(size_t)k * nb + b] : 0;
      const unsigned on = __ballot_sync(0xffffffffu, any);
      if (b < nb) ms_map[(size_t)i * nb + b] = (unsigned char)any;
      if (any) ms_list[(size_t)i * nb + n + __popc(on & ((1u << lane) - 1u))] = b;
      n += __popc(on);
    }
    if (n == 0 && lane == 0) ms_list[(size_t)i * nb] = 0;
    if (lane == 0) ms_n[i] = max(n, 1);
    return;
  }
  i -= n_qt;
  if (i >= n_pt + n_pp) {
    const int kb = (i - n_pt - n_pp) * 32 + lane;
    if (kb >= nkb) return;
    int any = 0;
    for (int t = 0; t < n_pt; ++t) any |= bits[(size_t)t * nkb + kb] & es::kAny;
    live[kb] = any || kb == 0;
    return;
  }
  const bool pair = i >= n_pt;
  if (pair) i -= n_pt;
  const int t0 = pair ? 2 * i : i, t1 = pair ? min(2 * i + 1, n_pt - 1) : i;
  uint32_t* list = (pair ? pp_list : pt_list) + (size_t)i * nkb;
  const int end = lo_kb ? max(lo_kb[t0], lo_kb[t1]) : 0;
  int n = 0;
  for (int kb0 = 0; kb0 < nkb; kb0 += 32) {
    const int kb = kb0 + lane;
    uint32_t b = 0;
    if (kb < nkb) b = bits[(size_t)t0 * nkb + kb] | bits[(size_t)t1 * nkb + kb];
    const unsigned on = __ballot_sync(0xffffffffu, (b & es::kAny) != 0);
    if (b & es::kAny)
      list[n + __popc(on & ((1u << lane) - 1u))] =
          (uint32_t)kb << 8 | (b & (es::kJ | es::kJlo)) | (kb < end ? es::kHlo : 0u);
    n += __popc(on);
  }
  if (n == 0 && lane == 0) list[0] = 0;
  if (lane == 0) (pair ? pp_n : pt_n)[i] = max(n, 1);
}

// [rows][cols] -> [cols][rows], FP16: 64 x 64 tiles, moved with 4-byte
// (half2) loads and stores where two neighbouring elements are in range.
__global__ void transpose_h_kernel(const __half* __restrict__ in, int rows, int cols,
                                   __half* __restrict__ out) {
  __shared__ __half t[64][66];
  const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64;
  const int x2 = 2 * threadIdx.x;
  for (int y = threadIdx.y; y < 64; y += blockDim.y) {
    const int r = r0 + y, c = c0 + x2;
    __half a = __float2half_rn(0.f), b = a;
    if (r < rows) {
      if (c + 1 < cols && (cols & 1) == 0) {
        const __half2 v = *reinterpret_cast<const __half2*>(in + (size_t)r * cols + c);
        a = __low2half(v);
        b = __high2half(v);
      } else {
        if (c < cols) a = in[(size_t)r * cols + c];
        if (c + 1 < cols) b = in[(size_t)r * cols + c + 1];
      }
    }
    t[y][x2] = a;
    t[y][x2 + 1] = b;
  }
  __syncthreads();
  for (int y = threadIdx.y; y < 64; y += blockDim.y) {
    const int c = c0 + y, r = r0 + x2;
    if (c >= cols) continue;
    if (r + 1 < rows && (rows & 1) == 0) {
      *reinterpret_cast<__half2*>(out + (size_t)c * rows + r) = __halves2half2(t[x2][y], t[x2 + 1][y]);
    } else {
      if (r < rows) out[(size_t)c * rows + r] = t[x2][y];
      if (r + 1 < rows) out[(size_t)c * rows + r + 1] = t[x2 + 1][y];
    }
  }
}

// ------------------------------------------------------------ E-step -----
// num, den, B and C from contractions with H = 1/(s + c) only: with I = [s <= 0]
// (H = 0 there), J = k (k - 1) and s/(s+c) = 1 - c/(s+c),
//   den = K . (M'S)^T                  B   = k_tot - n_1 - c (K . H^T)
//   C   = K . H^T + J . H^T            num = k2_tot - n_1 - n_J
//   n_1 = K . I^T                      n_J = J . I^T
// with k_tot and k2_tot summed exactly at bind (a pixel with 0 < s < 1e-10
// counts in B and C but not in num: its k^2 is added to n_J through a plane T).
// These are differences of whole numbers, exact while sum k^2 stays below 2^24 and
// the counts below 2,049 (k (k - 1) in 22 bits).  Where some pattern of the plan
// exceeds that (a beam spot or hot pixels, which may lie outside every slice) the
// differences would keep rounding of what they take out, so the plane of I holds V =
// [s >= 1e-10] instead, and a tile with an invalid pixel sums what is covered:
//   num = K . V^T + J . V^T      B = K . V^T + K . T^T - c (K . H^T)
// over all its blocks, K . V^T and K . T^T in n_1's columns and num in n_J's.
// (A tile without invalid pixels takes nothing out, and keeps k_tot and k2_tot.)
// What each 64-pixel block of a pattern tile needs is decided at bind too:
// nothing where no pattern of the tile counts, K x [M'S | H] where every count
// is 0 or 1 (J = 0), J x H where one is larger, the products with I only where
// the rotation tile has an invalid pixel.  The four-contraction form multiplied
// K and K^2 by four operands on every block: at 128^3 x 20,000 patterns of 5,000
// photons 4.4 products of 128 columns per block, 1.1 to 2.3 here.
//
// TMEM has room for four of the five sums: den and K.H in columns 0-255, n_1 and
// J.H in 256-383 and 384-511.  Where a tile needs n_J, J x H and J x I run first
// (pass A): J.H stays where it is, and the epilogue warps move n_J, whose columns
// n_1 takes, out into the tile's own part of L, which they overwrite at the end
// (with J x [H | I] as one product both sums had to go: 7,795 -> 7,620 us at 128^3
// with 80 photons per pattern, 17,790 -> 17,450 with 5,000, 2,332 -> 2,263 at 96^3).
// One CTA owns 128 patterns x 128 rotations, or (PAIR) a cluster of
// two 256 x 128 with 256-row MMAs issued by rank 0: each CTA then holds its own
// 128 patterns and 64 of the 128 rows of every rotation operand, [M'S | H] side by
// side, so the columns of that 256-column product come in
// quarters (den 0-63, K.H 0-63, den 64-127, K.H 64-127).  Per 64-pixel block and
// CTA that is 32 KB for a 256 x 256 x 64 product (the M-step's ratio).
//
// The passes: A as above; C, K x H's lo half on the blocks before the count tail;
// B, K x [M'S | H], K x I and, in tiles without pass A, J x H.  The tensor core
// cuts a sum's last bits off at every addition, so small terms come first: C
// before B, and every pass from the dim outer blocks to the bright inner ones,
// which keeps the sums small for most of their additions.  Every stage of
// a tile has the same places in shared memory (six slots of 32 KB to four of 56
// KB on a pair), so that the threads that issue loads and products spend few
// instructions on a stage: a plain block's products take 512 clocks, and
// working out places for stages of many shapes took 750.  For the same reason
// 256-column products are preferred: four issue in 370 clocks, whatever their
// width, and run 512 (256 at 128 columns).
namespace es {
constexpr int BM = 128;        // patterns per tile (TMEM lanes)
constexpr int BN = 128;        // rotations per tile
constexpr int BK = 64;         // pixels per stage (128 B rows, 128B swizzle)
constexpr int CHUNK = 8192;    // 64 rows of one operand
constexpr int CHUNKS = 27;
constexpr int NB = 8;          // slots at most
// A thread takes over 100 clocks for each TMA load it issues: one producer for
// the three to six loads of a stage would set the pace, so three warps share them.
constexpr int PRODUCERS = 3;   // pattern side | first | second rotation operand
constexpr int MMA_WARP = PRODUCERS, EPI_WARP0 = PRODUCERS + 1;
constexpr int EPI_WARPS = 16;  // four per TMEM lane quarter, 32 columns each
constexpr int EPI_PARTS = EPI_WARPS / 4;
constexpr int THREADS = 32 * (EPI_WARP0 + EPI_WARPS);
static_assert(EPI_WARP0 % 4 == 0, "epilogue warp w reads TMEM lane quarter w % 4");
// The block list with the rotation tile's flags is put together in shared
// memory before the loop.  Entries beyond kList (more than 70,400 pixels with
// counts) are read from global memory.
constexpr int kList = 1100;
constexpr uint32_t kInv = 16, kTiny = 32;  // flags of the rotation tile in an entry
constexpr uint32_t kNJ = 64;               // of all entries: the tile needs n_J
// barriers, per-rotation rows (128 float4), epilogue parts, list
constexpr int EXTRA = 256 + BN * 16 + (EPI_PARTS - 1) * BM * 8 + kList * 4 + 16;
constexpr int SMEM_BYTES = CHUNKS * CHUNK + EXTRA + 1024;
static_assert(SMEM_BYTES <= 232448, "shared memory of the likelihood kernel");
}  // namespace es

// Tile of CTA b in a grouped raster over n_pt pattern tiles x n_rt rotation
// tiles.  raster > 0: groups of `raster` rotation tiles, each group visiting
// the pattern tiles in turn (the group's rotation panels are read by
// consecutive CTAs); raster < 0: groups of -raster pattern tiles visiting the
// rotation tiles in turn.
__device__ __forceinline__ void raster_tile(int b, int raster, int n_pt, int n_rt, int& pt,
                                            int& rt) {
  if (raster > 0) {
    const int per_group = raster * n_pt;
    const int g = b / per_group, within = b % per_group;
    const int rt0 = g * raster;
    const int gsz = min(raster, n_rt - rt0);
    rt = rt0 + within % gsz;
    pt = within / gsz;
  } else {
    const int G = -raster;
    const int per_group = G * n_rt;
    const int g = b / per_group, within = b % per_group;
    const int pt0 = g * G;
    const int gsz = min(G, n_pt - pt0);
    pt = pt0 + within % gsz;
    rt = within / gsz;
  }
}

struct TcEstepArgs {
  int N, R, n_pt, n_rt, nkb;
  int raster;                     // tile order (raster_tile)
  int tile0;                      // CTA b runs tile tile0 + b of the order
  int gh_lo;                      // H lo: bit 0 in K.H before the tail, bit 1 everywhere
  const int2* tiles;              // pruned iteration: (pattern tile, rotation tile) per CTA
  const uint32_t* list;           // [tiles][nkb] blocks of each pattern tile (pair)
  const int* list_n;              // [tiles]
  const unsigned char* rot_inv;   // [n_rt][nkb] the rotation tile has an s <= 0 there
  const unsigned char* rot_tiny;  // [n_rt][nkb] ... an s in (0, 1e-10)
  const float* rot_cnt;
  const float* rot_A;
  const float* rotw;
  const float* cnorm;   // c_i (phi is stored as c_i num/den)
  const float* ktot;    // [N] sum k
  const float* k2tot;   // [N] sum k^2
  float k_inv;          // 1 / count_scale of the K and J operands
  int ms_lo;            // pass C multiplies M'S lo
  int zrow;             // a row past the rotation operands: TMA reads it as zeros
  const float* sigma;   // [1] annealing width (device memory)
  int known_intensity;
  float* L;
  float* PHI;
  float2* part;
  int* bad;
  int* status;
  uint32_t spin;  // polls per pipeline wait (ptx::kSpinLimit unless a debug option lowers it)
};

// The stages of a tile, from the bits of all its entries: where each operand
// lies, in chunks from the slot's first (the pattern side takes two, a rotation
// operand RC: 64 rows of a pair's 128, or all).
template <bool PAIR>
struct EsStages {
  static constexpr int RC = PAIR ? 1 : 2;
  // pass A: J, H, I (or V); then what few tiles have: J lo, H lo, K, T
  static constexpr int aJ = 0, aH = 2, aI = 2 + RC;
  int aJl, aHl, aK, aT;
  // pass B: K, [M'S (or H lo) | H], I (or V); in tiles without pass A: J, J lo, H lo;
  // beside V: T
  static constexpr int bK = 0, bMS = 2, bH = 2 + RC, bI = 2 + 2 * RC;
  int bJ, bJl, bHl, bT;
  // pass C: K, [0 | H lo] (256 columns: a pair's K.H lies in two column quarters
  // that one 128-column product cannot reach, and den starts from the 0, or with lo
  // terms in every product from K x M'S lo)
  static constexpr int cK = 0, cZ = 2, cHl = 2 + RC;
  int size, slots;
  // jh: J x H lo as well; full_h: H lo in M'S's place; vis: sums over V
  __device__ __forceinline__ EsStages(uint32_t seen, bool nj, bool jh, bool full_h, bool vis) {
    const int jl = (seen & es::kJlo) ? 2 : 0;
    int o = aI + RC;
    aJl = o;
    o += jl;
    aHl = o;
    o += jh ? RC : 0;
    aK = o;
    o += vis || (seen & es::kTiny) ? 2 : 0;
    aT = o;
    o += !vis && (seen & es::kTiny) ? RC : 0;
    const bool j = !nj && (seen & es::kJ);
    int q = bI + (vis || (seen & es::kInv) ? RC : 0);
    bJ = q;
    q += j ? 2 : 0;
    bJl = q;
    q += j ? jl : 0;
    bHl = q;
    q += j && jh && !full_h ? RC : 0;
    bT = q;
    q += vis && (seen & es::kTiny) ? RC : 0;
    size = max(q, nj ? o : 0);
    slots = min(es::NB, es::CHUNKS / size);
  }
};

// Entry b of a tile's work: its pattern tile's list entry with the rotation
// tile's flags of that block.
__device__ __forceinline__ uint32_t es_entry(const uint32_t* list, const unsigned char* inv,
                                             const unsigned char* tiny, int b) {
  const uint32_t e = __ldg(list + b);
  const uint32_t kb = e >> 8;
  return e | (inv[kb] ? es::kInv : 0u) | (tiny[kb] ? es::kTiny : 0u);
}

// a / b for normal a and b whose quotient is normal too: the hardware
// reciprocal, the quotient by it, and one residual correction (Markstein 1990),
// which leaves at most the last bit.  Half the instructions of the general
// division, whose range checks num and den do not need.
__device__ __forceinline__ float quotient(float a, float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  const float q = a * r;
  return __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
}

// Epilogue of the likelihood kernel (warps EPI_WARP0 ..): EPI_PARTS warps per
// TMEM lane quarter, each on a part of the 128 columns.  Reads the accumulators
// of this CTA's 128 patterns x 128 rotations from TMEM, writes L and phi and
// the tile's (max, sum exp) per pattern.
template <bool PAIR>
__device__ __forceinline__ void estep_epilogue(const TcEstepArgs& a, uint32_t tmem, uint64_t* accum,
                                               uint64_t* jdone, uint32_t jfree, const float4* s_rot,
                                               float2* s_half, int warp,
                                               int lane, int n0, int r0, int rt, uint32_t seen,
                                               bool vis) {
  using namespace es;
  const int quarter = warp & 3;  // TMEM lanes this warp may access
  const int half = (warp - EPI_WARP0) >> 2;  // column part
  const int row = quarter * 32 + lane;
  const int n = n0 + row;
  const bool nok = n < a.N;
  const float ci = nok ? a.cnorm[n] : 1.0f;
  // what n_1 and n_J are taken from, and with which sign (vis: they are the sums)
  const float ktot = nok && !vis ? a.ktot[n] : 0.0f, k2tot = nok && !vis ? a.k2tot[n] : 0.0f;
  const float k_1 = vis ? a.k_inv : -a.k_inv, k2_1 = vis ? 0.0f : -a.k_inv;
  const bool full_h = a.known_intensity && (a.gh_lo & 2);
  // which of the sums received a product (their columns hold old data otherwise)
  const bool nj = seen & kNJ, have_j = seen & kJ, have_1 = vis || (seen & kInv);
  const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
  const int cbeg = half * (BN / EPI_PARTS), cend = cbeg + BN / EPI_PARTS;
  if (nj) {
    // pass A's n_J to L; the columns, which n_1 takes, go back before the stores,
    // whose completion the arrival would otherwise wait for
    constexpr int CN = BN / EPI_PARTS;
    float vn[CN];
    const bool got = ptx::mbar_wait_sleep(jdone, 0, a.status, 13, 64, a.spin);
    if (got) {
      ptx::tc_fence_after();
      ptx::tmem_ld16(lane_addr + 256 + cbeg, reinterpret_cast<float(&)[16]>(vn[0]));
      ptx::tmem_ld16(lane_addr + 256 + cbeg + 16, reinterpret_cast<float(&)[16]>(vn[16]));
      ptx::tmem_wait_ld();
      ptx::tc_fence_before();
    }
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive_cluster(jfree);
    if (got) {
      const int jn = nok ? min(CN, a.R - (r0 + cbeg)) : 0;
      float* Lp = a.L + (size_t)(r0 + cbeg) * a.N + n;
#pragma unroll
      for (int j = 0; j < CN; ++j) {
        if (j < jn) *Lp = vn[j];
        Lp += a.N;
      }
    }
  }
  float m = -INFINITY, ssum = 0.0f;
  int nbad = 0;
  if (ptx::mbar_wait_sleep(accum, 0, a.status, 2, 256, a.spin)) {
    ptx::tc_fence_after();
    constexpr int CG = 8;
    for (int c0 = cbeg; c0 < cend; c0 += CG) {
      float vd[CG], vh[CG], vj[CG], vn[CG];
      const int cd = PAIR ? c0 + (c0 & 64) : c0;  // column of den; K.H follows
      ptx::tmem_ld8(lane_addr + cd, vd);
      ptx::tmem_ld8(lane_addr + cd + (PAIR ? 64 : 128), vh);
      if (have_1) ptx::tmem_ld8(lane_addr + 256 + c0, vn);
      if (have_j) ptx::tmem_ld8(lane_addr + 384 + c0, vj);
      ptx::tmem_wait_ld();
      float mx = m;
      // eight independent chains, then their exponentials: the running
      // (max, sum exp) is updated once per eight columns
      const int jn = nok ? min(CG, a.R - (r0 + c0)) : 0;  // columns that are pairs
      const size_t o0 = (size_t)(r0 + c0) * a.N + n;
      float* const Lp = a.L + o0;
      float* const Pp = a.PHI + o0;
      float vq[CG];  // n_J
      if (nj) {      // this thread's own stores, all loads in flight together
#pragma unroll
        for (int j = 0; j < CG; ++j) vq[j] = j < jn ? Lp[(size_t)j * a.N] : 0.0f;
      }
#pragma unroll
      for (int j = 0; j < CG; ++j) {
        const float n1 = have_1 ? vn[j] : 0.0f;
        const float kh = (full_h ? vh[j] + vd[j] : vh[j]) * a.k_inv;
        const float B = __fmaf_rn(-kPoisC, kh, __fmaf_rn(k_1, n1, ktot));
        const float Cc = have_j ? __fmaf_rn(vj[j], a.k_inv, kh) : kh;
        const float4 rc = s_rot[c0 + j];  // A_r, 1 / (2 sigma^2 count_r), log w_r
        bool ok = true;
        float iphi = 1.0f, phi = 1.0f;
        if (!a.known_intensity) {
          const float rest = __fmaf_rn(k2_1, n1, k2tot);
          const float num = nj ? __fmaf_rn(k_1, vq[j], rest) : rest;
          const float den = vd[j] * (256.0f * a.k_inv);
          ok = num > 0.0f && den > 0.0f;
          iphi = quotient(den, num);
          phi = quotient(ci * num, den);
        }
        ok = ok && rc.y > 0.0f;
        const float Sig = __fmaf_rn(__fmaf_rn(Cc, iphi, -2.0f * B), iphi, rc.x);
        float L = ok ? __fmaf_rn(-Sig, rc.y, rc.z) : -INFINITY;
        if (j < jn) {
          nbad += ok ? 0 : 1;
          Lp[(size_t)j * a.N] = L;
          Pp[(size_t)j * a.N] = ok ? phi : 1.0f;
        } else {
          L = -INFINITY;
        }
        vh[j] = fmaxf(L, -INFINITY);  // a NaN (a rotation weight that is none) is left out
        mx = fmaxf(mx, L);
      }
      if (mx > -INFINITY) {
        float s = 0.0f;
#pragma unroll
        for (int j = 0; j < CG; ++j) s += expf(vh[j] - mx);
        ssum = ssum * expf(m - mx) + s;
        m = mx;
      }
    }
  }
  // combine the parts' (max, sum exp) of each row
  if (half > 0) s_half[(half - 1) * BM + row] = make_float2(m, ssum);
  asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");  // epilogue warps only
  if (half == 0) {
    float M = m;
    for (int q = 1; q < EPI_PARTS; ++q) M = fmaxf(M, s_half[(q - 1) * BM + row].x);
    float S = 0.0f;
    if (M > -INFINITY) {
      S = ssum * expf(m - M);
      for (int q = 1; q < EPI_PARTS; ++q) {
        const float2 o = s_half[(q - 1) * BM + row];
        S += o.y * expf(o.x - M);
      }
    }
    if (nok) a.part[(size_t)rt * a.N + n] = make_float2(M, S);
  }
  if (nbad) atomicAdd(a.bad, nbad);
}

// BRIGHT: the plan's I operand is V (bright counts).  A variant of its own: the branches
// slow the threads that issue loads and products, 3.7 % of an iteration at 96^3.  A tile
// that sums over V takes more products: 4,000 patterns x 6,300 rotations at 96^3 with
// 2,000 counts at pixels outside the volume, 1,308 us, without such counts 519.
template <bool PAIR, bool BRIGHT>
__global__ void __launch_bounds__(es::THREADS, 1)
    tc_estep_kernel(const __grid_constant__ CUtensorMap mK, const __grid_constant__ CUtensorMap mJ,
                    const __grid_constant__ CUtensorMap mJl, const __grid_constant__ CUtensorMap mMS,
                    const __grid_constant__ CUtensorMap mHh, const __grid_constant__ CUtensorMap mHl,
                    const __grid_constant__ CUtensorMap mIv, const __grid_constant__ CUtensorMap mTv,
                    const __grid_constant__ CUtensorMap mMSl, TcEstepArgs a) {
  using namespace es;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + CHUNKS * CHUNK);
  uint64_t* empty = full + NB;
  uint64_t* accum = empty + NB;
  uint64_t* drain = accum + 1;  // the MMA issuer's own completion wait before TMEM is freed
  uint64_t* jdone = drain + 1;  // pass A's products are complete
  uint64_t* jfree = jdone + 1;  // (rank 0) n_J has been moved out of TMEM
  uint32_t* tmem_slot = (uint32_t*)(jfree + 1);
  float4* s_rot = (float4*)(smem + CHUNKS * CHUNK + 256);
  float2* s_half = (float2*)(s_rot + BN);  // [EPI_PARTS-1][BM] (max, sum exp) of column parts 1..
  uint32_t* s_list = (uint32_t*)(s_half + (EPI_PARTS - 1) * BM);  // [kList]
  uint32_t* s_seen = s_list + kList;  // the bits of all entries; entries passes A and C look at

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? ptx::cluster_ctarank() : 0u;
  const float sg = *a.sigma;
  const float inv2s2 = 1.0f / (2.0f * sg * sg);
  int pt, rt;  // pattern tile (pair of tiles), rotation tile
  if (!PAIR && a.tiles) {  // pruned: the listed tiles only
    const int2 t = a.tiles[blockIdx.x];
    pt = t.x;
    rt = t.y;
  } else {
    raster_tile((int)(PAIR ? blockIdx.x >> 1 : blockIdx.x) + a.tile0, a.raster,
                PAIR ? (a.n_pt + 1) / 2 : a.n_pt, a.n_rt, pt, rt);
  }
  // a pair's second tile may be n_pt (no patterns) when n_pt is odd
  const int n0 = (PAIR ? 2 * pt + (int)rank : pt) * BM, r0 = rt * BN;
  const uint32_t* list = a.list + (size_t)pt * a.nkb;
  const int cnt = a.list_n[pt];
  const unsigned char* inv = a.rot_inv + (size_t)rt * a.nkb;
  const unsigned char* tiny = a.rot_tiny + (size_t)rt * a.nkb;
  const bool full_h = a.known_intensity && (a.gh_lo & 2);  // phi = 1: no den, H lo throughout

  if (threadIdx.x == 0) {
    for (int s = 0; s < NB; ++s) {
      ptx::mbar_init(&full[s], 1);
      ptx::mbar_init(&empty[s], 1);
    }
    ptx::mbar_init(accum, 1);
    ptx::mbar_init(drain, 1);
    ptx::mbar_init(jdone, 1);
    ptx::mbar_init(jfree, EPI_WARPS * (PAIR ? 2 : 1));
    ptx::fence_mbar_init();
    s_seen[0] = s_seen[1] = s_seen[2] = 0;
  }
  uint32_t seen = 0, last_a = 0, last_c = 0;
  for (int b = threadIdx.x; b < cnt; b += THREADS) {
    const uint32_t e = es_entry(list, inv, tiny, b);
    if (b < kList) s_list[b] = e;
    seen |= e & 0xff;
    // n_J is needed: invalid pixels where counts exceed 1, or an s in (0, 1e-10)
    const bool takes = (e & kInv) && (BRIGHT || (e & kJ));
    if ((takes || (e & kTiny)) && !a.known_intensity) seen |= kNJ;
    if (e & (kJ | kTiny)) last_a = b + 1;
    if (e & kHlo) last_c = b + 1;
  }
  if (threadIdx.x < BN) {
    const int r = r0 + threadIdx.x;
    const float c = r < a.R ? a.rot_cnt[r] : 0.0f;
    // scale < 0: invalid rotation
    s_rot[threadIdx.x] = make_float4(r < a.R ? a.rot_A[r] : 0.0f, c > 0.0f ? inv2s2 / c : -1.0f,
                                     r < a.R ? logf(a.rotw[r]) : 0.0f, 0.0f);
  }
  if (warp == MMA_WARP) {
    if (PAIR) {
      ptx::tmem_alloc_pair(tmem_slot, 512);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(tmem_slot, 512);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  seen = __reduce_or_sync(0xffffffffu, seen);
  last_a = __reduce_max_sync(0xffffffffu, last_a);
  if (lane == 0 && seen) atomicOr(s_seen, seen);
  last_c = __reduce_max_sync(0xffffffffu, last_c);
  if (lane == 0 && last_a) atomicMax(s_seen + 1, last_a);
  if (lane == 0 && last_c) atomicMax(s_seen + 2, last_c);
  __syncthreads();
  if (PAIR) ptx::cluster_sync();  // both CTAs' barriers initialised and TMEM allocated
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  auto entry = [&](uint32_t b) { return b < kList ? s_list[b] : es_entry(list, inv, tiny, (int)b); };
  const bool known = a.known_intensity != 0;
  const bool jh = (a.gh_lo & 2) != 0;  // H lo in every product
  const uint32_t all = *s_seen;
  const bool nj = all & kNJ;  // the tile has a pass A
  const bool vis = BRIGHT && (all & (kInv | kTiny));  // sums over the covered pixels
  const EsStages<PAIR> st(known && !vis ? all & ~kTiny : all, nj, jh, full_h, vis);
  // entries of each pass: A those with J (or T; all with V), B all, C those before the
  // count tail
  const uint32_t n_b = (uint32_t)cnt, n_a = !nj ? 0u : vis ? n_b : s_seen[1];
  const uint32_t n_c = full_h || !a.gh_lo ? 0u : (jh ? n_b : s_seen[2]);
  const uint32_t in_c = jh ? ~0u : kHlo;

  if (warp < PRODUCERS) {
    // ------------------------------------------------ TMA producers (both CTAs of a pair)
    if (ptx::elect_one()) {
      constexpr int RC = EsStages<PAIR>::RC;
      const int rr = r0 + 64 * (int)rank;  // this CTA's rows of the rotation operands
      const uint32_t full0 = ptx::smem_u32(full);
      const uint32_t fb0 = PAIR ? ptx::mapa_shared(full0, 0) : full0;
      uint32_t it = 0, slot = 0, phase = 1;  // stages issued; the next one's slot and parity
      bool run = true;
      auto ld = [&](int o, const CUtensorMap* m, uint32_t e, int y) {
        unsigned char* to = smem + ((int)slot * st.size + o) * CHUNK;
        const int x = (int)(e >> 8) * BK;
        if (PAIR)
          ptx::tma_load_2d_pair(to, m, x, y, fb0 + 8 * slot);
        else
          ptx::tma_load_2d(to, m, x, y, fb0 + 8 * slot);
      };
      auto ldr = [&](int o, const CUtensorMap* m, uint32_t e) {  // 64 rotation rows, or 128 in two boxes
        ld(o, m, e, rr);
        if (!PAIR) ld(o + 1, m, e, rr + 64);
      };
      auto ldz = [&](int o, const CUtensorMap* m, uint32_t e) {  // as many rows of zeros
        ld(o, m, e, a.zrow);
        if (!PAIR) ld(o + 1, m, e, a.zrow);
      };
      // a free slot, armed by the first producer for a stage of `chunks`
      // (rank 0's barriers count both CTAs' bytes)
      auto open = [&](int chunks) {
        if (!ptx::mbar_wait(&empty[slot], phase, a.status, 0, a.spin)) return run = false;
        if (warp == 0 && rank == 0)
          ptx::mbar_arrive_expect_tx(&full[slot], (uint32_t)chunks * (CHUNK * (PAIR ? 2 : 1)));
        return true;
      };
      auto next = [&]() {
        ++it;
        if (++slot == (uint32_t)st.slots) {
          slot = 0;
          phase ^= 1;
        }
      };
      for (uint32_t u = n_a; u-- > 0;) {  // pass A
        const uint32_t e = entry(u);
        if (!vis && !(e & (kJ | kTiny))) continue;
        const bool j = e & kJ, jl = j && (e & kJlo), hl = j && jh, t = !vis && (e & kTiny);
        if (!open((j ? 2 + RC : 0) + (j || vis ? RC : 0) + (jl ? 2 : 0) + (hl ? RC : 0) +
                  (t || vis ? 2 : 0) + (t ? RC : 0)))
          break;
        if (warp == 0) {
          if (j) ld(st.aJ, &mJ, e, n0);
          if (jl) ld(st.aJl, &mJl, e, n0);
          if (t || vis) ld(st.aK, &mK, e, n0);
        } else if (warp == 1) {
          if (j) ldr(st.aH, &mHh, e);
          if (hl) ldr(st.aHl, &mHl, e);
        } else {
          if (j || vis) ldr(st.aI, &mIv, e);
          if (t) ldr(st.aT, &mTv, e);
        }
        next();
      }
      for (uint32_t u = n_c; run && u-- > 0;) {  // pass C
        const uint32_t e = entry(u);
        if (!(e & in_c)) continue;
        if (!open(2 + 2 * RC)) break;
        if (warp == 0) {
          ld(st.cK, &mK, e, n0);
        } else if (warp == 1) {
          if (a.ms_lo)
            ldr(st.cZ, &mMSl, e);
          else
            ldz(st.cZ, &mHl, e);
        } else {
          ldr(st.cHl, &mHl, e);
        }
        next();
      }
      for (uint32_t u = n_b; run && u-- > 0;) {  // pass B
        const uint32_t e = entry(u);
        const bool j = !nj && (e & kJ), jl = j && (e & kJlo);
        const bool hl = j && jh && !full_h, i = vis || (e & kInv), t = vis && (e & kTiny);
        if (!open(2 + 2 * RC + (i ? RC : 0) + (j ? 2 : 0) + (jl ? 2 : 0) + (hl ? RC : 0) +
                  (t ? RC : 0)))
          break;
        if (warp == 0) {
          ld(st.bK, &mK, e, n0);
          if (jl) ld(st.bJl, &mJl, e, n0);
          if (hl) ldr(st.bHl, &mHl, e);
        } else if (warp == 1) {
          ldr(st.bMS, full_h ? &mHl : &mMS, e);
          if (j) ld(st.bJ, &mJ, e, n0);
        } else {
          ldr(st.bH, &mHh, e);
          if (i) ldr(st.bI, &mIv, e);
          if (t) ldr(st.bT, &mTv, e);
        }
        next();
      }
      // no copy may still be landing in shared memory when the CTA exits: after
      // a normal run the MMAs have consumed them all (no wait)
      if (warp == 0 && rank == 0) ptx::drain_loads(full, st.slots, it, a.status, 11);
    }
  } else if (warp == MMA_WARP) {
    // ------------------------------------------------ MMA issuer (rank 0 of a pair)
    if (rank == 0 && ptx::elect_one()) {
      constexpr int M = PAIR ? 2 * BM : BM;
      constexpr uint32_t idesc2 = ptx::idesc_f16(M, 2 * BN);
      constexpr uint32_t idesc1 = ptx::idesc_f16(M, BN);
      auto mma = [&](uint32_t d, uint64_t x, uint64_t y, uint32_t id, uint32_t acc) {
        if (PAIR)
          ptx::mma_f16_pair(d, x, y, id, acc);
        else
          ptx::mma_f16(d, x, y, id, acc);
      };
      const uint32_t t256 = tmem + 256, t384 = tmem + 384;
      const uint64_t desc0 = ptx::smem_desc(ptx::smem_u32(smem), 1024, 2);
      uint32_t slot = 0, phase = 0;
      uint64_t base = 0;
      bool run = true;
      // descriptors count 16-byte units (no carry past the 14-bit address field)
      auto d = [&](int o, int ks) { return base + (uint64_t)(o * (CHUNK / 16) + ks * 2); };
      auto mma4 = [&](uint32_t t, int x, int y, uint32_t id, uint32_t acc) {
#pragma unroll
        for (int ks = 0; ks < BK / 16; ++ks) mma(t, d(x, ks), d(y, ks), id, ks ? 1u : acc);
      };
      auto open = [&]() {
        if (!ptx::mbar_wait(&full[slot], phase, a.status, 1, a.spin)) return run = false;
        ptx::tc_fence_after();
        base = desc0 + (uint64_t)(slot * (uint32_t)st.size * (CHUNK / 16));
        return true;
      };
      auto close = [&]() {
        if (PAIR)
          ptx::mma_commit_pair(&empty[slot], 0x3);
        else
          ptx::mma_commit(&empty[slot]);
        if (++slot == (uint32_t)st.slots) {
          slot = 0;
          phase ^= 1;
        }
      };
      uint32_t accJ = 0, accN = 0;  // J.H, n_J hold a product
      for (uint32_t u = n_a; u-- > 0;) {
        const uint32_t e = entry(u);
        if (!vis && !(e & (kJ | kTiny))) continue;
        if (!open()) break;
        const bool j = e & kJ, jl = j && (e & kJlo);
        if (j) {
          mma4(t384, st.aJ, st.aH, idesc1, accJ);  // J.H
          if (jl) mma4(t384, st.aJl, st.aH, idesc1, 1u);
          if (jh) mma4(t384, st.aJ, st.aHl, idesc1, 1u);
          mma4(t256, st.aJ, st.aI, idesc1, accN);  // n_J
          if (jl) mma4(t256, st.aJl, st.aI, idesc1, 1u);
          accJ = accN = 1;
        }
        if (vis) {
          mma4(t256, st.aK, st.aI, idesc1, accN);
          accN = 1;
        } else if (e & kTiny) {
          mma4(t256, st.aK, st.aT, idesc1, accN);
          if (j) mma4(t256, st.aJ, st.aT, idesc1, 1u);
          if (jl) mma4(t256, st.aJl, st.aT, idesc1, 1u);
          accN = 1;
        }
        close();
      }
      if (nj) {
        if (PAIR)
          ptx::mma_commit_pair(jdone, 0x3);
        else
          ptx::mma_commit(jdone);
      }
      uint32_t accB = 0;  // den | K.H holds a product
      for (uint32_t u = n_c; run && u-- > 0;) {  // pass C
        const uint32_t e = entry(u);
        if (!(e & in_c)) continue;
        if (!open()) break;
        mma4(tmem, st.cK, st.cZ, idesc2, accB);
        accB = 1;
        close();
      }
      uint32_t acc1 = 0;  // n_1 holds a product
      bool taken = nj;    // pass A's n_J is still there
      for (uint32_t u = n_b; run && u-- > 0;) {
        const uint32_t e = entry(u);
        const bool j = !nj && (e & kJ);
        if (!open()) break;
        mma4(tmem, st.bK, st.bMS, idesc2, accB);  // den | K.H
        accB = 1;
        const bool i = vis || (e & kInv);
        if (taken && i) {
          if (!ptx::mbar_wait_cluster(jfree, 0, a.status, 13, a.spin)) break;
          ptx::tc_fence_after();
          taken = false;
        }
        if (j) {
          mma4(t384, st.bJ, st.bH, idesc1, accJ);
          accJ = 1;
          if (e & kJlo) mma4(t384, st.bJl, st.bH, idesc1, 1u);
          if (jh) mma4(t384, st.bJ, full_h ? st.bMS : st.bHl, idesc1, 1u);
        }
        if (i) {
          mma4(t256, st.bK, st.bI, idesc1, acc1);
          acc1 = 1;
          if (vis && (e & kTiny)) mma4(t256, st.bK, st.bT, idesc1, 1u);
        }
        close();
      }
      // accum fires when every MMA issued above has completed (after a timeout
      // the epilogue's own bounded wait reports it); drain: TMEM is freed only
      // after every MMA issued here has completed, also when the epilogue
      // stopped waiting (both CTAs' TMEM is written by a pair's MMAs)
      if (PAIR) {
        ptx::mma_commit_pair(accum, 0x3);
        ptx::mma_commit_pair(drain, 0x1);
      } else {
        ptx::mma_commit(accum);
        ptx::mma_commit(drain);
      }
      ptx::mbar_wait(drain, 0, a.status, 12);
    }
  } else {
    // ------------------------------------------------ epilogue
    estep_epilogue<PAIR>(a, tmem, accum, jdone, ptx::mapa_shared(ptx::smem_u32(jfree), 0), s_rot,
                         s_half, warp, lane, n0, r0, rt, *s_seen, vis);
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (PAIR) ptx::cluster_sync();  // the pair's MMAs and barrier traffic are over in both CTAs
  if (threadIdx.x == 32 * MMA_WARP) ptx::settle_after_timeout(a.status);
  __syncthreads();
  if (warp == MMA_WARP) {
    ptx::tc_fence_after();
    if (PAIR)
      ptx::tmem_dealloc_pair(tmem, 512);
    else
      ptx::tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------ E-step, true Poisson -----
// L_ri = log w_r + c_i sum_p k_ip log s~_rp + K_i log(K_i / S_r) - K_i,
// s~ = max(s, floor), K_i = c_i sum_p k_ip, S_r = sum_p s~_rp, phi = K_i / S_r
// (known intensity: phi = 1, L = log w_r + c_i sum k log s~ - S_r), as the
// FP32 path.  One contraction K . (log S~)^T with log S~ as FP16 hi + lo, over the
// pattern tile's 64-pixel blocks with counts (the others' products are zero).
// Persistent: a CTA (pair) takes tiles first, first + grid, ..; the stage ring runs
// on across tiles and the accumulator is double-buffered in TMEM, so that a tile's
// epilogue -- 256 columns of logarithms, exponentials and stores -- overlaps the
// next one's MMAs.  Bound by the tensor pipe in pairs (48 KB per CTA and 64 pixels,
// 47 B/clk), by L2 reads in single CTAs (80 KB for the same time).  Each 128-rotation
// half of a tile leaves one (max, sum exp) partial.  All blocks, single CTAs of 32
// pixels a stage and no overlap before: 112^3, 10,860 rotations, 10,000 patterns
// 3,210 us, now 943; 128^3 pruned 2,428, now 1,124.
namespace ep {
constexpr int BM = 128;  // patterns per CTA (TMEM lanes)
constexpr int BN = 256;  // rotations per tile
constexpr int BK = 64;   // pixels per block
constexpr int EPI_WARPS = 16;  // four per TMEM lane quarter, 64 columns each
constexpr int THREADS = 64 + 32 * EPI_WARPS;
// A pair (256 patterns x 256 rotations, each CTA half of the log-slices) takes a
// block per stage; a single CTA half a block, so that more of them are in flight.
template <bool PAIR>
struct Ring {
  static constexpr int kPix = PAIR ? 64 : 32;  // 128 B rows, 128B swizzle; 64 B, 64B
  static constexpr int kA = BM * kPix * 2, kB = (PAIR ? BN / 2 : BN) * kPix * 2;
  static constexpr int kStage = kA + 2 * kB;
  static constexpr int kStages = PAIR ? 4 : 5;
  // barriers, two rows of BN floats, the (max, sum exp) of the odd column parts
  static constexpr int kSmem = kStages * kStage + 256 + 2 * BN * 4 + 2 * BM * 8 + 1024;
  static_assert(kSmem <= 232448, "shared memory of the true-Poisson likelihood");
};
}  // namespace ep

struct TcEstepPoisArgs {
  int N, R, n_pt, n_rt, nkb;  // n_pt: pattern tiles (pairs of tiles)
  int raster;             // tile order (raster_tile)
  int tile0, n_tiles;     // the tiles tile0 .. + n_tiles of the order
  const int2* tiles;      // pruned iteration: n_tiles of (pattern tile, 256-rotation tile)
  const uint32_t* list;   // [n_pt][nkb] blocks with counts << 8, ascending
  const int* list_n;      // at least one
  int n_part;             // 128-rotation partial tiles
  const float* rot_ssum;  // S_r
  const float* rotw;
  const float* Ksum;      // K_i (normalised counts)
  const float* cnorm;     // c_i
  int known_intensity;
  float* L;
  float* PHI;
  float2* part;
  int* status;
  uint32_t spin;  // polls per pipeline wait
};

template <bool PAIR>
__global__ void __launch_bounds__(ep::THREADS, 1)
    tc_estep_pois_kernel(const __grid_constant__ CUtensorMap mK,
                         const __grid_constant__ CUtensorMap mLh,
                         const __grid_constant__ CUtensorMap mLl, TcEstepPoisArgs a) {
  using namespace ep;
  using Rg = Ring<PAIR>;
  constexpr int STAGES = Rg::kStages, STAGE_BYTES = Rg::kStage;
  constexpr int SUB = BK / Rg::kPix;  // stages per block
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;  // [2] accumulator ready
  uint64_t* tempty = tfull + 2;      // [2] (rank 0) accumulator drained
  uint64_t* drain = tempty + 2;  // the MMA issuer's own completion wait before TMEM is freed
  uint32_t* tmem_slot = (uint32_t*)(drain + 1);
  float* s_ss = (float*)(smem + STAGES * STAGE_BYTES + 256);
  float* s_lw = s_ss + BN;
  float2* s_half = (float2*)(s_lw + BN);  // [2][BM]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? ptx::cluster_ctarank() : 0u;
  const int first = (int)(PAIR ? blockIdx.x >> 1 : blockIdx.x);
  const int step = (int)(PAIR ? gridDim.x >> 1 : gridDim.x);
  auto tile = [&](int t, int& pt, int& rt) {
    if (!PAIR && a.tiles) {  // pruned: the listed tiles only
      const int2 v = __ldg(a.tiles + t);
      pt = v.x;
      rt = v.y;
    } else {
      raster_tile(t + a.tile0, a.raster, a.n_pt, a.n_rt, pt, rt);
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&full[s], 1);
      ptx::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&tfull[b], 1);
      ptx::mbar_init(&tempty[b], (PAIR ? 2 : 1) * EPI_WARPS);
    }
    ptx::mbar_init(drain, 1);
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    if (PAIR) {
      ptx::tmem_alloc_pair(tmem_slot, 512);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(tmem_slot, 512);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (PAIR) ptx::cluster_sync();  // both CTAs' barriers initialised and TMEM allocated
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------ TMA producer (both CTAs of a pair)
    if (ptx::elect_one()) {
      const uint32_t full0 = ptx::smem_u32(full);
      const uint32_t fb0 = PAIR ? ptx::mapa_shared(full0, 0) : full0;
      uint32_t it = 0;
      bool ok = true;
      for (int t = first; t < a.n_tiles && ok; t += step) {
        int pt, rt;
        tile(t, pt, rt);
        // a pair's second pattern tile may be past the last (zeros)
        const int n0 = (PAIR ? 2 * pt + (int)rank : pt) * BM;
        const int r0 = rt * BN + (PAIR ? BN / 2 * (int)rank : 0);
        const uint32_t* list = a.list + (size_t)pt * a.nkb;
        const int cnt = a.list_n[pt];
        uint32_t next = __ldg(list);
        for (int u = 0; u < cnt * SUB; ++u, ++it) {
          const int x = (int)(next >> 8) * BK + (u % SUB) * Rg::kPix;
          if (u % SUB == SUB - 1 && u + 1 < cnt * SUB) next = __ldg(list + u / SUB + 1);
          const uint32_t s = it % STAGES;
          if (!ptx::mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1, a.status, 8, a.spin)) {
            ok = false;
            break;
          }
          // rank 0's barriers count both CTAs' bytes
          if (rank == 0) ptx::mbar_arrive_expect_tx(&full[s], STAGE_BYTES * (PAIR ? 2 : 1));
          unsigned char* st = smem + s * STAGE_BYTES;
          if (PAIR) {
            ptx::tma_load_2d_pair(st, &mK, x, n0, fb0 + 8 * s);
            ptx::tma_load_2d_pair(st + Rg::kA, &mLh, x, r0, fb0 + 8 * s);
            ptx::tma_load_2d_pair(st + Rg::kA + Rg::kB, &mLl, x, r0, fb0 + 8 * s);
          } else {
            ptx::tma_load_2d(st, &mK, x, n0, fb0 + 8 * s);
            ptx::tma_load_2d(st + Rg::kA, &mLh, x, r0, fb0 + 8 * s);
            ptx::tma_load_2d(st + Rg::kA + Rg::kB, &mLl, x, r0, fb0 + 8 * s);
          }
        }
      }
      if (rank == 0) ptx::drain_loads(full, STAGES, it, a.status, 11);  // none in flight at exit
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer (rank 0 of a pair)
    if (rank == 0 && ptx::elect_one()) {
      constexpr uint32_t idesc = ptx::idesc_f16(PAIR ? 2 * BM : BM, BN);
      uint32_t it = 0;
      bool ok = true;
      int j = 0;
      for (int t = first; t < a.n_tiles && ok; t += step, ++j) {
        const int b = j & 1;
        const uint32_t d = tmem + (uint32_t)(b * BN);
        int pt, rt;
        tile(t, pt, rt);
        const int n = a.list_n[pt] * SUB;
        if (!ptx::mbar_wait_cluster(&tempty[b], ((j >> 1) & 1) ^ 1, a.status, 7, a.spin)) break;
        ptx::tc_fence_after();
        for (int u = 0; u < n; ++u, ++it) {
          const uint32_t s = it % STAGES;
          if (!ptx::mbar_wait(&full[s], (it / STAGES) & 1, a.status, 9, a.spin)) {
            ok = false;
            break;
          }
          ptx::tc_fence_after();
          const uint32_t base = ptx::smem_u32(smem + s * STAGE_BYTES);
#pragma unroll
          for (int ks = 0; ks < Rg::kPix / 16; ++ks) {
            constexpr int sbo = PAIR ? 1024 : 512, sw = PAIR ? 2 : 4;
            const uint64_t aK = ptx::smem_desc(base + ks * 32, sbo, sw);
            const uint64_t bh = ptx::smem_desc(base + Rg::kA + ks * 32, sbo, sw);
            const uint64_t bl = ptx::smem_desc(base + Rg::kA + Rg::kB + ks * 32, sbo, sw);
            if (PAIR) {
              ptx::mma_f16_pair(d, aK, bh, idesc, (u | ks) ? 1u : 0u);
              ptx::mma_f16_pair(d, aK, bl, idesc, 1u);
            } else {
              ptx::mma_f16(d, aK, bh, idesc, (u | ks) ? 1u : 0u);
              ptx::mma_f16(d, aK, bl, idesc, 1u);
            }
          }
          if (PAIR)
            ptx::mma_commit_pair(&empty[s], 0x3);
          else
            ptx::mma_commit(&empty[s]);
        }
        if (PAIR)
          ptx::mma_commit_pair(&tfull[b], 0x3);
        else
          ptx::mma_commit(&tfull[b]);
      }
      if (PAIR)
        ptx::mma_commit_pair(drain, 0x1);  // both CTAs' TMEM is written by these MMAs
      else
        ptx::mma_commit(drain);
      ptx::mbar_wait(drain, 0, a.status, 12);
    }
  } else {
    // ------------------------------------------------ epilogue
    const int quarter = warp & 3;      // TMEM lanes this warp may access
    const int part = (warp - 2) >> 2;  // which of the tile's columns
    const int row = quarter * 32 + lane;
    const int c_beg = part * (BN / 4), c_end = c_beg + BN / 4;
    bool ok = true;
    int j = 0;
    for (int t = first; t < a.n_tiles; t += step, ++j) {
      const int b = j & 1;
      int pt, rt;
      tile(t, pt, rt);
      const int n = (PAIR ? 2 * pt + (int)rank : pt) * BM + row, r0 = rt * BN;
      const bool nok = n < a.N;
      const float ci = nok ? a.cnorm[n] : 1.0f;
      const float Ki = nok ? a.Ksum[n] : 0.0f;
      const int e = (int)threadIdx.x - 64;
      if (e < BN) {  // the last tile's readers have passed its second barrier
        const int r = r0 + e;
        s_ss[e] = r < a.R ? a.rot_ssum[r] : 1.0f;
        s_lw[e] = r < a.R ? logf(a.rotw[r]) : 0.0f;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
      // after a wait that gave up the warp only keeps the other warps' barriers going
      ok = ok && ptx::mbar_wait_sleep(&tfull[b], (j >> 1) & 1, a.status, 10, 128, a.spin);
      float m = -INFINITY, ssum = 0.0f;
      if (ok) {
        ptx::tc_fence_after();
        const uint32_t col = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * BN);
        constexpr int CG = 8;
        for (int c0 = c_beg; c0 < c_end; c0 += CG) {
          float v[CG];
          ptx::tmem_ld8(col + c0, v);
          ptx::tmem_wait_ld();
          const int jn = nok ? min(CG, a.R - (r0 + c0)) : 0;  // columns that are pairs
          float* Lp = a.L + (size_t)(r0 + c0) * a.N + n;
          float* Pp = a.PHI + (size_t)(r0 + c0) * a.N + n;
          float mx = m;
#pragma unroll
          for (int i = 0; i < CG; ++i) {
            const float acc = ci * v[i], lw = s_lw[c0 + i], Sr = s_ss[c0 + i];
            float l, f;
            if (a.known_intensity) {
              f = 1.0f;
              l = lw + acc - Sr;
            } else if (Ki > 0.0f) {
              f = Ki / Sr;
              l = lw + acc + Ki * logf(f) - Ki;
            } else {
              f = 0.0f;
              l = lw;
            }
            if (i < jn) {
              *Lp = l;
              *Pp = f;
            } else {
              l = -INFINITY;
            }
            Lp += a.N;
            Pp += a.N;
            v[i] = fmaxf(l, -INFINITY);  // a NaN (a rotation weight that is none) is left out
            mx = fmaxf(mx, l);
          }
          if (mx > -INFINITY) {
            float s = 0.0f;
#pragma unroll
            for (int i = 0; i < CG; ++i) s += expf(v[i] - mx);
            ssum = ssum * expf(m - mx) + s;
            m = mx;
          }
        }
      }
      // this warp's reads of buffer b are complete: hand it back to the MMA warp
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR && rank != 0)
          ptx::mbar_arrive_cluster(ptx::mapa_shared(ptx::smem_u32(&tempty[b]), 0));
        else
          ptx::mbar_arrive(&tempty[b]);
      }
      // one partial per 128-rotation half: parts 0 and 1, 2 and 3
      if (part & 1) s_half[(part >> 1) * BM + row] = make_float2(m, ssum);
      asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
      const int tp = 2 * rt + (part >> 1);
      if (!(part & 1) && nok && tp < a.n_part) {
        const float2 o = s_half[(part >> 1) * BM + row];
        const float M = fmaxf(m, o.x);
        float S = 0.0f;
        if (M > -INFINITY) S = ssum * expf(m - M) + o.y * expf(o.x - M);
        a.part[(size_t)tp * a.N + n] = make_float2(M, S);
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (PAIR) ptx::cluster_sync();  // the pair's MMAs and barrier traffic are over in both CTAs
  if (threadIdx.x == 32) ptx::settle_after_timeout(a.status);
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    if (PAIR)
      ptx::tmem_dealloc_pair(tmem, 512);
    else
      ptx::tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------ M-step -----
namespace ms {
constexpr int BM = 128;   // rotations per tile (TMEM lanes)
constexpr int BN = 256;   // pixels per tile
constexpr int BK = 64;    // patterns per stage (128 B rows, 128B swizzle)
constexpr int A_BYTES = BM * BK * 2;  // 16 KB
constexpr int B_BYTES = BN * BK * 2;  // 32 KB
constexpr int EPI_WARPS = 16;         // four per TMEM lane quarter, 64 columns each
constexpr int EPI_COLS = BN / (EPI_WARPS / 4);
constexpr int THREADS = 64 + 32 * EPI_WARPS;
constexpr int XYZ_BYTES = 2 * BN * 16;  // pixel coordinates of two tiles
}  // namespace ms

struct TcMstepArgs {
  int R, Kp, Np, P_eff, n_qt, n_rt, nkb, n_tiles;
  int raster;  // tile order (raster_tile over pixel tiles x rotation tiles)
  const float* T;
  const float* qscale;  // [R] 2^-e_r
  float k_inv;          // 1 / count_scale of the K^T operand
  const float* rot;
  const float *cx, *cy, *cz;
  int side, interp, deterministic;
  int aggregate;  // 1: lanes hitting the same voxel combine before one atomic
  float* model;
  float* weight;
  ulonglong2* fix2;
  float2* acc2;
  const float2* fix_scale;  // {model, weight} fixed-point scales (deterministic mode)
  float* u;                 // sorted mode: pair values [P_eff][ldu] instead of insertion
  int ldu;
  int q_lo;  // 1: Q hi + lo, 0: Q hi only
  // pruned iteration: the pattern k-blocks of rotation tile rt are
  // kb_list[kb_off[rt] .. kb_off[rt+1]) (Q is zero elsewhere); nullptr: all
  const int* kb_off;
  const int* kb_list;
  // per pixel tile, the pattern k-blocks in which it has counts (list, count,
  // map; K is zero elsewhere)
  const int* ms_list;
  const int* ms_n;
  const unsigned char* ms_map;
  int* status;
  uint32_t spin;  // polls per pipeline wait
};

__device__ __forceinline__ void tc_add(const TcMstepArgs& a, size_t v, float val, float w) {
  if (a.deterministic) {
    const float2 sc = __ldg(a.fix_scale);
    atomicAdd(&a.fix2[v].x, (unsigned long long)fixed_from_float(__fmul_rn(val, sc.x)));
    atomicAdd(&a.fix2[v].y, (unsigned long long)fixed_from_float(__fmul_rn(w, sc.y)));
  } else {
    atomicAdd(a.acc2 + v, make_float2(val, w));  // model and weight in one 8-byte atomic
  }
}

// Nearest-voxel insertion of one value per lane.  With aggregation (float
// atomics only), lanes of the warp whose voxels coincide -- neighbouring
// rotations at the same small-radius pixel -- add their values in registers
// and their lowest lane issues one atomic.  Called by all 32 lanes.
__device__ __forceinline__ void tc_insert_nearest(const TcMstepArgs& a, bool on, long long v,
                                                  float val, float w) {
  if (a.aggregate && !a.deterministic) {
    const unsigned act = __ballot_sync(0xffffffffu, on);
    if (!on) return;
    const unsigned peers = __match_any_sync(act, v);
    const int me = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    // every lane of a peer group runs the same sequence of shuffles
    for (unsigned m = peers & (peers - 1); m; m &= m - 1) {
      const int src = __ffs(m) - 1;
      const float pv = __shfl_sync(peers, val, src);
      const float pw = __shfl_sync(peers, w, src);
      if (me == leader) {
        val += pv;
        w += pw;
      }
    }
    if (me == leader) atomicAdd(a.acc2 + v, make_float2(val, w));
    return;
  }
  if (on) tc_add(a, (size_t)v, val, w);
}

// Trilinear insertion of one value per lane; called by all 32 lanes.  What bounds
// it is the L2 atomic unit, by the 32-byte sectors that an instruction touches: a
// cell's eight corners at one lane's hands are eight sectors (sixteen with model and
// weight in arrays of their own).  So the two corners of an x edge, neighbours in
// memory, and with fixed-point sums the model and the weight of each, go to
// neighbouring lanes of one instruction: 2 (float) or 4 (fixed) lanes take their
// group's points in turn.  Fixed-point insertion of 10,860 slices of 7,236 pixels
// (1.3e9 atomic additions): 6,790 us, now 3,070.
__device__ __forceinline__ void tc_insert_trilinear(const TcMstepArgs& a, bool on, const RotMat& R,
                                                    float x, float y, float z, float val,
                                                    float w) {
  const int side = a.side, lane = threadIdx.x & 31;
  const float cx = voxel_coord(side, rotate_row(R, 0, x, y, z));
  const float cy = voxel_coord(side, rotate_row(R, 1, x, y, z));
  const float cz = voxel_coord(side, rotate_row(R, 2, x, y, z));
  const float fx0 = floorf(cx), fy0 = floorf(cy), fz0 = floorf(cz);
  const int x0 = (int)fx0, y0 = (int)fy0, z0 = (int)fz0;
  const float tx = cx - fx0, ty = cy - fy0, tz = cz - fz0;
  const unsigned n = (unsigned)side;
  // bits 0, 1: x0 and x0 + 1 inside; 2, 3: y; 4, 5: z
  unsigned in = 0;
  if (on)
    in = ((unsigned)x0 < n) | ((unsigned)x0 + 1 < n) << 1 | ((unsigned)y0 < n) << 2 |
         ((unsigned)y0 + 1 < n) << 3 | ((unsigned)z0 < n) << 4 | ((unsigned)z0 + 1 < n) << 5;
  const int base = on ? (z0 * side + y0) * side + x0 : 0;
  const int group = a.deterministic ? 4 : 2;
  const float2 sc = a.deterministic ? __ldg(a.fix_scale) : make_float2(1.0f, 1.0f);
  for (int s = 0; s < group; ++s) {
    const int src = (lane & ~(group - 1)) + s;
    const unsigned pin = __shfl_sync(0xffffffffu, in, src);
    const int pbase = __shfl_sync(0xffffffffu, base, src);
    const float px = __shfl_sync(0xffffffffu, tx, src), py = __shfl_sync(0xffffffffu, ty, src);
    const float pz = __shfl_sync(0xffffffffu, tz, src);
    const float pv = __shfl_sync(0xffffffffu, val, src), pw = __shfl_sync(0xffffffffu, w, src);
    const int hx = a.deterministic ? (lane >> 1) & 1 : lane & 1;
    if (!((pin >> hx) & 1)) continue;
    const float fx = hx ? px : 1.0f - px;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (!((pin >> (2 + (k & 1))) & (pin >> (4 + (k >> 1))) & 1)) continue;
      const float f = fx * ((k & 1) ? py : 1.0f - py) * ((k >> 1) ? pz : 1.0f - pz);
      if (f <= 0.0f) continue;
      const int v = pbase + hx + ((k & 1) + (k >> 1) * side) * side;
      if (a.deterministic) {
        const bool wt = lane & 1;
        atomicAdd(wt ? &a.fix2[v].y : &a.fix2[v].x,
                  (unsigned long long)fixed_from_float(
                      __fmul_rn(wt ? pw * f : pv * f, wt ? sc.y : sc.x)));
      } else {
        atomicAdd(a.acc2 + v, make_float2(pv * f, pw * f));
      }
    }
  }
}

// The coordinates of a tile's 256 pixels into shared memory, by the first 256 of
// the epilogue's threads; read by all of them after the barrier.  Two buffers: a
// thread that writes the tile after next has passed the next tile's barrier, so
// every thread is done with this one.
__device__ __forceinline__ const float4* ms_stage_pixels(const TcMstepArgs& a, float4* s_xyz,
                                                         int tile, int q0) {
  float4* dst = s_xyz + (tile & 1) * ms::BN;
  const int e = (int)threadIdx.x - 64;
  if (e < ms::BN && q0 + e < a.P_eff)
    dst[e] = make_float4(__ldg(a.cx + q0 + e), __ldg(a.cy + q0 + e), __ldg(a.cz + q0 + e), 0.0f);
  asm volatile("bar.sync 1, %0;" ::"n"(ms::EPI_WARPS * 32) : "memory");
  return dst;
}

// The insertion of one tile by one epilogue warp: rotation r0 + its lane's row,
// TMEM columns c_beg .. + EPI_COLS (pixels q0 + column).  Sixteen voxels are
// worked out before the first of their atomics: with one pixel at a time, its
// coordinates loaded from global memory between two atomics and U divided by
// T_r and multiplied again, a column took a warp 1,050 clocks (73 us for a tile,
// all of a small problem's M-step and most of a pruned one's).
__device__ __forceinline__ void ms_insert(const TcMstepArgs& a, uint32_t taddr, const float4* xyz,
                                          int q0, int c_beg, int r, bool rok, float Tr, float qs,
                                          const RotMat& Rm) {
  const bool live = rok && Tr > 1e-10f;
  const int side = a.side;
  for (int c0 = c_beg; c0 < c_beg + ms::EPI_COLS; c0 += 16) {
    const int nc = a.P_eff - (q0 + c0);  // columns that are pixels (uniform over the warp)
    if (nc <= 0) break;
    float u[16];
    ptx::tmem_ld16(taddr + c0, u);
    ptx::tmem_wait_ld();
    if (a.u) {  // sorted mode: a coalesced store per column (lanes: rotations)
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (rok && j < nc) a.u[(size_t)(q0 + c0 + j) * a.ldu + r] = live ? u[j] * qs : 0.0f;
    } else if (a.interp == EMC_INTERP_NEAREST) {
      int v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float4 p = xyz[c0 + j];
        const int ix = voxel_round(voxel_coord(side, rotate_row(Rm, 0, p.x, p.y, p.z)));
        const int iy = voxel_round(voxel_coord(side, rotate_row(Rm, 1, p.x, p.y, p.z)));
        const int iz = voxel_round(voxel_coord(side, rotate_row(Rm, 2, p.x, p.y, p.z)));
        const bool in = live && j < nc && (unsigned)ix < (unsigned)side &&
                        (unsigned)iy < (unsigned)side && (unsigned)iz < (unsigned)side;
        v[j] = in ? (iz * side + iy) * side + ix : -1;
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) tc_insert_nearest(a, v[j] >= 0, v[j], u[j] * qs, Tr);
    } else if (__any_sync(0xffffffffu, live)) {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < nc) {
          const float4 p = xyz[c0 + j];
          tc_insert_trilinear(a, live, Rm, p.x, p.y, p.z, u[j] * qs, Tr);
        }
    }
  }
}

// Tile t of the grouped raster (raster_tile over pixel tiles x rotation
// tiles; the default -16: groups of 16 pixel tiles run through all rotation
// tiles, 5-6 % faster than groups of 8 rotation tiles at 128^3 and 256^3).
__device__ __forceinline__ void ms_tile(const TcMstepArgs& a, int t, int& r0, int& q0) {
  int qt, rt;
  raster_tile(t, a.raster, a.n_qt, a.n_rt, qt, rt);
  r0 = rt * ms::BM;
  q0 = qt * ms::BN;
}

// The k-blocks of (rotation tile rt, pixel tile qt): those with counts in the pixel
// tile, of all pattern blocks or (pruned) of the rotation tile's list, of which the
// first is always taken, so that the accumulator is written.  Called by a whole warp,
// which looks at 32 entries at a time (one thread on its own waited for two dependent
// loads per entry, longer than a block's products); f(kb) is called by all lanes and
// returns false, in all, to stop.
template <typename F>
__device__ __forceinline__ bool ms_each_block(const TcMstepArgs& a, int rt, int qt, F&& f) {
  const int lane = threadIdx.x & 31;
  const int* list = a.kb_off ? a.kb_list + a.kb_off[rt] : a.ms_list + (size_t)qt * a.nkb;
  const int n = a.kb_off ? a.kb_off[rt + 1] - a.kb_off[rt] : a.ms_n[qt];
  const unsigned char* map = a.kb_off ? a.ms_map + (size_t)qt * a.nkb : nullptr;
  for (int j0 = 0; j0 < n; j0 += 32) {
    const int j = j0 + lane, kb = j < n ? __ldg(list + j) : 0;
    unsigned m = __ballot_sync(0xffffffffu, j < n && (!map || j == 0 || __ldg(map + kb)));
    for (; m; m &= m - 1)
      if (!f(__shfl_sync(0xffffffffu, kb, __ffs(m) - 1))) return false;
  }
  return true;
}
__device__ __forceinline__ int ms_block_count(const TcMstepArgs& a, int rt, int qt) {
  if (!a.kb_off) return a.ms_n[qt];
  const int lane = threadIdx.x & 31;
  const int* list = a.kb_list + a.kb_off[rt];
  const int n = a.kb_off[rt + 1] - a.kb_off[rt];
  int c = 0;
  for (int j0 = 0; j0 < n; j0 += 32) {
    const int j = j0 + lane;
    const bool on = j < n && (j == 0 || __ldg(a.ms_map + (size_t)qt * a.nkb + __ldg(list + j)));
    c += __popc(__ballot_sync(0xffffffffu, on));
  }
  return c;
}

// Stage ring of the single-CTA M-step: Q hi (+ Q lo) and the 256 K^T rows of
// a 64-pattern k-block.  Without the Q lo slot a stage is 48 KB and four fit
// where three of 64 KB do: a third more bytes in flight for the same ring.
template <int QLO>
struct MsRing {
  static constexpr int kStageBytes = (QLO ? 2 : 1) * ms::A_BYTES + ms::B_BYTES;
  static constexpr int kStages = QLO ? 3 : 4;
  static constexpr int kOffK = (QLO ? 2 : 1) * ms::A_BYTES;  // K^T tile in a stage
  static constexpr int kSmem = kStages * kStageBytes + 256 + ms::XYZ_BYTES + 1024;
  static_assert(kSmem <= 232448, "shared memory of the M-step ring");
};

// Persistent: CTA b takes tiles b, b + grid, ...  The k-block ring runs on
// across tiles, and the accumulator is double-buffered in TMEM (columns
// 0-255 and 256-511), so the insertion epilogue of one tile overlaps the
// MMAs of the next.
template <int QLO>
__global__ void __launch_bounds__(ms::THREADS, 1)
    tc_mstep_kernel(const __grid_constant__ CUtensorMap mQh, const __grid_constant__ CUtensorMap mQl,
                    const __grid_constant__ CUtensorMap mKt, TcMstepArgs a) {
  using namespace ms;
  using Ring = MsRing<QLO>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + Ring::kStages * Ring::kStageBytes);
  uint64_t* empty = full + Ring::kStages;
  uint64_t* tfull = empty + Ring::kStages;  // [2] accumulator ready
  uint64_t* tempty = tfull + 2;      // [2] accumulator drained (one arrival per epilogue warp)
  uint64_t* drain = tempty + 2;      // the MMA issuer's own completion wait before TMEM is freed
  uint32_t* tmem_slot = (uint32_t*)(drain + 1);
  float4* s_xyz = (float4*)(smem + Ring::kStages * Ring::kStageBytes + 256);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < Ring::kStages; ++s) {
      ptx::mbar_init(&full[s], 1);
      ptx::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&tfull[b], 1);
      ptx::mbar_init(&tempty[b], EPI_WARPS);
    }
    ptx::mbar_init(drain, 1);
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------ TMA producer
    uint32_t it = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < a.n_tiles && ok; t += gridDim.x) {
      int r0, q0;
      ms_tile(a, t, r0, q0);
      ok = ms_each_block(a, r0 / BM, q0 / BN, [&](int kb) {
        bool go = true;
        if (ptx::elect_one()) {
          const int s = it % Ring::kStages;
          go = ptx::mbar_wait(&empty[s], ((it / Ring::kStages) & 1) ^ 1, a.status, 4, a.spin);
          if (go) {
            ptx::mbar_arrive_expect_tx(&full[s], Ring::kStageBytes);
            unsigned char* st = smem + s * Ring::kStageBytes;
            ptx::tma_load_2d(st, &mQh, kb * BK, r0, &full[s]);
            if (QLO) ptx::tma_load_2d(st + A_BYTES, &mQl, kb * BK, r0, &full[s]);
            ptx::tma_load_2d(st + Ring::kOffK, &mKt, kb * BK, q0, &full[s]);
          }
        }
        go = __all_sync(0xffffffffu, go);
        it += go;
        return go;
      });
    }
    if (ptx::elect_one())
      ptx::drain_loads(full, Ring::kStages, it, a.status, 11);  // none in flight at exit
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer
    constexpr uint32_t idesc = ptx::idesc_f16(BM, BN);
    uint32_t it = 0;
    bool ok = true;
    int j = 0;
    for (int t = blockIdx.x; t < a.n_tiles && ok; t += gridDim.x, ++j) {
      const int b = j & 1;
      const uint32_t d = tmem + (uint32_t)(b * BN);
      int r0t, q0t;
      ms_tile(a, t, r0t, q0t);
      // a tile with no k-block leaves the buffer as it was: its rotations
      // have no responsibility (T_r = 0), so the epilogue inserts nothing
      const int nk = ms_block_count(a, r0t / BM, q0t / BN);
      if (ptx::elect_one()) {
        const bool drained = ptx::mbar_wait(&tempty[b], ((j >> 1) & 1) ^ 1, a.status, 7, a.spin);
        if (drained) ptx::tc_fence_after();
        ok = drained;
        for (int kb = 0; kb < nk && ok; ++kb) {
          const uint32_t i = it + (uint32_t)kb;
          const int s = i % Ring::kStages;
          if (!ptx::mbar_wait(&full[s], (i / Ring::kStages) & 1, a.status, 5, a.spin)) {
            ok = false;
            break;
          }
          ptx::tc_fence_after();
          const uint32_t base = ptx::smem_u32(smem + s * Ring::kStageBytes);
#pragma unroll
          for (int ks = 0; ks < BK / 16; ++ks) {
            const uint64_t dQh = ptx::smem_desc(base + ks * 32, 1024, 2);
            const uint64_t dQl = ptx::smem_desc(base + A_BYTES + ks * 32, 1024, 2);
            const uint64_t dK = ptx::smem_desc(base + Ring::kOffK + ks * 32, 1024, 2);
            ptx::mma_f16(d, dQh, dK, idesc, (kb | ks) ? 1u : 0u);
            if (QLO) ptx::mma_f16(d, dQl, dK, idesc, 1u);
          }
          ptx::mma_commit(&empty[s]);
        }
        if (drained) ptx::mma_commit(&tfull[b]);  // fires when this tile's MMAs have completed
      }
      ok = __all_sync(0xffffffffu, ok);
      it += (uint32_t)nk;
    }
    if (ptx::elect_one()) {
      ptx::mma_commit(drain);  // TMEM is freed only after every MMA issued here has completed
      ptx::mbar_wait(drain, 0, a.status, 12);
    }
  } else {
    // ------------------------------------------------ insertion epilogue
    const int quarter = warp & 3;       // TMEM lanes this warp may access
    const int part = (warp - 2) >> 2;   // which of the tile's columns
    const int rl = quarter * 32 + lane;
    bool ok = true;
    int j = 0;
    for (int t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ++j) {
      const int b = j & 1;
      int r0, q0;
      ms_tile(a, t, r0, q0);
      const int r = r0 + rl;
      const bool rok = r < a.R;
      const float Tr = rok ? a.T[r] : 0.0f;
      const float qs = rok ? a.qscale[r] * a.k_inv : 0.0f;
      RotMat Rm = {};
      if (rok) Rm = quat_to_matrix(a.rot + 4 * (size_t)r);
      const float4* xyz = ms_stage_pixels(a, s_xyz, j, q0);
      // after a wait that gave up the warp only keeps the other warps' barrier going
      ok = ok && ptx::mbar_wait_sleep(&tfull[b], (j >> 1) & 1, a.status, 6, 128, a.spin);
      if (ok) {
        ptx::tc_fence_after();
        ms_insert(a, tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * BN), xyz, q0,
                  part * EPI_COLS, r, rok, Tr, qs, Rm);
      }
      // this warp's reads of buffer b are complete: hand it back to the MMA warp
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&tempty[b]);
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 32) ptx::settle_after_timeout(a.status);
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------- M-step on CTA pairs -----
// The M-step's tiles as 256 rotations x 256 pixels per cluster of two CTAs:
// 256-row MMAs (cta_group::2) issued by rank 0, each CTA holding the Q rows
// of its own 128 rotations and 128 of the tile's 256 pixel rows of K^T.  Per
// 64-pattern stage a CTA loads 32 KB instead of 48 KB for the same MMA work
// and its tensor core reads half of the pixel-side operand.  Persistent over
// the cluster's tiles; each CTA's TMEM holds its 128 rotations x 256 pixels,
// double-buffered (2 x 256 columns), so the insertion epilogue of one tile
// overlaps the MMAs of the next.  Both CTAs' loads complete on rank 0's
// `full` barriers; rank 0's commits multicast to both CTAs' `empty` and
// `tfull`; the epilogue warps of both CTAs hand a buffer back on rank 0's
// `tempty`.  Full scans, and pruned ones whose lists span the pair's 256 rotations
// (true Poisson); the pruned reference likelihood's M-step runs single CTAs.
namespace ms2 {
constexpr int A_BYTES = ms::BM * ms::BK * 2;  // 16 KB: 128 rotations x 64 patterns
constexpr int B_BYTES = 128 * ms::BK * 2;     // 16 KB: 128 pixels x 64 patterns
// stage: Q hi (+ Q lo) and the CTA's half of K^T; six 32 KB stages without
// the Q lo slot, four of 48 KB with it
template <int QLO>
struct Ring {
  static constexpr int kStageBytes = (QLO ? 2 : 1) * A_BYTES + B_BYTES;
  static constexpr int kStages = QLO ? 4 : 6;
  static constexpr int kOffK = (QLO ? 2 : 1) * A_BYTES;
  static constexpr int kSmem = kStages * kStageBytes + 256 + ms::XYZ_BYTES + 1024;
  static_assert(kSmem <= 232448, "shared memory of the pair M-step");
};
}  // namespace ms2

template <int QLO>
__global__ void __launch_bounds__(ms::THREADS, 1)
    tc_mstep_pair_kernel(const __grid_constant__ CUtensorMap mQh,
                         const __grid_constant__ CUtensorMap mQl,
                         const __grid_constant__ CUtensorMap mKt128, TcMstepArgs a) {
  using namespace ms;
  constexpr int STAGES = ms2::Ring<QLO>::kStages;
  constexpr int STAGE_BYTES = ms2::Ring<QLO>::kStageBytes;
  constexpr int OFF_K = ms2::Ring<QLO>::kOffK;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;  // [2] accumulator ready (both CTAs)
  uint64_t* tempty = tfull + 2;      // [2] rank 0: accumulator drained by both CTAs
  uint64_t* drain = tempty + 2;      // rank 0's MMA issuer waits on it before TMEM is freed
  uint32_t* tmem_slot = (uint32_t*)(drain + 1);
  float4* s_xyz = (float4*)(smem + STAGES * STAGE_BYTES + 256);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  const int cl = (int)(blockIdx.x >> 1), ncl = (int)(gridDim.x >> 1);
  const int n_rp = (a.n_rt + 1) / 2;  // rotation-tile pairs
  const int n_tiles = n_rp * a.n_qt;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&full[s], 1);
      ptx::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&tfull[b], 1);
      ptx::mbar_init(&tempty[b], 2 * EPI_WARPS);
    }
    ptx::mbar_init(drain, 1);
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(tmem_slot, 512);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();  // both CTAs' barriers initialised and TMEM allocated
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------ TMA producer (both CTAs)
    uint32_t it = 0;
    bool ok = true;
    for (int t = cl; t < n_tiles && ok; t += ncl) {
      int qt, rp;
      raster_tile(t, a.raster, a.n_qt, n_rp, qt, rp);
      const int r0 = (2 * rp + (int)rank) * BM, q0 = qt * BN + 128 * (int)rank;
      ok = ms_each_block(a, 2 * rp, qt, [&](int kb) {
        bool go = true;
        if (ptx::elect_one()) {
          const int s = it % STAGES;
          go = ptx::mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1, a.status, 4, a.spin);
          if (go) {
            // both CTAs' loads
            if (rank == 0) ptx::mbar_arrive_expect_tx(&full[s], 2 * STAGE_BYTES);
            const uint32_t fb = ptx::mapa_shared(ptx::smem_u32(&full[s]), 0);
            unsigned char* st = smem + s * STAGE_BYTES;
            ptx::tma_load_2d_pair(st, &mQh, kb * BK, r0, fb);
            if (QLO) ptx::tma_load_2d_pair(st + ms2::A_BYTES, &mQl, kb * BK, r0, fb);
            ptx::tma_load_2d_pair(st + OFF_K, &mKt128, kb * BK, q0, fb);
          }
        }
        go = __all_sync(0xffffffffu, go);
        it += go;
        return go;
      });
    }
    // rank 0's barriers count both CTAs' bytes of the stages it armed
    if (rank == 0 && ptx::elect_one()) ptx::drain_loads(full, STAGES, it, a.status, 11);
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer (rank 0)
    if (rank == 0) {
      constexpr uint32_t idesc = ptx::idesc_f16(2 * BM, BN);  // 256 x 256
      uint32_t it = 0;
      bool ok = true;
      int j = 0;
      for (int t = cl; t < n_tiles && ok; t += ncl, ++j) {
        const int b = j & 1;
        const uint32_t d = tmem + (uint32_t)(b * BN);
        int qt, rp;
        raster_tile(t, a.raster, a.n_qt, n_rp, qt, rp);
        const int nk = ms_block_count(a, 2 * rp, qt);
        if (ptx::elect_one()) {
          const bool drained =
              ptx::mbar_wait_cluster(&tempty[b], ((j >> 1) & 1) ^ 1, a.status, 7, a.spin);
          if (drained) ptx::tc_fence_after();
          ok = drained;
          for (int kb = 0; kb < nk && ok; ++kb) {
            const uint32_t i = it + (uint32_t)kb;
            const int s = i % STAGES;
            if (!ptx::mbar_wait(&full[s], (i / STAGES) & 1, a.status, 5, a.spin)) {
              ok = false;
              break;
            }
            ptx::tc_fence_after();
            const uint32_t base = ptx::smem_u32(smem + s * STAGE_BYTES);
#pragma unroll
            for (int ks = 0; ks < BK / 16; ++ks) {
              const uint64_t dQh = ptx::smem_desc(base + ks * 32, 1024, 2);
              const uint64_t dQl = ptx::smem_desc(base + ms2::A_BYTES + ks * 32, 1024, 2);
              const uint64_t dK = ptx::smem_desc(base + OFF_K + ks * 32, 1024, 2);
              ptx::mma_f16_pair(d, dQh, dK, idesc, (kb | ks) ? 1u : 0u);
              if (QLO) ptx::mma_f16_pair(d, dQl, dK, idesc, 1u);
            }
            ptx::mma_commit_pair(&empty[s], 0x3);
          }
          if (drained) ptx::mma_commit_pair(&tfull[b], 0x3);  // when this tile's MMAs have completed
        }
        ok = __all_sync(0xffffffffu, ok);
        it += (uint32_t)nk;
      }
      if (ptx::elect_one()) {
        ptx::mma_commit_pair(drain, 0x1);  // both CTAs' TMEM is written by these MMAs
        ptx::mbar_wait(drain, 0, a.status, 12);
      }
    }
  } else {
    // ------------------------------------------------ insertion epilogue
    const int quarter = warp & 3;      // TMEM lanes this warp may access
    const int part = (warp - 2) >> 2;  // which of the tile's columns
    const int rl = quarter * 32 + lane;
    bool ok = true;
    const uint32_t back = rank == 0 ? 0u : 1u;
    int j = 0;
    for (int t = cl; t < n_tiles; t += ncl, ++j) {
      const int b = j & 1;
      int qt, rp;
      raster_tile(t, a.raster, a.n_qt, n_rp, qt, rp);
      const int r0 = (2 * rp + (int)rank) * BM, q0 = qt * BN;  // TMEM column c: pixel q0 + c
      const int r = r0 + rl;
      const bool rok = r < a.R;
      const float Tr = rok ? a.T[r] : 0.0f;
      const float qs = rok ? a.qscale[r] * a.k_inv : 0.0f;
      RotMat Rm = {};
      if (rok) Rm = quat_to_matrix(a.rot + 4 * (size_t)r);
      const float4* xyz = ms_stage_pixels(a, s_xyz, j, q0);
      // after a wait that gave up the warp only keeps the other warps' barrier going
      ok = ok && ptx::mbar_wait_sleep(&tfull[b], (j >> 1) & 1, a.status, 6, 128, a.spin);
      if (ok) {
        ptx::tc_fence_after();
        ms_insert(a, tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * BN), xyz, q0,
                  part * EPI_COLS, r, rok, Tr, qs, Rm);
      }
      // this warp's reads of buffer b are complete: hand it back to rank 0's MMA warp
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (back)
          ptx::mbar_arrive_cluster(ptx::mapa_shared(ptx::smem_u32(&tempty[b]), 0));
        else
          ptx::mbar_arrive(&tempty[b]);
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();  // the pair's MMAs and barrier traffic are over in both CTAs
  if (threadIdx.x == 32) ptx::settle_after_timeout(a.status);
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_pair(tmem, 512);
  }
}

// ------------------------------------------------------------ host -------
struct TcState {
  CUtensorMap mK, mJ, mJl, mQh, mQl, mKt;
  CUtensorMap mKt128;  // K^T in 128-row boxes (pair M-step halves)
  CUtensorMap mMS, mHh, mHl, mIv, mTv, mMSl;  // rotation operands: 64-row boxes
  CUtensorMap mLh, mLl;  // true Poisson, single CTAs: log-slices hi / lo, 256 rows x 32
  CUtensorMap mK64, mLh64, mLl64;  // and pairs: 128 rows x 64
  __half *MS, *Hh, *Hl, *Iv, *Tv, *MSl, *Lh, *Ll;
  int* status;
};

static TcState* state(emc_plan* p) { return (TcState*)p->tc; }

int tc_bind(emc_plan* p) {
  emc_ctx* ctx = p->ctx;
  if (!p->counts_integer || (!p->counts_fp16_exact && !p->counts_round))
    return fail(ctx, EMC_ERR_UNSUPPORTED,
                "mixed precision needs integer counts in [0, 2048] (exact in FP16), or in [0, "
                "65504] with EMC_OPT_COUNTS_ROUND (largest count here %d)", p->count_max);
  if (p->d.diff != EMC_DIFF_POISSON && p->d.diff != EMC_DIFF_TRUE_POISSON)
    return fail(ctx, EMC_ERR_UNSUPPORTED,
                "mixed precision implements the poisson and true-poisson likelihoods");
  const bool pois = p->d.diff == EMC_DIFF_TRUE_POISSON;
  const int Np = p->Np, Kp = p->Kp, Rp = p->Rp;
  if (pois) {
    p->count_scale = 1.0f;
  } else {
    // the largest FP16 count squared times the scale stays below 2^15
    const float km = __half2float(__float2half_rn((float)p->count_max));
    int e = 7;
    while (km * km * std::ldexp(1.0f, -e) > 32768.0f) ++e;
    p->count_scale = std::ldexp(1.0f, -e);
  }
  int rc = EMC_OK;
  if (!p->tc) {
    TcState* st = new TcState();
    std::memset(st, 0, sizeof(*st));
    p->tc = st;
    const size_t pk = (size_t)Np * Kp, rk = (size_t)Rp * Kp;
    if (!rc) rc = plan_alloc(p, (void**)&p->Kh, pk * 2);
    if (!rc) rc = plan_alloc(p, (void**)&p->KhT, pk * 2);
    const size_t n_pt = (size_t)(Np / 128), nkb = (size_t)(Kp / 64), n_pp = (n_pt + 1) / 2;
    if (!rc) rc = plan_alloc(p, (void**)&p->blk_bits, n_pt * nkb);
    if (!rc) rc = plan_alloc(p, (void**)&p->blk_live, nkb);
    if (!rc) rc = plan_alloc(p, (void**)&p->pt_list, n_pt * nkb * 4);
    if (!rc) rc = plan_alloc(p, (void**)&p->pt_n, n_pt * 4);
    if (!rc) rc = plan_alloc(p, (void**)&p->pp_list, n_pp * nkb * 4);
    if (!rc) rc = plan_alloc(p, (void**)&p->pp_n, n_pp * 4);
    const size_t n_qt = (size_t)ceil_div(Kp, ms::BN), npb = 2 * n_pt;
    if (!rc) rc = plan_alloc(p, (void**)&p->sub_any, nkb * npb);
    if (!rc) rc = plan_alloc(p, (void**)&p->ms_map, n_qt * npb);
    if (!rc) rc = plan_alloc(p, (void**)&p->ms_list, n_qt * npb * 4);
    if (!rc) rc = plan_alloc(p, (void**)&p->ms_n, n_qt * 4);
    if (!pois) {
      if (!rc) rc = plan_alloc(p, (void**)&p->Jh, pk * 2);
      if (!rc) rc = plan_alloc(p, (void**)&p->Jl, pk * 2);
      if (!rc) rc = plan_alloc(p, (void**)&p->ktot, (size_t)Np * 4);
      if (!rc) rc = plan_alloc(p, (void**)&p->k2tot, (size_t)Np * 4);
      if (!rc) rc = plan_alloc(p, (void**)&p->lo_kb, sizeof(int) * (n_pt + 2));
      p->d_bright = p->lo_kb + n_pt + 1;
      if (!rc) rc = plan_alloc(p, (void**)&p->rot_flags, (2 * (size_t)p->n_rt * nkb + 15) / 16 * 16);
    }
    __half** pois_ops[] = {&st->Lh, &st->Ll};
    __half** rot_ops[] = {&st->MS, &st->Hh, &st->Hl, &st->Iv, &st->Tv};
    for (int j = 0; j < (pois ? 2 : 5); ++j) {
      __half** op = pois ? pois_ops[j] : rot_ops[j];
      if (!rc) rc = plan_alloc(p, (void**)op, rk * 2);
      // rows R..Rp stay zero: the expand writes the operands of rows < R
      if (!rc) EMC_CUDA(ctx, cudaMemsetAsync(*op, 0, rk * 2, ctx->stream));
    }
    if (!rc) rc = plan_alloc(p, (void**)&p->Qh, (size_t)Rp * Np * 2);
    if (!rc) rc = plan_alloc(p, (void**)&p->qscale, (size_t)Rp * 4);
    if (!rc) rc = plan_alloc(p, (void**)&st->status, 64);
    if (rc) return rc;
    EMC_CUDA(ctx, cudaMemsetAsync(st->status, 0, 64, ctx->stream));
    EMC_CUDA(ctx, cudaMemsetAsync(p->Qh, 0, (size_t)Rp * Np * 2, ctx->stream));
    // tensor maps (fixed addresses for the plan's lifetime)
    if (pois) {
      if (!rc) rc = make_map(ctx, &st->mK, p->Kh, Np, Kp, 128, 32);
      if (!rc) rc = make_map(ctx, &st->mLh, st->Lh, Rp, Kp, 256, 32);
      if (!rc) rc = make_map(ctx, &st->mLl, st->Ll, Rp, Kp, 256, 32);
      if (!rc) rc = make_map(ctx, &st->mK64, p->Kh, Np, Kp, 128, 64);
      if (!rc) rc = make_map(ctx, &st->mLh64, st->Lh, Rp, Kp, 128, 64);
      if (!rc) rc = make_map(ctx, &st->mLl64, st->Ll, Rp, Kp, 128, 64);
    } else {
      if (!rc) rc = make_map(ctx, &st->mK, p->Kh, Np, Kp, 128, 64);
      if (!rc) rc = make_map(ctx, &st->mJ, p->Jh, Np, Kp, 128, 64);
      if (!rc) rc = make_map(ctx, &st->mJl, p->Jl, Np, Kp, 128, 64);
      CUtensorMap* rm[] = {&st->mMS, &st->mHh, &st->mHl, &st->mIv, &st->mTv};
      for (int j = 0; j < 5 && !rc; ++j) rc = make_map(ctx, rm[j], *rot_ops[j], Rp, Kp, 64, 64);
    }
    if (!rc) rc = make_map(ctx, &st->mQh, p->Qh, Rp, Np, 128, 64);
    if (!rc) rc = make_map(ctx, &st->mKt, p->KhT, Kp, Np, 256, 64);
    if (!rc) rc = make_map(ctx, &st->mKt128, p->KhT, Kp, Np, 128, 64);
    if (rc) return rc;
    for (auto* k : {tc_estep_kernel<false, false>, tc_estep_kernel<false, true>,
                    tc_estep_kernel<true, false>, tc_estep_kernel<true, true>})
      EMC_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         es::SMEM_BYTES));
    EMC_CUDA(ctx, cudaFuncSetAttribute(tc_estep_pois_kernel<false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       ep::Ring<false>::kSmem));
    EMC_CUDA(ctx, cudaFuncSetAttribute(tc_estep_pois_kernel<true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       ep::Ring<true>::kSmem));
    EMC_CUDA(ctx, cudaFuncSetAttribute(tc_mstep_kernel<0>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       MsRing<0>::kSmem));
    EMC_CUDA(ctx, cudaFuncSetAttribute(tc_mstep_kernel<1>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       MsRing<1>::kSmem));
    EMC_CUDA(ctx, cudaFuncSetAttribute(tc_mstep_pair_kernel<0>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       ms2::Ring<0>::kSmem));
    EMC_CUDA(ctx, cudaFuncSetAttribute(tc_mstep_pair_kernel<1>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       ms2::Ring<1>::kSmem));
  }
  if (p->mstep_q_lo && (rc = tc_ensure_qlo(p))) return rc;
  if ((rc = tc_ensure_mslo(p))) return rc;
  // counts already in FP16 from the bind's pattern pass when its scale holds
  if ((rc = tc_pattern_side(p, nullptr, p->fused_scale == p->count_scale))) return rc;
  p->bright = false;
  if (p->d_bright) {  // which kernels the iterations launch
    int bright = 0;
    EMC_CUDA(ctx, cudaMemcpyAsync(&bright, p->d_bright, sizeof(int), cudaMemcpyDeviceToHost,
                                  ctx->stream));
    EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    p->bright = bright != 0;
  }
  return EMC_OK;
}

// FP16 pattern operands for the pattern order perm (position -> input
// pattern; nullptr: input order).
// counts_done: the pattern pass already wrote Kh at the current scale (rows
// < N; the padding rows stay zero from the first bind).
int tc_pattern_side(emc_plan* p, const int* d_perm, bool counts_done) {
  emc_ctx* ctx = p->ctx;
  const int N = p->d.n_images, Np = p->Np, Kp = p->Kp;
  int rc;
  if (!counts_done) {
    tc_pattern_ops_kernel<<<(unsigned)Np * (unsigned)ceil_div(Kp, 256), 256, 0, ctx->stream>>>(
        p->images, p->pix, p->n2, N, Kp, p->Kh, d_perm, p->count_scale);
    if ((rc = after_launch(ctx, "tc_pattern_ops_kernel"))) return rc;
  }
  const int n_pt = Np / es::BM;
  tc_count_blocks_kernel<<<dim3(Kp / es::BK, (n_pt + 1) / 2), 256, 0, ctx->stream>>>(
      p->Kh, Kp, Kp / es::BK, n_pt, p->count_scale, p->Jh, p->Jl, p->blk_bits, p->sub_any);
  if ((rc = after_launch(ctx, "tc_count_blocks_kernel"))) return rc;
  if ((rc = tc_block_lists(p))) return rc;
  transpose_h_kernel<<<dim3(ceil_div(Kp, 64), ceil_div(Np, 64)), dim3(32, 8), 0, ctx->stream>>>(
      p->Kh, Np, Kp, p->KhT);
  return after_launch(ctx, "transpose_h_kernel");
}

int* tc_status(emc_plan* p) { return p->tc ? state(p)->status : nullptr; }

__half* tc_tiny_plane(emc_plan* p) { return state(p)->Tv; }

int tc_block_lists(emc_plan* p) {
  emc_ctx* ctx = p->ctx;
  const int nkb = p->Kp / es::BK, n_pt = p->Np / es::BM;
  int rc;
  if (p->lo_kb) {
    EMC_CUDA(ctx, cudaMemsetAsync(p->lo_kb, 0, sizeof(int) * (size_t)(n_pt + 2), ctx->stream));
    tc_count_rows_kernel<<<ceil_div(p->d.n_images, 8), 256, 0, ctx->stream>>>(
        p->Kh, p->Kp, nkb, p->d.n_images, p->count_scale, (float)p->hlo_tail_ppm * 1e-6f, p->ktot,
        p->k2tot, p->lo_kb, p->d_bright);
    if ((rc = after_launch(ctx, "tc_count_rows_kernel"))) return rc;
  }
  const int n_qt = ceil_div(p->Kp, ms::BN);
  tc_block_lists_kernel<<<n_qt + n_pt + (n_pt + 1) / 2 + ceil_div(nkb, 32), 32, 0, ctx->stream>>>(
      p->blk_bits, n_pt, nkb, p->lo_kb, p->pt_list, p->pt_n, p->pp_list, p->pp_n, p->blk_live,
      p->sub_any, n_qt, p->ms_map, p->ms_list, p->ms_n);
  return after_launch(ctx, "tc_block_lists_kernel");
}

// The FP16 lo half of the M-step operand and its tensor map, allocated the
// first time an M-step that uses it is requested (it is never read otherwise).
int tc_ensure_qlo(emc_plan* p) {
  if (!p->tc || p->Ql) return EMC_OK;
  emc_ctx* ctx = p->ctx;
  const size_t bytes = (size_t)p->Rp * p->Np * 2;
  int rc = plan_alloc(p, (void**)&p->Ql, bytes);
  if (rc) return rc;
  EMC_CUDA(ctx, cudaMemsetAsync(p->Ql, 0, bytes, ctx->stream));
  return make_map(ctx, &state(p)->mQl, p->Ql, p->Rp, p->Np, 128, 64);
}

// M'S in every product as hi + lo: with H lo everywhere, where a scaling is fitted.
static bool estep_ms_lo(const emc_plan* p) {
  return p->d.diff != EMC_DIFF_TRUE_POISSON && !p->d.known_intensity && p->estep_gh_lo >= 0 &&
         (p->estep_gh_lo & 2);
}

// Its plane and tensor map, allocated the first time it is asked for.
int tc_ensure_mslo(emc_plan* p) {
  if (!p->tc || !estep_ms_lo(p) || state(p)->MSl) return EMC_OK;
  emc_ctx* ctx = p->ctx;
  const size_t bytes = (size_t)p->Rp * p->Kp * 2;
  __half* plane = nullptr;
  int rc = plan_alloc(p, (void**)&plane, bytes);
  if (rc) return rc;
  // rows R..Rp stay zero, as those of the other operands
  EMC_CUDA(ctx, cudaMemsetAsync(plane, 0, bytes, ctx->stream));
  if ((rc = make_map(ctx, &state(p)->mMSl, plane, p->Rp, p->Kp, 64, 64))) return rc;
  state(p)->MSl = plane;
  return EMC_OK;
}

// A kernel on clusters of two CTAs.
template <typename... P, typename... A>
static cudaError_t launch_pairs(emc_ctx* ctx, void (*kernel)(P...), int pairs, int threads, int smem,
                                const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// The true-Poisson likelihood over tiles [first, first + count) of the full
// (pattern tile, rotation tile) grid in the order `raster`, or over the plan's
// pruned tile list (full == false and a list exists; first/count ignored).  Full
// scans run on CTA pairs unless those are switched off: half the reads of the
// log-slices per pattern; the pruned lists name single pattern tiles.
static int estep_pois_launch(emc_plan* p, int raster, int first, int count, bool full) {
  emc_ctx* ctx = p->ctx;
  TcState* st = state(p);
  TcEstepPoisArgs a;
  a.N = p->d.n_images;
  a.R = p->d.n_rot;
  a.n_rt = ceil_div(p->Rp, ep::BN);
  a.nkb = p->Kp / ep::BK;
  a.raster = raster;
  a.tiles = full ? nullptr : p->prune_tiles;
  a.n_part = p->n_rt;
  a.rot_ssum = p->rot_ssum;
  a.rotw = p->rotw;
  a.Ksum = p->Ksum;
  a.cnorm = p->cnorm;
  a.known_intensity = p->d.known_intensity;
  a.L = p->L;
  a.PHI = p->PHI;
  a.part = p->part;
  a.status = st->status;
  a.spin = p->debug_spin ? p->debug_spin : ptx::kSpinLimit;
  const int n_pt = p->Np / ep::BM;
  if (p->estep_pair && !a.tiles) {
    a.n_pt = (n_pt + 1) / 2;
    a.list = p->pp_list;
    a.list_n = p->pp_n;
    const int total = a.n_pt * a.n_rt;
    a.tile0 = std::max(0, std::min(first, total));
    a.n_tiles = std::min(total - a.tile0, count);
    if (a.n_tiles == 0) return EMC_OK;
    const cudaError_t e =
        launch_pairs(ctx, tc_estep_pois_kernel<true>, std::min(a.n_tiles, ctx->sm_count / 2),
                     ep::THREADS, ep::Ring<true>::kSmem, st->mK64, st->mLh64, st->mLl64, a);
    if (e == cudaSuccess) return after_launch(ctx, "tc_estep_pois_kernel (pairs)");
    // as in estep_launch: no pairs on this device, single CTAs from now on
    (void)cudaGetLastError();
    p->estep_pair = 0;
    first *= 2;
    count = count > INT_MAX / 2 ? INT_MAX : 2 * count;
  }
  a.n_pt = n_pt;
  a.list = p->pt_list;
  a.list_n = p->pt_n;
  const int total = a.n_pt * a.n_rt;
  a.tile0 = a.tiles ? 0 : std::max(0, std::min(first, total));
  a.n_tiles = a.tiles ? p->prune_n_tiles : std::min(total - a.tile0, count);
  if (a.n_tiles == 0) return EMC_OK;
  tc_estep_pois_kernel<false>
      <<<std::min(a.n_tiles, ctx->sm_count), ep::THREADS, ep::Ring<false>::kSmem, ctx->stream>>>(
          st->mK, st->mLh, st->mLl, a);
  return after_launch(ctx, "tc_estep_pois_kernel");
}

// The halves of H in force: bit 0 H lo in K . H before the count tail, bit 1 in
// every product (auto: when the intensity is known -- phi = 1 leaves the
// C = K^2 . H term unbalanced, and its rounding then shows in the likelihood).
static int estep_gh_lo(const emc_plan* p) {
  return p->estep_gh_lo >= 0 ? p->estep_gh_lo : (p->d.known_intensity ? 3 : 1);
}

static int estep_launch(emc_plan* p, int raster, int first, int count, bool full) {
  if (p->d.diff == EMC_DIFF_TRUE_POISSON) return estep_pois_launch(p, raster, first, count, full);
  emc_ctx* ctx = p->ctx;
  TcState* st = state(p);
  TcEstepArgs a;
  a.N = p->d.n_images;
  a.R = p->d.n_rot;
  a.n_pt = p->Np / es::BM;
  a.n_rt = p->Rp / es::BN;
  a.nkb = p->Kp / es::BK;
  a.raster = raster;
  a.gh_lo = estep_gh_lo(p);
  a.tiles = full ? nullptr : p->prune_tiles;
  a.rot_inv = p->rot_flags;
  a.rot_tiny = p->rot_flags + (size_t)a.n_rt * a.nkb;
  a.rot_cnt = p->rot_cnt;
  a.rot_A = p->rot_A;
  a.rotw = p->rotw;
  a.cnorm = p->cnorm;
  a.ktot = p->ktot;
  a.k2tot = p->k2tot;
  a.k_inv = 1.0f / p->count_scale;
  a.ms_lo = estep_ms_lo(p) && st->MSl;
  a.zrow = p->Rp;
  a.sigma = p->sigma_dev;
  a.known_intensity = p->d.known_intensity;
  a.L = p->L;
  a.PHI = p->PHI;
  a.part = p->part;
  a.bad = p->flags + 4;
  a.status = st->status;
  a.spin = p->debug_spin ? p->debug_spin : ptx::kSpinLimit;
  if (p->estep_pair && !a.tiles) {
    // CTA pairs: tiles are (pattern-tile pair, rotation tile)
    a.list = p->pp_list;
    a.list_n = p->pp_n;
    const int total = ((a.n_pt + 1) / 2) * a.n_rt;
    first = std::max(0, std::min(first, total));
    const int pairs = std::min(total - first, count);
    a.tile0 = first;
    if (pairs == 0) return EMC_OK;
    auto* kernel = p->bright ? tc_estep_kernel<true, true> : tc_estep_kernel<true, false>;
    const cudaError_t e =
        launch_pairs(ctx, kernel, pairs, es::THREADS, es::SMEM_BYTES, st->mK, st->mJ, st->mJl,
                     st->mMS, st->mHh, st->mHl, st->mIv, st->mTv, st->mMSl, a);
    if (e == cudaSuccess) return after_launch(ctx, "tc_estep_kernel (pairs)");
    // a refused launch configuration (a GPU or partition that cannot
    // co-schedule the pairs) is not a sticky error: single CTAs from now on
    (void)cudaGetLastError();
    p->estep_pair = 0;
    first *= 2;  // about the same part of the grid, in single-CTA tiles
    count = count > INT_MAX / 2 ? INT_MAX : 2 * count;
  }
  a.list = p->pt_list;
  a.list_n = p->pt_n;
  const int total = a.n_pt * a.n_rt;
  first = a.tiles ? 0 : std::max(0, std::min(first, total));
  const int grid = a.tiles ? p->prune_n_tiles : std::min(total - first, count);
  a.tile0 = first;
  if (grid == 0) return EMC_OK;
  auto* kernel = p->bright ? tc_estep_kernel<false, true> : tc_estep_kernel<false, false>;
  kernel<<<grid, es::THREADS, es::SMEM_BYTES, ctx->stream>>>(
      st->mK, st->mJ, st->mJl, st->mMS, st->mHh, st->mHl, st->mIv, st->mTv, st->mMSl, a);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(ctx, e, "tc_estep_kernel launch");
  return after_launch(ctx, "tc_estep_kernel");
}

// The rotation operands are written by the expand (rot_ops_store4).
int tc_estep(emc_plan* p) { return estep_launch(p, p->estep_raster, 0, INT_MAX, false); }

RotOps tc_rot_ops(emc_plan* p) {
  RotOps o;
  if (!p->tc) return o;
  TcState* st = state(p);
  o.flags = p->flags;
  o.live = p->blk_live;
  o.nkb = p->Kp / es::BK;
  if (p->d.diff == EMC_DIFF_TRUE_POISSON) {
    o.Lh = st->Lh;
    o.Ll = st->Ll;
    return o;
  }
  const int gh = estep_gh_lo(p);
  o.MS = st->MS;
  o.Hh = st->Hh;
  o.Iv = st->Iv;
  o.bright = p->bright;
  o.inv = p->rot_flags;
  o.tiny = p->rot_flags + (size_t)p->n_rt * o.nkb;
  o.Hl = gh ? st->Hl : nullptr;
  o.MSl = estep_ms_lo(p) ? st->MSl : nullptr;
  if (gh == 1) o.hl_end = p->lo_kb + p->Np / es::BM;
  return o;
}

// One timed launch of the likelihood kernel over tiles [first, first + count)
// of the order `raster` (CUDA events on the plan's stream; synchronises).  The
// rotation operands are those of the last expansion.
int tc_time_estep(emc_plan* p, int raster, int first, int count, float* ms) {
  emc_ctx* ctx = p->ctx;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  EMC_CUDA(ctx, cudaEventCreate(&e0));
  cudaError_t ce = cudaEventCreate(&e1);
  int rc = EMC_OK;
  if (ce == cudaSuccess) ce = cudaEventRecord(e0, ctx->stream);
  if (ce == cudaSuccess && !(rc = estep_launch(p, raster, first, count, true)))
    ce = cudaEventRecord(e1, ctx->stream);
  if (ce == cudaSuccess && !rc) ce = cudaEventSynchronize(e1);
  if (ce == cudaSuccess && !rc) ce = cudaEventElapsedTime(ms, e0, e1);
  if (ce != cudaSuccess && !rc) rc = cuda_fail(ctx, ce, "likelihood timing");
  cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  return rc;
}

// Units of the full likelihood grid as estep_launch counts them: tiles, or
// CTA-pair tiles for the pair kernel.
int tc_estep_tiles(emc_plan* p) {
  const int n_pt = p->Np / 128;
  return (p->estep_pair ? (n_pt + 1) / 2 : n_pt) *
         (p->d.diff == EMC_DIFF_TRUE_POISSON ? ceil_div(p->Rp, ep::BN) : p->Rp / es::BN);
}

// Raster autotuner.  The likelihood kernel streams two operand panels per
// CTA (the pattern tile's and the rotation tile's, 128 rows x the compacted
// pixel count each); which CTAs run side by side decides how often a panel
// is served from L2 rather than HBM, and the best order depends on the panel
// length and the tile counts: on 256^3 workloads (51,020 pixels) groups of 4
// rotation tiles run at 5.7 ms per 1,000 tiles while groups of 8 swing
// between 5.5 and 10.3 ms depending on where in the grid they are timed; at
// 128^3 all orders are within 5 %.  Candidates: groups of 2..16 rotation
// tiles, or of 8..76 pattern tiles.  Each is timed on two windows of `waves`
// x SM-count tiles inside the grid (at 30 % and 65 % of its order; the whole
// grid when it is smaller) and scored by the slower window, so an order that
// is fast only at times loses to a steady one.  The rotation operands are
// those of the last expansion; the timed launches overwrite
// responsibilities and scaling of the tiles they cover.
int tc_autotune(emc_plan* p, int waves, int* best, float* best_ms) {
  emc_ctx* ctx = p->ctx;
  int rc = EMC_OK;
  const bool pois = p->d.diff == EMC_DIFF_TRUE_POISSON;
  const bool pair = p->estep_pair != 0;
  const int n_pt = pair ? (p->Np / 128 + 1) / 2 : p->Np / 128;
  const int n_rt = pois ? ceil_div(p->Rp, ep::BN) : p->Rp / es::BN;
  const int total = n_pt * n_rt;
  const int count = std::min(total, std::max(1, waves) * (pair ? ctx->sm_count / 2 : ctx->sm_count));
  std::vector<int> firsts;
  if (count >= total) {
    firsts.push_back(0);
  } else {
    for (double f : {0.30, 0.65})
      firsts.push_back(std::min(total - count, (int)(f * total)));
  }
  std::vector<int> cand;
  for (int g : {8, 2, 4, 16, -8, -19, -38, -76}) {
    const int c = g > 0 ? std::min(g, n_rt) : -std::min(-g, n_pt);
    if (std::find(cand.begin(), cand.end(), c) == cand.end()) cand.push_back(c);
  }
  std::vector<float> t(cand.size(), 0.0f);
  for (size_t j = 0; j < cand.size() && !rc; ++j) {
    for (int first : firsts) {
      float ms = 0.0f;
      if ((rc = tc_time_estep(p, cand[j], first, count, &ms))) break;
      t[j] = std::max(t[j], ms);
    }
  }
  if (rc) return rc;
  // the default order (first candidate) unless another is 2 % faster: orders
  // that tie in time differ in HBM traffic (at 128^3 from 63 to 217 GB per
  // launch), and the default one reads the least there
  size_t b = 0;
  for (size_t j = 1; j < cand.size(); ++j)
    if (t[j] < t[b]) b = j;
  if (t[0] <= 1.02f * t[b]) b = 0;
  int raster = cand[b];
  float raster_ms = t[b];
  // tile shape: CTA pairs (256 patterns x 128 rotations, 256-row MMAs) or
  // single CTAs (128 x 128).  The single-CTA kernel, in its default order,
  // is timed on the same windows in its own tile units (twice the tiles,
  // the same (pattern, rotation) work); it replaces the pairs when 2 %
  // faster.  The shapes' results differ only by the FP32 rounding of the
  // accumulation (1e-6 relative).
  if (pair) {
    p->estep_pair = 0;
    const int s_total = (p->Np / 128) * n_rt;
    const int s_count = std::min(s_total, 2 * count);
    float ts = 0.0f;
    for (int first : firsts) {
      float ms = 0.0f;
      if ((rc = tc_time_estep(p, 8, std::min(2 * first, s_total - s_count), s_count, &ms))) break;
      ts = std::max(ts, ms);
    }
    if (!rc && ts < 0.98f * raster_ms) {
      raster = 8;
      raster_ms = ts;
    } else {
      p->estep_pair = 1;
    }
    if (rc) return rc;
  }
  p->estep_raster = raster;
  if (best) *best = raster;
  if (best_ms) *best_ms = raster_ms;
  return EMC_OK;
}


int tc_mstep(emc_plan* p, float* model, float* weight) {
  emc_ctx* ctx = p->ctx;
  TcState* st = state(p);
  TcMstepArgs a;
  a.R = p->d.n_rot;
  a.Kp = p->Kp;
  a.Np = p->Np;
  a.P_eff = p->P_eff;
  a.n_qt = p->Kp / ms::BN + (p->Kp % ms::BN ? 1 : 0);
  a.n_rt = p->Rp / ms::BM;
  a.nkb = p->Np / ms::BK;
  a.raster = p->mstep_raster;
  a.T = p->T;
  a.qscale = p->qscale;
  a.k_inv = 1.0f / p->count_scale;
  a.rot = p->rot;
  a.cx = p->cx;
  a.cy = p->cy;
  a.cz = p->cz;
  a.side = p->d.side;
  a.interp = p->d.interp;
  a.deterministic = p->d.insert_mode == EMC_INSERT_DETERMINISTIC;
  a.model = model;
  a.weight = weight;
  a.fix2 = p->fix2;
  a.acc2 = p->acc2;
  a.q_lo = p->mstep_q_lo;
  a.aggregate = p->mstep_aggregate;
  a.ms_list = p->ms_list;
  a.ms_n = p->ms_n;
  a.ms_map = p->ms_map;
  a.kb_off = p->prune_kb_off;
  a.kb_list = p->prune_kb_list;
  a.fix_scale = reinterpret_cast<const float2*>(p->red + kRedFixScale);
  a.u = p->d.insert_mode == EMC_INSERT_SORTED ? p->ins_u : nullptr;
  a.ldu = p->ins_ldu;
  a.status = st->status;
  a.spin = p->debug_spin ? p->debug_spin : ptx::kSpinLimit;
  a.n_tiles = a.n_qt * a.n_rt;
  // pruned: the pair's two rotation tiles have one list in true-Poisson plans, whose
  // masks span 256 rotations (prune_finish)
  const bool one_list = !a.kb_off || p->d.diff == EMC_DIFF_TRUE_POISSON;
  if (p->mstep_pair && one_list && a.n_rt > 1 && ctx->sm_count >= 2) {
    // CTA pairs, persistent: one cluster per two SMs
    const int tiles = ((a.n_rt + 1) / 2) * a.n_qt;
    const int clusters = std::min(tiles, ctx->sm_count / 2);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * clusters);
    cfg.blockDim = dim3(ms::THREADS);
    cfg.dynamicSmemBytes = a.q_lo ? ms2::Ring<1>::kSmem : ms2::Ring<0>::kSmem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e =
        a.q_lo ? cudaLaunchKernelEx(&cfg, tc_mstep_pair_kernel<1>, st->mQh, st->mQl, st->mKt128, a)
               : cudaLaunchKernelEx(&cfg, tc_mstep_pair_kernel<0>, st->mQh, st->mQl, st->mKt128, a);
    if (e == cudaSuccess) return after_launch(ctx, "tc_mstep_pair_kernel");
    // a refused launch configuration is not a sticky error: single CTAs from now on
    (void)cudaGetLastError();
    p->mstep_pair = 0;
  }
  const int grid = std::min(a.n_tiles, ctx->sm_count);
  if (a.q_lo)
    tc_mstep_kernel<1><<<grid, ms::THREADS, MsRing<1>::kSmem, ctx->stream>>>(st->mQh, st->mQl,
                                                                              st->mKt, a);
  else
    tc_mstep_kernel<0><<<grid, ms::THREADS, MsRing<0>::kSmem, ctx->stream>>>(st->mQh, st->mQl,
                                                                              st->mKt, a);
  return after_launch(ctx, "tc_mstep_kernel");
}

void tc_free(emc_plan* p) {
  delete state(p);
  p->tc = nullptr;
}

// ------------------------------------------------------- self-test -------
// One CTA computes D[128 x BN] = A[128 x K] B[BN x K]^T with the same TMA,
// shared-memory descriptor, MMA and TMEM-load code as the iteration kernels,
// in their two operand layouts: (BN = 128) 64B swizzle with 32-wide k-blocks, as the
// true-Poisson likelihood's single CTAs load, and (BN = 256) 128B swizzle with 64-wide
// k-blocks, as all others do.  Single-stage pipeline.
template <int BN, int BK>
__global__ void __launch_bounds__(128, 1)
    tc_gemm_selftest_kernel(const __grid_constant__ CUtensorMap mA,
                            const __grid_constant__ CUtensorMap mB, int K, float* D, int* status) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int A_BYTES = 128 * BK * 2, B_BYTES = BN * BK * 2;
  constexpr uint32_t SW = BK == 64 ? 2 : 4;
  constexpr uint32_t SBO = BK * 2 * 8;
  uint64_t* full = (uint64_t*)(smem + A_BYTES + B_BYTES);
  uint64_t* done = full + 1;
  uint32_t* tslot = (uint32_t*)(done + 1);
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    ptx::mbar_init(full, 1);
    ptx::mbar_init(done, 1);
    ptx::fence_mbar_init();
  }
  if (warp == 0) {
    ptx::tmem_alloc(tslot, BN);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tslot;
  bool ok = true;
  for (int kb = 0; kb < K / BK && ok; ++kb) {
    if (threadIdx.x == 0) {
      ptx::mbar_arrive_expect_tx(full, A_BYTES + B_BYTES);
      ptx::tma_load_2d(smem, &mA, kb * BK, 0, full);
      ptx::tma_load_2d(smem + A_BYTES, &mB, kb * BK, 0, full);
    }
    ok = ptx::mbar_wait(full, kb & 1, status, 0);
    ptx::tc_fence_after();
    if (threadIdx.x == 0 && ok) {
      const uint32_t base = ptx::smem_u32(smem);
      for (int ks = 0; ks < BK / 16; ++ks)
        ptx::mma_f16(tmem, ptx::smem_desc(base + ks * 32, SBO, SW),
                     ptx::smem_desc(base + A_BYTES + ks * 32, SBO, SW), ptx::idesc_f16(128, BN),
                     (kb | ks) ? 1u : 0u);
      ptx::mma_commit(done);
    }
    if (ok) ok = ptx::mbar_wait(done, kb & 1, status, 1);
    ptx::tc_fence_after();
    __syncthreads();
  }
  if (ok) {
    const int q = warp & 3;
    const uint32_t la = tmem + ((uint32_t)(q * 32) << 16);
    const int row = q * 32 + (threadIdx.x & 31);
    for (int c0 = 0; c0 < BN; c0 += 16) {
      float v[16];
      ptx::tmem_ld16(la + c0, v);
      ptx::tmem_wait_ld();
      for (int j = 0; j < 16; ++j) D[(size_t)row * BN + c0 + j] = v[j];
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, BN);
  }
}

}  // namespace emc

// Diagnostic: D[128 x n] = A[128 x k] B[n x k]^T (FP16 in, FP32 out, device
// pointers) through the tcgen05 building blocks; n = 128 uses 64B-swizzled 32-wide
// k-blocks, n = 256 128B-swizzled 64-wide ones.  k must be a multiple of the k-block.
extern "C" int emc_tc_gemm_selftest(emc_ctx* ctx, const void* d_a, const void* d_b, float* d_d,
                                    int n, int k) {
  using namespace emc;
  EMC_CHECK_CTX(ctx);
  EMC_REQUIRE(ctx, d_a && d_b && d_d, "tc_gemm_selftest: null pointer");
  EMC_REQUIRE(ctx, n == 128 || n == 256, "tc_gemm_selftest: n must be 128 or 256");
  const int bk = n == 128 ? 32 : 64;
  EMC_REQUIRE(ctx, k > 0 && k % bk == 0, "tc_gemm_selftest: k %% %d != 0", bk);
  CUtensorMap mA, mB;
  int rc = make_map(ctx, &mA, d_a, 128, k, 128, bk);
  if (!rc) rc = make_map(ctx, &mB, d_b, n, k, n, bk);
  if (rc) return rc;
  int* status = nullptr;
  EMC_CUDA(ctx, cudaMallocAsync((void**)&status, sizeof(int), ctx->stream));
  EMC_CUDA(ctx, cudaMemsetAsync(status, 0, sizeof(int), ctx->stream));
  const int smem = 128 * bk * 2 + n * bk * 2 + 1024 + 1024;
  if (n == 128) {
    EMC_CUDA(ctx, cudaFuncSetAttribute(tc_gemm_selftest_kernel<128, 32>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    tc_gemm_selftest_kernel<128, 32><<<1, 128, smem, ctx->stream>>>(mA, mB, k, d_d, status);
  } else {
    EMC_CUDA(ctx, cudaFuncSetAttribute(tc_gemm_selftest_kernel<256, 64>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    tc_gemm_selftest_kernel<256, 64><<<1, 128, smem, ctx->stream>>>(mA, mB, k, d_d, status);
  }
  if ((rc = after_launch(ctx, "tc_gemm_selftest_kernel"))) return rc;
  int h = 0;
  EMC_CUDA(ctx, cudaMemcpyAsync(&h, status, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  EMC_CUDA(ctx, cudaFreeAsync(status, ctx->stream));
  EMC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (h) return fail(ctx, EMC_ERR_TIMEOUT, "tc_gemm_selftest: wait timed out (0x%x)", h);
  return EMC_OK;
}
