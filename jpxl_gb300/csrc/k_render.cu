// k_render.cu — sm_103a kernels of the plan renderer / decoder tail:
//   R1 k_render8<kind>, k_render_rect<R,C>, k_render_64<R,C>
//                        dequantize, HF CfL, LLF from the LF planes, IDCT_2D,
//                        in-frame scatter and the per-block EPF sigma
//   R2 k_gaborish        J.3 3x3 with FMA, mirrored borders
//   R3 k_epf<step>       J.4 steps 0/1/2
//   R4 k_colour_out      L.2.2 opsin inverse and the output encoding
// Operation order follows jpxl-plan-render lib.rs:749 render_inner and the
// jpxl-core kernels it calls; -fmad=false keeps every unfused product.
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "jpxlg_common.cuh"
#include "jpxlg_internal.h"
#include "jpxlg_kernels.h"

namespace jpxlg {

extern __constant__ float c_scale_f[32];
extern __constant__ float c_quant_bias[3];

__constant__ float c_opsin_m[9];
__constant__ float c_opsin_bias[3];
__constant__ float c_opsin_bias_cbrt[3];
// dct.rs:631 the 64-point DCT-II matrix (rows u, columns x), f32 entries.
__device__ __align__(16) float g_dct64[64 * 64];

// dct.rs:678 matrix_pass for N = 64 (the reference's transforms above 32
// points): each output an f64 dot product of f32 entries, rounded once, then
// the normative factor sqrt(64) = 8.  The dot product runs in double-float on
// the FP32 pipe (GB300's FP64 rate is a small fraction of its FP32 rate):
// each product is exact as p + e (e from one FMA) and a compensated sum
// carries the rest, rounded to f32 once at the end.  Both that sum and the
// reference's sequential f64 sum lie within ~1e-15 (relative) of the exact
// dot product, so they round to the same f32 unless the exact value lies
// that close to a rounding midpoint.
//
// The matrix's f32 entries are exactly symmetric, M[u][63 - x] = +-M[u][x]
// by u's parity, and so are its even rows again over half the columns, and
// so on: the sum falls apart by levels as idct_share's does, odd multiples of
// 2^t at level t, which leaves 1366 products of 4096 per column.
__device__ __forceinline__ void df_acc(float& hi, float& lo, float a, float b) {
  const float p = a * b;
  const float e = __fmaf_rn(a, b, -p);  // a*b = p + e exactly
  const float s = hi + p;
  const float bb = s - hi;
  const float err = (hi - (s - bb)) + (p - bb);  // hi + p = s + err exactly
  hi = s;
  lo = lo + (err + e);
}
__device__ __forceinline__ float2 df_sum(float2 a, float2 b) {
  const float s = a.x + b.x;
  const float bb = s - a.x;
  const float err = (a.x - (s - bb)) + (b.x - bb);
  return make_float2(s, a.y + (err + b.y));
}
__device__ __forceinline__ float2 df_neg(float2 a) { return make_float2(-a.x, -a.y); }

// Share `g` < 16 of a column's 64-point inverse: put(row, double-float) in
// idct_share's rows; rows 62 and 63 hold the products of inputs 32 and 0.
template <typename Get, typename Put>
__device__ __forceinline__ void idct64_share(int g, Get get, Put put) {
  if (g < 15) {
    // level t: 64 >> (t + 1) outputs, four per share, of as many terms
    const int t = g < 8 ? 0 : (g < 12 ? 1 : (g < 14 ? 2 : 3));
    const int k = 4 * (g < 8 ? g : (g < 12 ? g - 8 : (g < 14 ? g - 12 : 0)));
    const int terms = 32 >> t;
    float h[4] = {0.0f, 0.0f, 0.0f, 0.0f}, l[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
    for (int m = 0; m < terms; ++m) {
      const int u = (2 * m + 1) << t;
      const float4 row = __ldg(reinterpret_cast<const float4*>(g_dct64 + u * 64 + k));
      const float x = get(u);
      df_acc(h[0], l[0], row.x, x);
      df_acc(h[1], l[1], row.y, x);
      df_acc(h[2], l[2], row.z, x);
      df_acc(h[3], l[3], row.w, x);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) put(64 - (64 >> t) + k + i, make_float2(h[i], l[i]));
    return;
  }
  // level 4 (inputs 16 and 48, two outputs) and the last two products
  const float x16 = get(16), x48 = get(48), x32 = get(32), x0 = get(0);
  float2 o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    df_acc(o[i].x, o[i].y, g_dct64[16 * 64 + i], x16);
    df_acc(o[i].x, o[i].y, g_dct64[48 * 64 + i], x48);
  }
  df_acc(o[2].x, o[2].y, g_dct64[32 * 64], x32);
  df_acc(o[3].x, o[3].y, g_dct64[0], x0);
#pragma unroll
  for (int i = 0; i < 4; ++i) put(60 + i, o[i]);
}

// Outputs k and 63 - k (k < 32) from the rows of idct64_share.
template <typename Get>
__device__ __forceinline__ void idct64_pair(int k, Get get, float* lo, float* hi) {
  int at[6];
  at[0] = k;
#pragma unroll
  for (int t = 1; t < 6; ++t) {
    const int m = 64 >> (t + 1);
    at[t] = at[t - 1] < m ? at[t - 1] : 2 * m - 1 - at[t - 1];
  }
  float2 even = get(63);
#pragma unroll
  for (int t = 5; t >= 1; --t) {
    const float2 odd = get(64 - (64 >> t) + at[t]);
    even = df_sum(even, at[t - 1] < (64 >> (t + 1)) ? odd : df_neg(odd));
  }
  const float2 odd = get(at[0]);
  const float2 a = df_sum(even, odd), b = df_sum(even, df_neg(odd));
  // one correct rounding of the double-float sum, then the factor 8
  *lo = (a.x + a.y) * 8.0f;
  *hi = (b.x + b.y) * 8.0f;
}

// jpxl-core dct.rs:982 idct_2d_in_place for the small shapes of the 8x8
// special transforms: coef is landscape (min x max), out ROWS x COLS samples.
template <int ROWS, int COLS>
__device__ __forceinline__ void idct2d_raw(const float* coef, float* out) {
  float s[ROWS * COLS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int c = 0; c < COLS; ++c)
      s[c * ROWS + r] = COLS > ROWS ? coef[r * COLS + c] : coef[c * ROWS + r];
#pragma unroll
  for (int k = 0; k < ROWS; ++k) {
    float v[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) v[i] = s[i * ROWS + k];
    idct_1d<COLS>(v);
#pragma unroll
    for (int i = 0; i < COLS; ++i) s[i * ROWS + k] = v[i];
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int c = 0; c < COLS; ++c) out[r * COLS + c] = s[c * ROWS + r];
#pragma unroll
  for (int c = 0; c < COLS; ++c) {
    float v[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) v[i] = out[i * COLS + c];
    idct_1d<ROWS>(v);
#pragma unroll
    for (int i = 0; i < ROWS; ++i) out[i * COLS + c] = v[i];
  }
}

__device__ double g_afv[256];  // Table I.11, uploaded by the host

// varblock.rs:917 DCT2x2: aux_idct_2x2 (:898) with s = 2, 4, 8, each stage
// reading the previous one; b (row-major, LLF at 0) becomes the samples.
__device__ __forceinline__ void dct2x2_block(float* b) {
  float r[64];
#pragma unroll
  for (int st = 2; st <= 8; st *= 2) {
    const int h = st / 2;
#pragma unroll
    for (int i = 0; i < 64; ++i) r[i] = b[i];
#pragma unroll
    for (int y = 0; y < h; ++y)
#pragma unroll
      for (int x = 0; x < h; ++x) {
        const float c00 = b[y * 8 + x], c01 = b[y * 8 + h + x];
        const float c10 = b[(y + h) * 8 + x], c11 = b[(y + h) * 8 + h + x];
        r[(2 * y) * 8 + 2 * x] = ((c00 + c01) + c10) + c11;
        r[(2 * y) * 8 + 2 * x + 1] = ((c00 + c01) - c10) - c11;
        r[(2 * y + 1) * 8 + 2 * x] = ((c00 - c01) + c10) - c11;
        r[(2 * y + 1) * 8 + 2 * x + 1] = ((c00 - c01) - c10) + c11;
      }
#pragma unroll
    for (int i = 0; i < 64; ++i) b[i] = r[i];
  }
}


// The 8x8 special transforms of jpxl-core varblock.rs:926-1230 on a
// dequantized block b (row-major, LLF at 0): KIND 2 Hornuss, 3 DCT4x4,
// 4 DCT8x4, 5 DCT4x8, 6..9 AFV0..AFV3.  Evaluation order follows the
// reference expression by expression.
template <int KIND>
__device__ __forceinline__ void special_block(const float* b, float* o) {
  auto at = [&](int x, int y) { return b[y * 8 + x]; };
  auto set = [&](int x, int y, float v) { o[y * 8 + x] = v; };
  if constexpr (KIND == 2 || KIND == 3) {
    const float c00 = b[0], c01 = b[1], c10 = b[8], c11 = b[9];
    const float dcs[4] = {((c00 + c01) + c10) + c11, ((c00 + c01) - c10) - c11,
                          ((c00 - c01) + c10) - c11, ((c00 - c01) - c10) + c11};
#pragma unroll
    for (int y = 0; y < 2; ++y)
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        if constexpr (KIND == 2) {
          float rs = 0.0f;
#pragma unroll
          for (int iy = 0; iy < 4; ++iy)
#pragma unroll
            for (int ix = (iy == 0 ? 1 : 0); ix < 4; ++ix) rs += at(x + ix * 2, y + iy * 2);
          const float centre = dcs[y * 2 + x] - rs / 16.0f;
          set(4 * x + 1, 4 * y + 1, centre);
#pragma unroll
          for (int iy = 0; iy < 4; ++iy)
#pragma unroll
            for (int ix = 0; ix < 4; ++ix)
              if (!(ix == 1 && iy == 1)) set(x * 4 + ix, y * 4 + iy, at(x + ix * 2, y + iy * 2) + centre);
          set(4 * x, 4 * y, at(x + 2, y + 2) + centre);
        } else {
          float blk[16], smp[16];
#pragma unroll
          for (int iy = 0; iy < 4; ++iy)
#pragma unroll
            for (int ix = 0; ix < 4; ++ix) blk[iy * 4 + ix] = at(x + ix * 2, y + iy * 2);
          blk[0] = dcs[y * 2 + x];
          idct2d_raw<4, 4>(blk, smp);
#pragma unroll
          for (int l = 0; l < 4; ++l)
#pragma unroll
            for (int k = 0; k < 4; ++k) set(4 * x + k, 4 * y + l, smp[l * 4 + k]);
        }
      }
  } else if constexpr (KIND == 4 || KIND == 5) {
    const float coef0 = at(0, 0), coef1 = at(0, 1);
    const float dcs[2] = {coef0 + coef1, coef0 - coef1};
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float g[32], smp[32];
#pragma unroll
      for (int iy = 0; iy < 4; ++iy)
#pragma unroll
        for (int ix = 0; ix < 8; ++ix) g[iy * 8 + ix] = at(ix, half + iy * 2);
      g[0] = dcs[half];
      if constexpr (KIND == 4) {
        idct2d_raw<8, 4>(g, smp);
#pragma unroll
        for (int iy = 0; iy < 8; ++iy)
#pragma unroll
          for (int ix = 0; ix < 4; ++ix) set(4 * half + ix, iy, smp[iy * 4 + ix]);
      } else {
        idct2d_raw<4, 8>(g, smp);
#pragma unroll
        for (int iy = 0; iy < 4; ++iy)
#pragma unroll
          for (int ix = 0; ix < 8; ++ix) set(ix, 4 * half + iy, smp[iy * 8 + ix]);
      }
    }
  } else {
    constexpr int n = KIND - 6, fx = n & 1, fy = n / 2;
    float ca[16], sa[16];
    ca[0] = ((at(0, 0) + at(0, 1)) + at(1, 0)) * 4.0f;
#pragma unroll
    for (int iy = 0; iy < 4; ++iy)
#pragma unroll
      for (int ix = (iy == 0 ? 1 : 0); ix < 4; ++ix) ca[iy * 4 + ix] = at(ix * 2, iy * 2);
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      double acc = 0.0;
#pragma unroll
      for (int j = 0; j < 16; ++j) acc += (double)ca[j] * g_afv[j * 16 + q];
      sa[q] = (float)acc;
    }
#pragma unroll
    for (int iy = 0; iy < 4; ++iy)
#pragma unroll
      for (int ix = 0; ix < 4; ++ix) {
        const int sx = fx ? 3 - ix : ix, sy = fy ? 3 - iy : iy;
        set(fx * 4 + ix, fy * 4 + iy, sa[sy * 4 + sx]);
      }
    float c44[16], s44[16];
#pragma unroll
    for (int iy = 0; iy < 4; ++iy)
#pragma unroll
      for (int ix = 0; ix < 4; ++ix) c44[iy * 4 + ix] = at(ix * 2 + 1, iy * 2);
    c44[0] = (at(0, 0) - at(1, 0)) + at(0, 1);
    idct2d_raw<4, 4>(c44, s44);
#pragma unroll
    for (int iy = 0; iy < 4; ++iy)
#pragma unroll
      for (int ix = 0; ix < 4; ++ix) set((fx ? 0 : 4) + ix, fy * 4 + iy, s44[iy * 4 + ix]);
    float c48[32], s48[32];
#pragma unroll
    for (int iy = 0; iy < 4; ++iy)
#pragma unroll
      for (int ix = 0; ix < 8; ++ix) c48[iy * 8 + ix] = at(ix, 1 + iy * 2);
    c48[0] = at(0, 0) - at(0, 1);
    idct2d_raw<4, 8>(c48, s48);
#pragma unroll
    for (int iy = 0; iy < 4; ++iy)
#pragma unroll
      for (int ix = 0; ix < 8; ++ix) set(ix, (fy ? 0 : 4) + iy, s48[iy * 8 + ix]);
  }
}

// ---------------------------------------------------------------------------
// R1, 8 x 8 — eight lanes per block, four blocks per warp, the three channels
// together: all of a block's loads are in flight at once, its two passes
// meet in shared memory within one warp, and no barrier of the block is
// needed.  KIND 0 is DCT8; KIND 1 (DCT2x2) and 2 .. 9 (special_block) run in
// the block's first three lanes, one channel each (a 128 x 128 stream's:
// 22.5 us with the channels in turn, now 15).  Bound by the reads of the coefficients and the writes of the
// samples (24 bytes per sample of three channels).
// ---------------------------------------------------------------------------

template <int KIND>
__global__ void __launch_bounds__(128) k_render8(RenderArgs a, const uint32_t* __restrict__ list,
                                                 int count) {
  __shared__ float T[16][3][8][9];
  // compact dequant slot of this transform
  constexpr int slot = KIND == 0 ? 0 : KIND == 1 ? 6 : KIND == 2 ? 9 : KIND == 3 ? 10
                       : KIND <= 5 ? 11 : 12;
  const int g = threadIdx.x / 8, j = threadIdx.x % 8;
  const int vi = blockIdx.x * 16 + g;
  const bool active = vi < count;
  const uint32_t packed = list[active ? vi : count - 1];  // idle lanes repeat the last block
  const int bx = packed & 0xffff, by = packed >> 16;
  const int x0 = bx * 8, y0 = by * 8;
  const Geo& geo = a.geo;
  const size_t cplane = (size_t)geo.W8 * geo.H8;
  const size_t bplane = (size_t)geo.bw * geo.bh;
  const size_t plane = (size_t)geo.w * geo.h;
  const size_t bi = (size_t)by * geo.bw + bx;
  int32_t q[3][8];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int y = 0; y < 8; ++y)
      q[c][y] = a.qcoeff[cplane * c + (size_t)(y0 + y) * geo.W8 + x0 + j];
  const float mul = hf_multiplier(a.mul_table, a.qs.global_scale, a.hf_mul[bi]);  // reconstruct.rs:27
  const int tile = (by / 8) * geo.tw + bx / 8;
  const float kx = 0.0f + (float)a.cfl_x[tile] / 84.0f;  // reconstruct.rs:96 cfl_factors
  const float kb = 1.0f + (float)a.cfl_b[tile] / 84.0f;
  // Dequantize column j (plan-render lib.rs:913: adjusted * (mul*qm) *
  // matrix, left to right; lib.rs:1344 apply_hf_cfl).
  float v[3][8];
  const int off = dq_offset(slot);
#pragma unroll
  for (int ci = 0; ci < 3; ++ci) {
    const int c = ci == 0 ? 1 : (ci == 1 ? 0 : 2);  // luma first: CfL needs it
    const float scale = mul * a.qs.qm[c], bias = c_quant_bias[c];
    const float* m = a.dq + c * kDequantTableFloats + off + j;
#pragma unroll
    for (int y = 0; y < 8; ++y) {
      const float d = bias_adjust_q(q[c][y], bias) * scale * __ldg(&m[y * 8]);
      v[c][y] = c == 1 ? d : d + (c == 0 ? kx : kb) * v[1][y];
    }
  }
  // The LLF sample (varblock.rs:817 llf_from_lf): LF dequantized
  // (reconstruct.rs:84) with the LF CfL (plan-render lib.rs:1314), times
  // scale_f(0) twice.
  if (j == 0) {
    float d[3];
    if (a.lf_float) {
#pragma unroll
      for (int c = 0; c < 3; ++c) d[c] = a.lf_float[bplane * c + bi];
    } else {
      float k_x_lf = a.k_x_lf, k_b_lf = a.k_b_lf;
      if (a.lf_factors_dev) {
        k_x_lf = 0.0f + (float)a.lf_factors_dev[0] / 84.0f;
        k_b_lf = 1.0f + (float)a.lf_factors_dev[1] / 84.0f;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) d[c] = a.qs.m_dc[c] * (float)a.lfq[bplane * c + bi] / 1.0f;
      d[0] = d[0] + k_x_lf * d[1];
      d[2] = d[2] + k_b_lf * d[1];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c][0] = d[c] * c_scale_f[0] * c_scale_f[0];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if constexpr (KIND == 0) idct_1d<8>(v[c]);
#pragma unroll
    for (int i = 0; i < 8; ++i) T[g][c][i][j] = v[c][i];
  }
  __syncwarp();
  if constexpr (KIND != 0) {
    if (j < 3) {
      float b[64], o[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) b[i] = T[g][j][i / 8][i % 8];
      if constexpr (KIND == 1) {
        dct2x2_block(b);
#pragma unroll
        for (int i = 0; i < 64; ++i) o[i] = b[i];
      } else {
        special_block<KIND>(b, o);
      }
#pragma unroll
      for (int i = 0; i < 64; ++i) T[g][j][i / 8][i % 8] = o[i];
    }
    __syncwarp();
  }
  const int fx = x0 + j;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[c][i] = KIND == 0 ? T[g][c][j][i] : T[g][c][i][j];
    if constexpr (KIND == 0) idct_1d<8>(v[c]);
    if (active && fx < geo.w) {
      float* p = a.planes + plane * c + (size_t)y0 * geo.w + fx;
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (y0 + r < geo.h) p[(size_t)r * geo.w] = v[c][r];
    }
  }
  // J.4.3 sigma (restoration.rs:338 vardct_sigma).
  if (active && j == 0) {
    int s = a.sharpness[bi];
    s = s > 7 ? 7 : s;
    const float lut = s == 7 ? 1.0f : (float)s / 7.0f;
    a.sigma[bi] = mul * 0.46f * lut;
  }
}

// ---------------------------------------------------------------------------
// R1, R x C with a side of 16 or 32 — one varblock by R C / 4 threads.
// Landscape coefficients L are crows = min x ccols = max.  IDCT_2D
// (dct.rs:982): scratch S (C x R) is L transposed when C > R, else L; step A
// runs length-C IDCTs down S's R columns; step B runs length-R IDCTs along
// the C rows of the result, producing sample column i from row i.
//
// A transform of 16 or 32 points in one thread is a chain of several hundred
// instructions behind a 254-register frame, and a frame has few such blocks:
// the kernel was as long as one block (1920x1080 of mixed squares: 80 us, now
// 34 with the 8x8 class beside it; 64x64: 24, now 17).  Here a warp takes a
// share of 32 columns (idct_share's split; as many blocks side by side as 32
// columns need) and all three channels pass through each phase together, so
// that between two barriers a warp has a hundred or two independent
// instructions per channel.  The shares are dealt so that the long ones (the
// odd half of the first level) spread over the warps.  Bound by the barriers'
// and the dependent loads' latency at a few blocks, by the FP32 pipe at many.
// Rows one float longer than the matrix keep the column and the row reads
// free of bank conflicts.
// ---------------------------------------------------------------------------

template <int R, int C>
struct RectShape {
  static constexpr int CR = R < C ? R : C, CC = R < C ? C : R;  // landscape rows, columns
  static constexpr bool portrait = R > C;
  static constexpr int BR = R / 8, BC = C / 8;
  static constexpr int LY = CR / 8, LX = CC / 8;  // LLF corner
  // compact dequant slot
  static constexpr int slot = CC == 64 ? (CR == 64 ? 7 : 8)
                              : R == C ? (R == 16 ? 1 : 2)
                                       : (CC == 16 ? 3 : (CR == 8 ? 4 : 5));
  // rows of c_scale_f
  static constexpr int SY = LY == 1 ? 0 : (LY == 2 ? 1 : (LY == 4 ? 2 : 3));
  static constexpr int SX = LX == 1 ? 0 : (LX == 2 ? 1 : (LX == 4 ? 2 : 3));
};

// An LF sample of channel c at block bi: as it stands in a decoded frame's LF
// image, else dequantized (reconstruct.rs:84) with the LF CfL (plan-render
// lib.rs:1314).
__device__ __forceinline__ float lf_sample(const RenderArgs& a, size_t bplane, int c, size_t bi) {
  if (a.lf_float) return a.lf_float[bplane * c + bi];
  const float dY = a.qs.m_dc[1] * (float)a.lfq[bplane + bi] / 1.0f;
  if (c == 1) return dY;
  float k = c == 0 ? a.k_x_lf : a.k_b_lf;
  if (a.lf_factors_dev)
    k = (c == 0 ? 0.0f : 1.0f) + (float)a.lf_factors_dev[c == 0 ? 0 : 1] / 84.0f;
  const float d = a.qs.m_dc[c] * (float)a.lfq[bplane * c + bi] / 1.0f;
  return d + k * dY;
}

// J.4.3 sigma of a block (restoration.rs:338 vardct_sigma).
__device__ __forceinline__ float block_sigma(const RenderArgs& a, float mul, size_t bi) {
  int s = a.sharpness[bi];
  s = s > 7 ? 7 : s;
  const float lut = s == 7 ? 1.0f : (float)s / 7.0f;
  return mul * 0.46f * lut;
}

// The LLF corner (varblock.rs:817 llf_from_lf) of one channel from its LF
// rectangle `rect` (landscape LY x LX): DCT_2D, times scale_f(y) *
// scale_f(x), by LX lanes and then LY lanes of one warp; put(y, x, value).
template <typename S, typename Put>
__device__ __forceinline__ void llf_corner(float* rect, int k, bool on, Put put) {
  constexpr int LY = S::LY, LX = S::LX;
  const float* sfy = &c_scale_f[S::SY * 8];
  const float* sfx = &c_scale_f[S::SX * 8];
  if (on && k < LX) {
    float v[LY];
#pragma unroll
    for (int r = 0; r < LY; ++r) v[r] = rect[r * LX + k];
    if constexpr (LY > 1) dct_1d<LY>(v);
#pragma unroll
    for (int r = 0; r < LY; ++r) rect[r * LX + k] = v[r];
  }
  __syncwarp();
  if (on && k < LY) {
    float v[LX];
#pragma unroll
    for (int r = 0; r < LX; ++r) v[r] = rect[k * LX + r];
    dct_1d<LX>(v);
    // a square's second pass leaves the matrix transposed (dct.rs:956)
#pragma unroll
    for (int r = 0; r < LX; ++r) {
      const int y = LX == LY ? r : k, x = LX == LY ? k : r;
      put(y, x, v[r] * sfy[y] * sfx[x]);
    }
  }
}

template <int R, int C>
__global__ void __launch_bounds__(R* C / 4 * (32 / (R < C ? R : C)))
    k_render_rect(RenderArgs a, const uint32_t* __restrict__ list, int count) {
  using S = RectShape<R, C>;
  constexpr int VPB = 32 / S::CR;                       // blocks per CTA
  constexpr int kWarpsA = VPB * R / 32, kWarpsB = VPB * C / 32;  // column groups of 32
  constexpr int kLlf = S::LY * S::LX;
  __shared__ float A[VPB][3][C][R + 1];
  __shared__ float B[VPB * 3 * (C * (R + 1) > R * (C + 1) ? C * (R + 1) : R * (C + 1))];
  __shared__ float rect[VPB][3][kLlf];
  const int t = threadIdx.x, warp = t / 32, lane = t % 32;
  const Geo& geo = a.geo;
  const size_t cplane = (size_t)geo.W8 * geo.H8;
  const size_t bplane = (size_t)geo.bw * geo.bh;
  const size_t plane = (size_t)geo.w * geo.h;
  const int v0 = blockIdx.x * VPB;
  // an idle place repeats the last block
  auto block = [&](int g) { return list[min(v0 + g, count - 1)]; };
  auto to_s = [](int y, int x, float(&m)[C][R + 1], float d) {
    if constexpr (C > R) m[x][y] = d;
    else m[y][x] = d;
  };
  // The LF rectangles, one thread per sample.
  if (t < VPB * 3 * kLlf) {
    const int g = t / (3 * kLlf), c = t / kLlf % 3, i = t % kLlf;
    const uint32_t pk = block(g);
    const int dy = i / S::BC, dx = i % S::BC;
    const size_t bi = (size_t)((pk >> 16) + dy) * geo.bw + (pk & 0xffff) + dx;
    rect[g][c][S::portrait ? dx * S::BR + dy : i] = lf_sample(a, bplane, c, bi);
  }
  // Dequantize four rows of landscape column x (plan-render lib.rs:913:
  // adjusted * (mul*qm) * matrix, left to right; lib.rs:1344 apply_hf_cfl).
  {
    const int x = t % S::CC, yg = t / S::CC % (S::CR / 4), g = t / (S::CC * S::CR / 4);
    const uint32_t pk = block(g);
    const int bx = pk & 0xffff, by = pk >> 16;
    int32_t q[3][4];
    float m[3][4], dY[4];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int y = 4 * yg + i;
        const size_t pos = S::portrait ? (size_t)(by * 8 + x) * geo.W8 + bx * 8 + y
                                       : (size_t)(by * 8 + y) * geo.W8 + bx * 8 + x;
        q[c][i] = a.qcoeff[cplane * c + pos];
        m[c][i] = __ldg(a.dq + c * kDequantTableFloats + dq_offset(S::slot) + y * S::CC + x);
      }
    const float mul = hf_multiplier(a.mul_table, a.qs.global_scale,
                                    a.hf_mul[(size_t)by * geo.bw + bx]);  // reconstruct.rs:27
    const int tile = (by / 8) * geo.tw + bx / 8;
    const float kx = 0.0f + (float)a.cfl_x[tile] / 84.0f;  // reconstruct.rs:96 cfl_factors
    const float kb = 1.0f + (float)a.cfl_b[tile] / 84.0f;
#pragma unroll
    for (int ci = 0; ci < 3; ++ci) {
      const int c = ci == 0 ? 1 : (ci == 1 ? 0 : 2);  // luma first: CfL needs it
      const float scale = mul * a.qs.qm[c], bias = c_quant_bias[c];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int y = 4 * yg + i;
        float d = bias_adjust_q(q[c][i], bias) * scale * m[c][i];
        if (c == 1) dY[i] = d;
        else d = d + (c == 0 ? kx : kb) * dY[i];
        if (y >= S::LY || x >= S::LX) to_s(y, x, A[g][c], d);
      }
    }
  }
  __syncthreads();
  if (warp == 0) {
    const int g = lane / (3 * S::LX), c = lane / S::LX % 3, k = lane % S::LX;
    static_assert(VPB * 3 * S::LX <= 64);
    llf_corner<S>(rect[min(g, VPB - 1)][c], k, g < VPB,
                  [&](int y, int x, float d) { to_s(y, x, A[g][c], d); });
    if constexpr (VPB * 3 * S::LX > 32) {  // 32 x 8: a second round of lanes
      const int l2 = lane + 32;
      const int g2 = l2 / (3 * S::LX), c2 = l2 / S::LX % 3, k2 = l2 % S::LX;
      __syncwarp();
      llf_corner<S>(rect[min(g2, VPB - 1)][c2], k2, g2 < VPB,
                    [&](int y, int x, float d) { to_s(y, x, A[g2][c2], d); });
    }
  }
  __syncthreads();
  // Step A: length C down R columns.
  const int shA = warp / kWarpsA, qa = (warp % kWarpsA) * 32 + lane, ga = qa / R, ja = qa % R;
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    float* const b = B + (ga * 3 + c) * C * (R + 1) + ja;
    idct_share<C>((shA + 3 * c) % (C / 4), [&](int i) { return A[ga][c][i][ja]; },
                  [&](int r, float v) { b[r * (R + 1)] = v; });
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = shA + h * (C / 4);
      const float* const b = B + (ga * 3 + c) * C * (R + 1) + ja;
      float lo, hi;
      idct_pair<C>(k, [&](int r) { return b[r * (R + 1)]; }, &lo, &hi);
      A[ga][c][k][ja] = lo;
      A[ga][c][C - 1 - k][ja] = hi;
    }
  __syncthreads();
  // Step B: length R along C rows, into sample columns.
  const int shB = warp / kWarpsB, qb = (warp % kWarpsB) * 32 + lane, gb = qb / C, jb = qb % C;
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    float* const b = B + (gb * 3 + c) * R * (C + 1) + jb;
    idct_share<R>((shB + 3 * c) % (R / 4), [&](int i) { return A[gb][c][jb][i]; },
                  [&](int r, float v) { b[r * (C + 1)] = v; });
  }
  __syncthreads();
  {
    const uint32_t pk = block(gb);
    const int fx = (pk & 0xffff) * 8 + jb, y0 = (pk >> 16) * 8;
    if (v0 + gb < count && fx < geo.w) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = shB + h * (R / 4);
          const float* const b = B + (gb * 3 + c) * R * (C + 1) + jb;
          float lo, hi;
          idct_pair<R>(k, [&](int r) { return b[r * (C + 1)]; }, &lo, &hi);
          float* p = a.planes + plane * c + fx;
          if (y0 + k < geo.h) p[(size_t)(y0 + k) * geo.w] = lo;
          if (y0 + R - 1 - k < geo.h) p[(size_t)(y0 + R - 1 - k) * geo.w] = hi;
        }
    }
  }
  if (t < VPB * S::BR * S::BC) {
    const int g = t / (S::BR * S::BC), i = t % (S::BR * S::BC);
    if (v0 + g < count) {
      const uint32_t pk = block(g);
      const size_t b0 = (size_t)(pk >> 16) * geo.bw + (pk & 0xffff);
      const size_t bi = b0 + (size_t)(i / S::BC) * geo.bw + i % S::BC;
      a.sigma[bi] = block_sigma(a, hf_multiplier(a.mul_table, a.qs.global_scale, a.hf_mul[b0]), bi);
    }
  }
}

// ---------------------------------------------------------------------------
// R1 with a side of 64 — one channel of one varblock per CTA of 512 threads
// (a chroma channel dequantizes its luma again for the CfL), the same two
// steps; the 64-point ones in double-float (idct64_share).  A thread's whole
// 64-point column was 41000 dependent-issue operations, six times in a row:
// 375 us however few the blocks; a 64 x 64 block now takes 28 us, a
// 64 x 32 one 17 (185).
// Bound by the FP32 pipe of the SMs that hold its three CTAs.
// ---------------------------------------------------------------------------

template <int R, int C>
struct Rect64Smem {
  float A[C][R + 1];
  float2 B[C * (R + 1) > R * (C + 1) ? C * (R + 1) : R * (C + 1)];
  float rect[RectShape<R, C>::LY * RectShape<R, C>::LX];
};

// One length-N transform of `cols` columns by 16 warps: get(i, column),
// put(k, column, value); B holds N x (cols + 1).
template <int N, int COLS, typename Get, typename Put>
__device__ __forceinline__ void rect64_pass(float2* B, int warp, int lane, Get get, Put put) {
  constexpr int kHalves = COLS / 32, kShares = N / 4, kItems = kHalves * kShares;
  float* const Bf = reinterpret_cast<float*>(B);
#pragma unroll 1
  for (int item = warp; item < kItems; item += 16) {
    // column half by half; the second half's shares start half way round, so
    // that a warp's two shares are a long and a short one
    const int half = item / kShares, j = half * 32 + lane;
    const int sh = (item + half * (kShares / 2)) % kShares;
    if constexpr (N == 64)
      idct64_share(sh, [&](int i) { return get(i, j); },
                   [&](int r, float2 v) { B[r * (COLS + 1) + j] = v; });
    else
      idct_share<N>(sh, [&](int i) { return get(i, j); },
                    [&](int r, float v) { Bf[r * (COLS + 1) + j] = v; });
  }
  __syncthreads();
#pragma unroll 1
  for (int item = warp; item < kHalves * N / 2; item += 16) {
    const int j = item / (N / 2) * 32 + lane, k = item % (N / 2);
    float lo, hi;
    if constexpr (N == 64)
      idct64_pair(k, [&](int r) { return B[r * (COLS + 1) + j]; }, &lo, &hi);
    else
      idct_pair<N>(k, [&](int r) { return Bf[r * (COLS + 1) + j]; }, &lo, &hi);
    put(k, j, lo);
    put(N - 1 - k, j, hi);
  }
}

template <int R, int C>
__global__ void __launch_bounds__(512) k_render_64(RenderArgs a, const uint32_t* __restrict__ list) {
  using S = RectShape<R, C>;
  extern __shared__ __align__(16) unsigned char smem64[];
  auto& sm = *reinterpret_cast<Rect64Smem<R, C>*>(smem64);
  const int t = threadIdx.x, warp = t / 32, lane = t % 32, c = blockIdx.y;
  const uint32_t pk = list[blockIdx.x];
  const int bx = pk & 0xffff, by = pk >> 16, x0 = bx * 8, y0 = by * 8;
  const Geo& geo = a.geo;
  const size_t cplane = (size_t)geo.W8 * geo.H8;
  const size_t bplane = (size_t)geo.bw * geo.bh;
  const size_t plane = (size_t)geo.w * geo.h;
  const size_t b0 = (size_t)by * geo.bw + bx;
  constexpr int kLlf = S::LY * S::LX;
  if (t < kLlf) {
    const int dy = t / S::BC, dx = t % S::BC;
    sm.rect[S::portrait ? dx * S::BR + dy : t] =
        lf_sample(a, bplane, c, b0 + (size_t)dy * geo.bw + dx);
  }
  const float mul = hf_multiplier(a.mul_table, a.qs.global_scale, a.hf_mul[b0]);  // reconstruct.rs:27
  const int tile = (by / 8) * geo.tw + bx / 8;
  const float kc = c == 0 ? 0.0f + (float)a.cfl_x[tile] / 84.0f   // reconstruct.rs:96 cfl_factors
                          : 1.0f + (float)a.cfl_b[tile] / 84.0f;
  auto to_s = [&](int y, int x, float d) {
    if constexpr (C > R) sm.A[x][y] = d;
    else sm.A[y][x] = d;
  };
  auto dequant = [&](int ch, size_t pos, int cell) {
    return bias_adjust_q(a.qcoeff[cplane * ch + pos], c_quant_bias[ch]) * (mul * a.qs.qm[ch]) *
           __ldg(a.dq + ch * kDequantTableFloats + dq_offset(S::slot) + cell);
  };
#pragma unroll 4
  for (int i = t; i < R * C; i += 512) {
    const int y = i / S::CC, x = i % S::CC;
    const size_t pos = S::portrait ? (size_t)(y0 + x) * geo.W8 + x0 + y
                                   : (size_t)(y0 + y) * geo.W8 + x0 + x;
    float d = dequant(c, pos, i);
    if (c != 1) d = d + kc * dequant(1, pos, i);  // lib.rs:1344 apply_hf_cfl
    if (y >= S::LY || x >= S::LX) to_s(y, x, d);
  }
  __syncthreads();
  if (warp == 0) llf_corner<S>(sm.rect, lane, true, to_s);
  __syncthreads();
  rect64_pass<C, R>(sm.B, warp, lane, [&](int i, int j) { return sm.A[i][j]; },
                    [&](int k, int j, float v) { sm.A[k][j] = v; });
  __syncthreads();
  rect64_pass<R, C>(sm.B, warp, lane, [&](int i, int j) { return sm.A[j][i]; },
                    [&](int k, int j, float v) {
                      if (x0 + j < geo.w && y0 + k < geo.h)
                        a.planes[plane * c + (size_t)(y0 + k) * geo.w + x0 + j] = v;
                    });
  if (c == 1 && t < S::BR * S::BC) {
    const size_t bi = b0 + (size_t)(t / S::BC) * geo.bw + t % S::BC;
    a.sigma[bi] = block_sigma(a, mul, bi);
  }
}

// The LLF rectangles and EPF sigma of the square varblocks of size N that
// the split-precision render (k_tc.cu) transforms, exactly as k_render_rect
// forms them: one thread per LF sample, then one per column and per row of a
// rectangle (one thread per rectangle took 8.5 us for ten tiles of 32 x 32,
// 5.2 so: the loads' latency once instead of sixteen blocks' sigma in
// turn).  llf receives 16 floats per channel per varblock.
constexpr int kLlfThreads = 128;
template <int N>
__global__ void __launch_bounds__(kLlfThreads) k_llf_sigma(RenderArgs a,
                                                           const uint32_t* __restrict__ list,
                                                           int count, float* __restrict__ llf) {
  using S = RectShape<N, N>;
  constexpr int n = N / 8, kPer = 3 * n * n, kBlocks = kLlfThreads / kPer;
  __shared__ float rect[kBlocks][3][n * n];
  const Geo& geo = a.geo;
  const size_t bplane = (size_t)geo.bw * geo.bh;
  const int t = threadIdx.x, v0 = blockIdx.x * kBlocks;
  const float* sf = &c_scale_f[S::SX * 8];
  {
    const int g = t / kPer, c = t / (n * n) % 3, i = t % (n * n);
    if (g < kBlocks && v0 + g < count) {
      const uint32_t pk = list[v0 + g];
      const size_t b0 = (size_t)(pk >> 16) * geo.bw + (pk & 0xffff);
      const size_t bi = b0 + (size_t)(i / n) * geo.bw + i % n;
      rect[g][c][i] = lf_sample(a, bplane, c, bi);
      if (c == 0)
        a.sigma[bi] = block_sigma(a, hf_multiplier(a.mul_table, a.qs.global_scale, a.hf_mul[b0]), bi);
    }
  }
  __syncthreads();
  const int g = t / (3 * n), c = t / n % 3, k = t % n;
  const bool on = g < kBlocks && v0 + g < count;
  float v[n];
  if constexpr (n > 1) {
    if (on) {
#pragma unroll
      for (int r = 0; r < n; ++r) v[r] = rect[g][c][r * n + k];
      dct_1d<n>(v);
#pragma unroll
      for (int r = 0; r < n; ++r) rect[g][c][r * n + k] = v[r];
    }
    __syncthreads();
  }
  if (!on) return;
#pragma unroll
  for (int r = 0; r < n; ++r) v[r] = rect[g][c][k * n + r];
  if constexpr (n > 1) dct_1d<n>(v);
  // the second pass leaves the matrix transposed (dct.rs:956)
  float* o = llf + (size_t)(v0 + g) * 48 + c * 16;
#pragma unroll
  for (int r = 0; r < n; ++r) o[r * n + k] = v[r] * sf[r] * sf[k];
}

int launch_llf_sigma(const RenderArgs& a, const uint32_t* const* lists, const int* counts,
                     float* const* llf, const cudaStream_t* s) {
  int k = 0;
  auto go = [&](auto kernel, int i, int blocks) {
    if (!counts[i]) return;
    kernel<<<(counts[i] + blocks - 1) / blocks, kLlfThreads, 0, s[i]>>>(a, lists[i], counts[i],
                                                                       llf[i]);
    ++k;
  };
  go(k_llf_sigma<8>, 0, kLlfThreads / 3);
  go(k_llf_sigma<16>, 1, kLlfThreads / 12);
  go(k_llf_sigma<32>, 2, kLlfThreads / 48);
  return k;
}

void launch_render_varblocks(const RenderArgs& a, const uint32_t* const* lists, const int* counts,
                             const cudaStream_t* s) {
  auto n8 = [&](int i) { return (counts[i] + 15) / 16; };
#define JPXLG_R8(IDX, KIND) \
  if (counts[IDX]) k_render8<KIND><<<n8(IDX), 128, 0, s[IDX]>>>(a, lists[IDX], counts[IDX]);
#define JPXLG_RECT(IDX, R, C)                                                                   \
  if (counts[IDX]) {                                                                            \
    constexpr int vpb = 32 / ((R) < (C) ? (R) : (C));                                           \
    k_render_rect<R, C><<<(counts[IDX] + vpb - 1) / vpb, (R) * (C) / 4 * vpb, 0, s[IDX]>>>(     \
        a, lists[IDX], counts[IDX]);                                                            \
  }
#define JPXLG_R64(IDX, R, C) \
  if (counts[IDX])           \
    k_render_64<R, C><<<dim3(counts[IDX], 3), 512, sizeof(Rect64Smem<R, C>), s[IDX]>>>(a, lists[IDX]);
  // shape classes in kShapeSel order: DCT8, 16x16, 32x32, 16x8, 8x16, 32x8,
  // 8x32, 32x16, 16x32, DCT2x2, 64x64, 64x32, 32x64 (rows x cols of samples)
  JPXLG_R8(0, 0)
  JPXLG_RECT(1, 16, 16)
  JPXLG_RECT(2, 32, 32)
  JPXLG_RECT(3, 16, 8)
  JPXLG_RECT(4, 8, 16)
  JPXLG_RECT(5, 32, 8)
  JPXLG_RECT(6, 8, 32)
  JPXLG_RECT(7, 32, 16)
  JPXLG_RECT(8, 16, 32)
  JPXLG_R8(9, 1)
  JPXLG_R64(10, 64, 64)
  JPXLG_R64(11, 64, 32)
  JPXLG_R64(12, 32, 64)
  JPXLG_R8(13, 2)  // Hornuss
  JPXLG_R8(14, 3)  // DCT4x4
  JPXLG_R8(15, 4)  // DCT8x4
  JPXLG_R8(16, 5)  // DCT4x8
  JPXLG_R8(17, 6)  // AFV0..AFV3
  JPXLG_R8(18, 7)
  JPXLG_R8(19, 8)
  JPXLG_R8(20, 9)
#undef JPXLG_R8
#undef JPXLG_RECT
#undef JPXLG_R64
}

// ---------------------------------------------------------------------------
// R2 — restoration.rs:148 gaborish_into: acc = fma(w, s, acc) over (dy, dx)
// in row-major order from 0, kernel from GaborKernel::new (:111, with FMA).
// ---------------------------------------------------------------------------

// A thread forms V columns of kGabRun rows, keeping three rows of its V + 2
// columns in registers: 16-byte reads and writes where the rows are aligned
// (V = 4), one column a lane otherwise.  The columns' shared edges come from
// the L1.  Bound: memory latency and issue slots (18 operations a sample).
// Measured at 2048x2048: 47.7 -> 21.8 us (0.68 of the copy rate for its 101
// MB; 32 x 32 tiles in shared memory before).
constexpr int kGabRun = 8;
constexpr int kGabThreads = 128;

template <int V>
__global__ void __launch_bounds__(kGabThreads) k_gaborish(const float* __restrict__ in,
                                                          float* __restrict__ out, int w, int h,
                                                          float centre, float edge, float corner) {
  const size_t plane = (size_t)w * h;
  in += plane * blockIdx.z;
  out += plane * blockIdx.z;
  const int x = V * (blockIdx.x * kGabThreads + threadIdx.x), y0 = blockIdx.y * kGabRun;
  if (x >= w) return;
  const int xl = mirror1d(x - 1, w), xr = mirror1d(x + V, w);
  float r[3][V + 2];
  auto fetch = [&](float* row, int y) {
    const float* p = in + (size_t)mirror1d(y, h) * w;
    row[0] = __ldg(p + xl);
    if constexpr (V == 4) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(p + x));
      row[1] = v.x;
      row[2] = v.y;
      row[3] = v.z;
      row[4] = v.w;
    } else {
      row[1] = __ldg(p + x);
    }
    row[V + 1] = __ldg(p + xr);
  };
  fetch(r[0], y0 - 1);
  fetch(r[1], y0);
#pragma unroll
  for (int i = 0; i < kGabRun; ++i) {
    if (y0 + i >= h) return;
    fetch(r[2], y0 + i + 1);
    float o[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      float acc = 0.0f;
#pragma unroll
      for (int dy = 0; dy < 3; ++dy)
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) {
          const float wt = dx == 1 && dy == 1 ? centre : (dx == 1 || dy == 1 ? edge : corner);
          acc = __fmaf_rn(wt, r[dy][k + dx], acc);
        }
      o[k] = acc;
    }
    float* q = out + (size_t)(y0 + i) * w + x;
    if constexpr (V == 4) *reinterpret_cast<float4*>(q) = make_float4(o[0], o[1], o[2], o[3]);
    else *q = o[0];
#pragma unroll
    for (int k = 0; k < V + 2; ++k) {
      r[0][k] = r[1][k];
      r[1][k] = r[2][k];
    }
  }
}

void launch_gaborish(const float* in, float* out, int w, int h, cudaStream_t s) {
  const float w1 = 0.115169525f, w2 = 0.061248592f;
  float unnorm = fmaf(4.0f, w2, fmaf(4.0f, w1, 1.0f));
  float scale = 1.0f / unnorm;
  const bool vec = w % 4 == 0 && (((uintptr_t)in | (uintptr_t)out) & 15) == 0;
  const int cols = kGabThreads * (vec ? 4 : 1);
  const dim3 grid((w + cols - 1) / cols, (h + kGabRun - 1) / kGabRun, 3);
  auto run = [&](auto* kernel) {
    kernel<<<grid, kGabThreads, 0, s>>>(in, out, w, h, scale, w1 * scale, w2 * scale);
  };
  if (vec) run(k_gaborish<4>);
  else run(k_gaborish<1>);
}

// ---------------------------------------------------------------------------
// R3 — restoration.rs:619 epf_step_rows_impl.  Distances: per tap,
// d = fma(|a-b|, channel_scale[c], d) over channels then the cross (step 2:
// the pixel alone); weight max(0, fma(pos_mul*d, -inv_sigma, 1)) (exactly 1
// for zero distance); output sum_t fma(v, w, acc) / sum_t w.  Blocks with
// sigma < 0.3 are copied.  pos_mul = 2/3 on the 8x8 border of the reference
// pixel.  Mirrored padding of 3.
// ---------------------------------------------------------------------------

// A tap and its opposite take one distance: with
// d_k(p) = sum |t(p+q) - t(p+k+q)| over the cross q (channels outside),
// d_-k(p) = sum |t(p+q) - t(p-k+q)| has d_k(p-k)'s terms in the same order,
// |a - b| being |b - a| to the bit.  So step 0's twelve taps need six
// distance fields and step 1's four need two.  A CTA forms the fields of a
// 64 x 24 region in shared memory, a thread six rows of one column (RUN; two
// or four in regions of 8 or 16 rows for small frames): each
// |t - t'| of a column serves the three crosses above one another that hold
// it, and the lanes' consecutive columns read without conflicts.  It then
// weighs the taps of the region's inner pixels (a field is read at most two
// to the left and above, and one to the right).
// Bound: issue slots (81 to 84 % of them by step: FMA pipe, reads and the
// weights' ALU together).
// Measured, the three steps: 2048x2048 225 -> 155 us, 1920x1080 111 -> 86,
// 501x333 33 -> 27 (a thread per pixel and every tap's own distance before).
// Runs of four or eight rows and regions of 20 to 40 rows measured 160 to
// 166 us at 2048x2048; taller regions leave 1920x1080 a nearly empty wave.
constexpr int kEpfCols = 64;                     // region columns, a thread each
constexpr int kEpfThreads = 256;                 // four runs of rows
constexpr int kEpfTileW = kEpfCols + 8;          // 16-byte columns around the region

template <int STEP, int RUN>
struct EpfSmem {
  static constexpr int kRows = 4 * RUN;   // region rows, RUN a thread
  static constexpr int kTileH = kRows + 4;  // region rows -1 .. kRows + 2
  static constexpr int kFields = STEP == 0 ? 6 : (STEP == 1 ? 2 : 0);
  // Pixels written: the region's columns 2 .. 61 and rows from 2 where fields
  // are read to their left, right and above, all of it in step 2.
  static constexpr int kEdge = STEP < 2 ? 2 : 0;
  static constexpr int kOutW = STEP < 2 ? kEpfCols - 4 : kEpfCols, kOutH = kRows - kEdge;
  static constexpr int kBlocksW = kOutW / 8 + 2, kBlocksH = kOutH / 8 + 2;
  float t[3][kTileH][kEpfTileW];
  float d[kFields > 0 ? kFields : 1][kFields > 0 ? kRows : 1][kEpfCols];
  float sigma[kBlocksH][kBlocksW], inv[kBlocksH][kBlocksW];  // of the 8x8 blocks under the tile
};

__device__ __forceinline__ constexpr float epf_scale(int c) {
  return c == 0 ? 40.0f : (c == 1 ? 5.0f : 3.5f);
}

// The distance fields of a thread's run of rows of region column x from row
// y (t's origin is region row -1, column -2): fields (1,0), (0,1) and, for
// step 0, (1,1), (-1,1), (2,0), (0,2).  Row by row, a cross's north, centre
// row and south terms enter its sum in the order centre, west, east, north,
// south.
template <int STEP, int RUN>
__device__ __forceinline__ void epf_fields(EpfSmem<STEP, RUN>& sm, int x, int y) {
  constexpr int NF = EpfSmem<STEP, RUN>::kFields;
  constexpr int kAhead = STEP == 0 ? 2 : 1;  // rows a tap reaches down
  constexpr int fx[6] = {1, 0, 1, -1, 2, 0}, fy[6] = {0, 1, 1, 1, 0, 2};
  float d[NF][RUN];
#pragma unroll
  for (int k = 0; k < NF; ++k)
#pragma unroll
    for (int i = 0; i < RUN; ++i) d[k][i] = 0.0f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float s = epf_scale(c);
    float r[kAhead + 1][6];  // columns x - 2 .. x + 3
    auto fetch = [&](float* row, int j) {
#pragma unroll
      for (int i = 0; i < 6; ++i) row[i] = sm.t[c][y + j][x + i];
    };
#pragma unroll
    for (int j = 0; j < kAhead; ++j) fetch(r[j], j);
    float north[NF];
#pragma unroll
    for (int j = 0; j < RUN + 2; ++j) {  // run row j - 1
      fetch(r[kAhead], j + kAhead);
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        auto diff = [&](int q) { return fabsf(r[0][q] - r[fy[k]][q + fx[k]]); };
        const float centre = diff(2);
        if (j >= 2) d[k][j - 2] = __fmaf_rn(centre, s, d[k][j - 2]);
        if (j >= 1 && j <= RUN) {
          float& a = d[k][j - 1];
          a = __fmaf_rn(centre, s, a);
          a = __fmaf_rn(diff(1), s, a);
          a = __fmaf_rn(diff(3), s, a);
          a = __fmaf_rn(north[k], s, a);
        }
        north[k] = centre;
      }
#pragma unroll
      for (int k = 0; k < kAhead; ++k)
#pragma unroll
        for (int i = 0; i < 6; ++i) r[k][i] = r[k + 1][i];
    }
  }
#pragma unroll
  for (int k = 0; k < NF; ++k)
#pragma unroll
    for (int i = 0; i < RUN; ++i) sm.d[k][y + i][x] = d[k][i];
}

template <int STEP, int RUN>
__global__ void __launch_bounds__(kEpfThreads, STEP == 0 ? 3 : 4)
    k_epf(const float* __restrict__ in, float* __restrict__ out, const float* __restrict__ sigma,
          int w, int h, float step_mul4) {
  extern __shared__ __align__(16) unsigned char epf_smem[];
  using Smem = EpfSmem<STEP, RUN>;
  Smem& sm = *reinterpret_cast<Smem*>(epf_smem);
  constexpr int kEpfTileH = Smem::kTileH;
  const size_t plane = (size_t)w * h;
  constexpr int kEdge = Smem::kEdge;
  const int x0 = blockIdx.x * Smem::kOutW, y0 = blockIdx.y * Smem::kOutH;
  // Tile columns x0-4 .., region rows -1 ..: 16 bytes at a time inside the frame,
  // else mirrored at its borders, a warp per row.
  const int tx0 = x0 - 4, ty0 = y0 - kEdge - 1;
  if (tx0 >= 0 && ty0 >= 0 && tx0 + kEpfTileW <= w && ty0 + kEpfTileH <= h && (w & 3) == 0 &&
      (reinterpret_cast<uintptr_t>(in) & 15) == 0) {
    constexpr int kVec = kEpfTileW / 4;
    const float* src = in + (size_t)ty0 * w + tx0;
    for (int i = threadIdx.x; i < 3 * kEpfTileH * kVec; i += kEpfThreads) {
      const int v = i % kVec, r = i / kVec, c = r / kEpfTileH, ly = r - c * kEpfTileH;
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sm.t[c][ly][4 * v]);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                   "l"(src + plane * c + (size_t)ly * w + 4 * v)
                   : "memory");
    }
  } else {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int gx[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) gx[i] = mirror1d(tx0 + lane + 32 * i, w);
    for (int r = warp; r < 3 * kEpfTileH; r += kEpfThreads / 32) {
      const int c = r / kEpfTileH, ly = r - c * kEpfTileH;
      const float* row = in + plane * c + (size_t)mirror1d(ty0 + ly, h) * w;
#pragma unroll
      for (int i = 0; i < 3; ++i)
        if (32 * i + lane < kEpfTileW) {
          const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sm.t[c][ly][32 * i + lane]);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(row + gx[i])
                       : "memory");
        }
    }
  }
  const int bw = (w + 7) / 8, bh = (h + 7) / 8;
  constexpr int kBW = Smem::kBlocksW, kBH = Smem::kBlocksH;
  if (threadIdx.x < kBW * kBH) {
    const int bx = x0 / 8 + threadIdx.x % kBW, by = y0 / 8 + threadIdx.x / kBW;
    const float bs = bx < bw && by < bh ? __ldg(sigma + (size_t)by * bw + bx) : 1.0f;
    sm.sigma[0][threadIdx.x] = bs;
    sm.inv[0][threadIdx.x] = step_mul4 / bs;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int rx = threadIdx.x % kEpfCols, ry = threadIdx.x / kEpfCols * RUN;
  if constexpr (STEP < 2) {
    epf_fields<STEP, RUN>(sm, rx, ry);
    __syncthreads();
  }
  const int gx = x0 - kEdge + rx;
  if (rx < kEdge || rx >= kEdge + Smem::kOutW || gx >= w) return;
  // J.4.4 taps: the 5-pixel cross, plus the diagonals and +-2 for step 0.
  constexpr int NT = STEP == 0 ? 13 : 5;
  constexpr int tkx[13] = {0, -1, 1, 0, 0, 1, 1, -1, -1, -2, 2, 0, 0};
  constexpr int tky[13] = {0, 0, 0, -1, 1, -1, 1, 1, -1, 0, 0, 2, -2};
  // The field of each tap and where it is read: at the pixel for the
  // field's own tap, at the pixel plus the tap for the opposite one.
  constexpr int fld[13] = {0, 0, 0, 1, 1, 3, 2, 3, 2, 4, 4, 5, 5};
  constexpr bool opp[13] = {false, true,  false, true, false, true, false,
                            false, true,  true,  false, false, true};
  const bool side = (gx & 7) == 0 || (gx & 7) == 7;
  const int bcol = gx / 8 - x0 / 8;
#pragma unroll 1
  for (int i = 0; i < RUN; ++i) {
    const int cy = ry + i, gy = y0 - kEdge + cy;
    if (cy < kEdge || gy >= h) continue;
    auto at = [&](int c, int dx, int dy) { return sm.t[c][cy + 1 + dy][rx + 4 - kEdge + dx]; };
    const int brow = gy / 8 - y0 / 8;
    const float inv_sigma = sm.inv[brow][bcol];
    const float pos_mul = side || (gy & 7) == 0 || (gy & 7) == 7 ? 2.0f / 3.0f : 1.0f;
    auto dist = [&](int tp) {
      if constexpr (STEP == 2) {
        float d = 0.0f;
#pragma unroll
        for (int c = 0; c < 3; ++c)
          d = __fmaf_rn(fabsf(at(c, 0, 0) - at(c, tkx[tp], tky[tp])), epf_scale(c), d);
        return d;
      } else {
        return sm.d[fld[tp]][cy + (opp[tp] ? tky[tp] : 0)][rx + (opp[tp] ? tkx[tp] : 0)];
      }
    };
    // A zero distance weighs exactly 1 through the same expression (sigma is
    // at least 0.3, so its inverse is finite); fmaxf takes 0 for a NaN.
    auto weight = [&](float d) {
      return fmaxf(__fmaf_rn(pos_mul * d, -inv_sigma, 1.0f), 0.0f);
    };
    // The centre tap's distance sums |s - s| over the centre's own patch:
    // exactly 0 (weight 1) when every sample there is finite, not a number
    // otherwise.  The next tap's distance takes |s - s'| of the same samples
    // with positive scales, so it is finite only if they all are; then the
    // centre's terms are skipped, else evaluated as written.
    const float d1 = dist(1);
    float w0 = 1.0f;
    if (!isfinite(d1)) {
      float d = 0.0f;
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < (STEP == 2 ? 1 : 5); ++k) {
          constexpr int ix[5] = {0, -1, 1, 0, 0}, iy[5] = {0, 0, 0, -1, 1};
          const float v = at(c, ix[k], iy[k]);
          d = __fmaf_rn(fabsf(v - v), epf_scale(c), d);
        }
      w0 = weight(d);
    }
    float sum_w = 0.0f, acc[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int tp = 0; tp < NT; ++tp) {
      const float wt = tp == 0 ? w0 : weight(tp == 1 ? d1 : dist(tp));
      sum_w += wt;
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[c] = __fmaf_rn(at(c, tkx[tp], tky[tp]), wt, acc[c]);
    }
    const bool copy = sm.sigma[brow][bcol] < 0.3f;
    const size_t p = (size_t)gy * w + gx;
#pragma unroll
    for (int c = 0; c < 3; ++c) out[plane * c + p] = copy ? at(c, 0, 0) : acc[c] / sum_w;
  }
}

void launch_epf_step(int step, const float* in, float* out, const float* sigma, int w, int h,
                     int num_sms, cudaStream_t s) {
  // restoration.rs:356 epf_inv_sigma: step_multiplier * 4 * (1 - sqrt(0.5)) / sigma,
  // evaluated left to right; the numerator is formed here once.
  float sc = step == 0 ? 0.9f : (step == 1 ? 1.0f : 6.5f);
  float sm = 1.65f * sc;
  float num = sm * 4.0f * (1.0f - sqrtf(0.5f));
  auto run = [&](auto* kernel, auto smem) {
    using Smem = typename decltype(smem)::type;
    const dim3 grid((w + Smem::kOutW - 1) / Smem::kOutW, (h + Smem::kOutH - 1) / Smem::kOutH);
    kernel<<<grid, kEpfThreads, sizeof(Smem), s>>>(in, out, sigma, w, h, num);
  };
  // Rows of a thread: two or four where at most two CTAs come to an SM, else
  // six.  A short run computes more of its fields twice but ends sooner (the
  // three steps of 64x64: 26.7 us with six rows, 20.4 with two; of 501x333:
  // 27.5, 26.4 with four); beyond that the work is the time.
  auto pick = [&](auto st) {
    constexpr int STEP = decltype(st)::value;
    auto fits = [&](auto smem) {
      using Smem = typename decltype(smem)::type;
      return (long long)((w + Smem::kOutW - 1) / Smem::kOutW) *
                 ((h + Smem::kOutH - 1) / Smem::kOutH) <= 2LL * num_sms;
    };
    const std::common_type<EpfSmem<STEP, 2>> two;
    const std::common_type<EpfSmem<STEP, 4>> four;
    const std::common_type<EpfSmem<STEP, 6>> six;
    if (fits(two)) run(k_epf<STEP, 2>, two);
    else if (fits(four)) run(k_epf<STEP, 4>, four);
    else run(k_epf<STEP, 6>, six);
  };
  if (step == 0) pick(std::integral_constant<int, 0>{});
  else if (step == 1) pick(std::integral_constant<int, 1>{});
  else pick(std::integral_constant<int, 2>{});
}

// ---------------------------------------------------------------------------
// R4 — color.rs:673 OpsinInverse::convert (cube without pow, FMA matrix),
// then the output: linear planes; 8-bit sRGB as the decoder writes it
// (decode.rs:3498 round(linear_to_srgb(v)*255) clamped) found by binary
// search in the host-bisected level thresholds (plan-render lib.rs:333,
// identical by construction); or the level's linear value (lib.rs:437).
// ---------------------------------------------------------------------------

__device__ __forceinline__ int level_of(float x, const float* thr, int n) {
  if (!isfinite(x)) return 0;
  int lo = 0, hi = n;  // count of thresholds <= x
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (thr[mid] <= x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// x's level among 0 .. maxv, estimated from the transfer curve with the fast
// powf.  The scaled code's error is below 1e-6 of maxv; where the code is
// further than `margin` from a half-integer the estimate is the bisected
// level (whose own curve and scaling round within 0.004 of a code at 16
// bits) and *certain is set.  Not for values that are not finite.
__device__ __forceinline__ int level_estimate(float x, float maxv, float margin, bool* certain) {
  const float a = fabsf(x);
  const float e = a <= 0.0031308f ? 12.92f * a : 1.055f * __powf(a, 1.0f / 2.4f) - 0.055f;
  const float s = (x < 0.0f ? -e : e) * maxv;
  const float k = rintf(s);
  *certain = fabsf(s - k) < 0.5f - margin;
  return (int)fminf(fmaxf(k, 0.0f), maxv);
}

// x's level by the estimate where it is certain, else by its n thresholds.
__device__ __forceinline__ int shallow_level(float x, float maxv, float margin, const float* thr,
                                             int n) {
  bool certain;
  const int k = level_estimate(x, maxv, margin, &certain);
  return certain ? k : level_of(x, thr, n);
}

__device__ __forceinline__ float level_margin(float maxv) { return 1e-3f + 1e-6f * maxv; }

// The linear value of x's level for deep outputs (more than 256 levels) where
// the bracket of the estimated level does not hold x: stepping by one, then
// by binary search.  The thresholds decide, so the result is exactly the
// bisected level's.
static __device__ __noinline__ float level_value_search(float x, int est,
                                                        const float4* __restrict__ br,
                                                        const float* __restrict__ thr,
                                                        const float* __restrict__ levels, int n) {
  if (!isfinite(x)) return __ldg(&levels[0]);
#pragma unroll 1
  for (int it = 0; it < 4; ++it) {
    const float4 v = __ldg(&br[est]);
    const bool lo_ok = v.x <= x, hi_ok = x < v.y;
    if (lo_ok && hi_ok) return v.z;
    est += lo_ok ? 1 : -1;
  }
  return __ldg(&levels[level_of(x, thr, n)]);
}

// The same from v, the bracket of the estimated level est.
__device__ __forceinline__ float deep_level_value(float x, int est, const float4& v,
                                                  const float4* __restrict__ br,
                                                  const float* __restrict__ thr,
                                                  const float* __restrict__ levels, int n) {
  return v.x <= x && x < v.y ? v.z : level_value_search(x, est, br, thr, levels, n);
}

// Bound: issue slots (the powf's, the metric's cube roots).  An 8-bit level
// searches its thresholds only next to a half-integer (1 in 400), and a
// deeper pixel's three bracket entries are loaded at once.  Measured:
// 2048x2048 to 16-bit levels and the metric's XYB 77 -> 64 us, 1920x1080 to
// 8 bits 31.5 -> 18.4.  A byte per level beside the curve in shared memory,
// in place of the table's gathers: 65 to 77, not kept.
constexpr int kColourThreads = 256;

template <int KIND>
__global__ void __launch_bounds__(kColourThreads, 6)
    k_colour_out(const float* __restrict__ xyb, size_t n, const float* __restrict__ thr,
                 const float* __restrict__ levels, const float4* __restrict__ bracket, int nlev,
                 void* __restrict__ out, float* __restrict__ pxyb) {
  __shared__ float s_thr[255];
  __shared__ float s_lev[256];
  const bool shallow = KIND == 2 || (KIND == 3 && nlev <= 256);
  if (shallow) {
    for (int i = threadIdx.x; i < nlev - 1; i += blockDim.x) s_thr[i] = thr[i];
    for (int i = threadIdx.x; i < nlev; i += blockDim.x) s_lev[i] = levels[i];
    __syncthreads();
  }
  const float maxv = (float)(nlev - 1), margin = level_margin(maxv);
  auto level = [&](float x) { return shallow_level(x, maxv, margin, s_thr, nlev - 1); };
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    float x = xyb[i], y = xyb[n + i], b = xyb[2 * n + i];
    float gm[3] = {y + x, y - x, b};
    float mix[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float v = gm[c] - c_opsin_bias_cbrt[c];
      mix[c] = ((v * v) * v + c_opsin_bias[c]) * 1.0f;
    }
    float rgb[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      float acc = 0.0f;
#pragma unroll
      for (int c = 0; c < 3; ++c) acc = __fmaf_rn(c_opsin_m[r * 3 + c], mix[c], acc);
      rgb[r] = acc;
    }
    if (KIND == 1) {
      float* o = (float*)out;
      o[i] = rgb[0];
      o[n + i] = rgb[1];
      o[2 * n + i] = rgb[2];
    } else if (KIND == 4) {
      // jpxl-core color.rs:490 linear_to_srgb, odd-symmetric, unclipped.
      float* o = (float*)out;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const float v = rgb[q], av = fabsf(v);
        const float e = av <= 0.0031308f ? 12.92f * av : 1.055f * powf(av, 1.0f / 2.4f) - 0.055f;
        o[q * n + i] = v < 0.0f ? -e : e;
      }
    } else if (KIND == 2) {
      uint8_t* o = (uint8_t*)out;
#pragma unroll
      for (int q = 0; q < 3; ++q) o[3 * i + q] = (uint8_t)level(rgb[q]);
    } else {
      float lin[3];
      if (shallow) {
#pragma unroll
        for (int q = 0; q < 3; ++q) lin[q] = s_lev[level(rgb[q])];
      } else {
        // One 16-byte load of the bracket table gives a level's thresholds and
        // value, the three channels' at once.
        int k[3];
        float4 v[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          bool unused;
          k[q] = level_estimate(rgb[q], maxv, margin, &unused);
          v[q] = __ldg(&bracket[k[q]]);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q)
          lin[q] = deep_level_value(rgb[q], k[q], v[q], bracket, thr, levels, nlev - 1);
      }
      float* o = (float*)out;
      o[i] = lin[0];
      o[n + i] = lin[1];
      o[2 * n + i] = lin[2];
      // The metric's positive XYB of the rendered pixel (candidate side of
      // SSIMULACRA2's first scale), when the caller scores it next.
      if (pxyb) {
        float px[3];
        positive_xyb(lin[0], lin[1], lin[2], px);
        pxyb[i] = px[0];
        pxyb[n + i] = px[1];
        pxyb[2 * n + i] = px[2];
      }
    }
  }
}

void launch_colour_out(const float* xyb, int w, int h, int out_kind, const float* thresholds,
                       const float* levels, const float4* bracket, int nlevels, void* out,
                       float* pxyb, int num_sms, cudaStream_t s) {
  const size_t n = (size_t)w * h;
  const int blocks = (int)std::max<size_t>(
      1, std::min<size_t>((n + kColourThreads - 1) / kColourThreads, (size_t)num_sms * 16));
  auto run = [&](auto* kernel, float* px) {
    kernel<<<blocks, kColourThreads, 0, s>>>(xyb, n, thresholds, levels, bracket, nlevels, out, px);
  };
  if (out_kind == 1) run(k_colour_out<1>, nullptr);
  else if (out_kind == 2) run(k_colour_out<2>, nullptr);
  else if (out_kind == 4) run(k_colour_out<4>, nullptr);
  else run(k_colour_out<3>, pxyb);
}

cudaError_t configure_render_kernels() {
  auto allow = [](auto* kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  cudaError_t e;
  if ((e = allow(k_epf<0, 2>, sizeof(EpfSmem<0, 2>))) != cudaSuccess) return e;
  if ((e = allow(k_epf<0, 4>, sizeof(EpfSmem<0, 4>))) != cudaSuccess) return e;
  if ((e = allow(k_epf<0, 6>, sizeof(EpfSmem<0, 6>))) != cudaSuccess) return e;
  if ((e = allow(k_epf<1, 2>, sizeof(EpfSmem<1, 2>))) != cudaSuccess) return e;
  if ((e = allow(k_epf<1, 4>, sizeof(EpfSmem<1, 4>))) != cudaSuccess) return e;
  if ((e = allow(k_epf<1, 6>, sizeof(EpfSmem<1, 6>))) != cudaSuccess) return e;
  if ((e = allow(k_epf<2, 2>, sizeof(EpfSmem<2, 2>))) != cudaSuccess) return e;
  if ((e = allow(k_epf<2, 4>, sizeof(EpfSmem<2, 4>))) != cudaSuccess) return e;
  if ((e = allow(k_epf<2, 6>, sizeof(EpfSmem<2, 6>))) != cudaSuccess) return e;
  if ((e = allow(k_render_64<64, 64>, sizeof(Rect64Smem<64, 64>))) != cudaSuccess) return e;
  if ((e = allow(k_render_64<64, 32>, sizeof(Rect64Smem<64, 32>))) != cudaSuccess) return e;
  return allow(k_render_64<32, 64>, sizeof(Rect64Smem<32, 64>));
}

// ---------------------------------------------------------------------------
// R5 — LF of a decoded frame (jpxl-decode vardct/lf.rs:448 dequantize_lf and
// :351 adaptive_smoothing, decode.rs:3246 over the whole frame): dequantize
// (m * q / 2^extra_precision), apply the LF CfL, then smooth interior cells.
// ---------------------------------------------------------------------------

// A cell dequantizes its own neighbours again: thirty multiplications and
// divisions against a second launch and a plane between them (11.8 us in three
// launches with the multipliers' table, 9 in one).
__global__ void __launch_bounds__(256) k_lf_prepare(const int32_t* __restrict__ lfq, int bw, int bh,
                                                    float m0, float m1, float m2, float div,
                                                    float kx, float kb, bool smooth,
                                                    float* __restrict__ out, uint32_t global_scale,
                                                    float* __restrict__ mul_table) {
  if (blockIdx.x == gridDim.x - 1) fill_mul_table(global_scale, mul_table);
  const size_t nb = (size_t)bw * bh;
  const float m[3] = {m0, m1, m2};
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nb;
       i += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % bw), y = (int)(i / bw);
    auto lf = [&](size_t at, float* v) {
      const float dx = m0 * (float)lfq[at] / div;
      const float dy = m1 * (float)lfq[nb + at] / div;
      const float db = m2 * (float)lfq[2 * nb + at] / div;
      v[0] = dx + kx * dy;
      v[1] = dy;
      v[2] = db + kb * dy;
    };
    float sv[3];
    lf(i, sv);
    if (!smooth || x == 0 || y == 0 || x == bw - 1 || y == bh - 1) {
#pragma unroll
      for (int c = 0; c < 3; ++c) out[c * nb + i] = sv[c];
      continue;
    }
    // in the reference's order: W + E + N + S, NW + NE + SW + SE
    const int side[4][2] = {{-1, 0}, {1, 0}, {0, -1}, {0, 1}};
    const int diag[4][2] = {{-1, -1}, {1, -1}, {-1, 1}, {1, 1}};
    float se[3], sd[3];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float e[3], d[3];
      lf((size_t)(y + side[k][1]) * bw + x + side[k][0], e);
      lf((size_t)(y + diag[k][1]) * bw + x + diag[k][0], d);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        se[c] = k == 0 ? e[c] : se[c] + e[c];
        sd[c] = k == 0 ? d[c] : sd[c] + d[c];
      }
    }
    float wa[3], gap = 0.5f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      wa[c] = (0.052262735f * sv[c] + 0.2034514f * se[c]) + 0.03348292f * sd[c];
      gap = fmaxf(gap, fabsf(wa[c] - sv[c]) / m[c]);
    }
    const float factor = fmaxf(3.0f - 4.0f * gap, 0.0f);
#pragma unroll
    for (int c = 0; c < 3; ++c) out[c * nb + i] = (wa[c] - sv[c]) * factor + sv[c];
  }
}

void launch_lf_prepare(const int32_t* lfq, int bw, int bh, const float m[3], float div, float kx,
                       float kb, bool smooth, float* out, uint32_t global_scale, float* mul_table,
                       int num_sms, cudaStream_t s) {
  const size_t nb = (size_t)bw * bh;
  const int blocks = (int)std::max<size_t>(1, std::min<size_t>((nb + 255) / 256, num_sms * 4));
  k_lf_prepare<<<blocks, 256, 0, s>>>(lfq, bw, bh, m[0], m[1], m[2], div, kx, kb, smooth, out,
                                      global_scale, mul_table);
}

// A thread moves 16 bytes of the block at a time, several loads in flight:
// bound by the host link where the block is pinned host memory (about 2 us of
// latency, 200 GB/s).  48 small streams: 659 us with each block copied whole,
// 625 copied narrow and widened, 599 read in place.
template <typename Q>
__global__ void __launch_bounds__(256) k_unstage(const uint4* __restrict__ src, size_t nq,
                                                 size_t nrest, uint4* __restrict__ dst) {
  constexpr int kPer = 16 / sizeof(Q);  // coefficients of a load
  const size_t stride = (size_t)gridDim.x * blockDim.x;
#pragma unroll 4
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nq + nrest; i += stride) {
    const uint4 v = src[i];
    if (i >= nq) {
      dst[nq * (kPer / 4) + (i - nq)] = v;
      continue;
    }
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    int32_t q[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      q[k] = (int32_t)(Q)(w[k * sizeof(Q) / 4] >> (8 * (k * sizeof(Q) % 4)));
#pragma unroll
    for (int k = 0; k < kPer / 4; ++k)
      dst[i * (kPer / 4) + k] = make_uint4(q[4 * k], q[4 * k + 1], q[4 * k + 2], q[4 * k + 3]);
  }
}

void launch_unstage(const void* src, int q_bytes, size_t n, size_t rest, void* dst, int num_sms,
                    cudaStream_t s) {
  const size_t nq = n * q_bytes / 16, nr = rest / 16;
  const int blocks = (int)std::max<size_t>(1, std::min<size_t>((nq + nr + 255) / 256, num_sms * 4));
  auto go = [&](auto q) {
    k_unstage<decltype(q)><<<blocks, 256, 0, s>>>((const uint4*)src, nq, nr, (uint4*)dst);
  };
  if (q_bytes == 1) go(int8_t{});
  else if (q_bytes == 2) go(int16_t{});
  else go(int32_t{});
}

// The stream's earlier work is visible to this thread, and the release makes
// it visible to the host that reads the flag.
__global__ void k_publish(const uint32_t* __restrict__ err, uint32_t* flag) {
  const uint32_t e = *err;
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(flag), "r"(e) : "memory");
}

void launch_publish(const uint32_t* err, uint32_t* flag, cudaStream_t s) {
  k_publish<<<1, 1, 0, s>>>(err, flag);
}

// The special transforms on given blocks, one thread per block (a
// diagnostic of jpxlg_diag_special_blocks): kind 1 DCT2x2, 2..9 as
// special_block.
template <int KIND>
__global__ void __launch_bounds__(64) k_special_diag(const float* __restrict__ coef, int n,
                                                     float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float b[64], o[64];
#pragma unroll
  for (int k = 0; k < 64; ++k) b[k] = coef[(size_t)i * 64 + k];
  if constexpr (KIND == 1) {
    dct2x2_block(b);
#pragma unroll
    for (int k = 0; k < 64; ++k) o[k] = b[k];
  } else {
    special_block<KIND>(b, o);
  }
#pragma unroll
  for (int k = 0; k < 64; ++k) out[(size_t)i * 64 + k] = o[k];
}

bool launch_special_diag(int kind, const float* coef, int n, float* out, cudaStream_t s) {
  const int blocks = (n + 63) / 64;
  switch (kind) {
    case 1: k_special_diag<1><<<blocks, 64, 0, s>>>(coef, n, out); return true;
    case 2: k_special_diag<2><<<blocks, 64, 0, s>>>(coef, n, out); return true;
    case 3: k_special_diag<3><<<blocks, 64, 0, s>>>(coef, n, out); return true;
    case 4: k_special_diag<4><<<blocks, 64, 0, s>>>(coef, n, out); return true;
    case 5: k_special_diag<5><<<blocks, 64, 0, s>>>(coef, n, out); return true;
    case 6: k_special_diag<6><<<blocks, 64, 0, s>>>(coef, n, out); return true;
    case 7: k_special_diag<7><<<blocks, 64, 0, s>>>(coef, n, out); return true;
    case 8: k_special_diag<8><<<blocks, 64, 0, s>>>(coef, n, out); return true;
    case 9: k_special_diag<9><<<blocks, 64, 0, s>>>(coef, n, out); return true;
    default: return false;
  }
}

// The short forms of a rule against the rule itself over the floats of bit
// patterns first .. first + count - 1 (a diagnostic of jpxlg_diag_sweep):
// WHAT 0 the codec's cube root, 1 the metric's, 2 an output level by the
// estimate, 3 a deep level's value.  Counts the differences.
template <int WHAT>
__global__ void __launch_bounds__(256) k_sweep_diag(uint32_t first, uint32_t count,
                                                    const float* __restrict__ thr,
                                                    const float* __restrict__ levels,
                                                    const float4* __restrict__ bracket, int nlev,
                                                    unsigned long long* __restrict__ wrong) {
  const float maxv = (float)(nlev - 1), margin = level_margin(maxv);
  for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < count; i += gridDim.x * 256u) {
    const float x = __uint_as_float(first + i);
    float got, want;
    if constexpr (WHAT == 0) {
      got = cbrt_core(x);
      want = cbrt_core_f64(x);
    } else if constexpr (WHAT == 1) {
      got = cbrt_perceptual(x);
      want = cbrt_perceptual_f64(x);
    } else if constexpr (WHAT == 2) {
      got = (float)shallow_level(x, maxv, margin, thr, nlev - 1);
      want = (float)level_of(x, thr, nlev - 1);
    } else {
      bool unused;
      const int k = level_estimate(x, maxv, margin, &unused);
      got = deep_level_value(x, k, __ldg(&bracket[k]), bracket, thr, levels, nlev - 1);
      want = __ldg(&levels[level_of(x, thr, nlev - 1)]);
    }
    if (__float_as_uint(got) != __float_as_uint(want)) atomicAdd(wrong, 1ull);
  }
}

void launch_sweep_diag(int what, uint32_t first, uint32_t count, const float* thr,
                       const float* levels, const float4* bracket, int nlev,
                       unsigned long long* wrong, int num_sms, cudaStream_t s) {
  auto run = [&](auto* kernel) {
    kernel<<<num_sms * 8, 256, 0, s>>>(first, count, thr, levels, bracket, nlev, wrong);
  };
  if (what == 0) run(k_sweep_diag<0>);
  else if (what == 1) run(k_sweep_diag<1>);
  else if (nlev <= 256) run(k_sweep_diag<2>);
  else run(k_sweep_diag<3>);
}

void upload_afv(const double* basis, cudaStream_t s) {
  cudaMemcpyToSymbolAsync(g_afv, basis, sizeof(double) * 256, 0, cudaMemcpyHostToDevice, s);
}

void upload_dct64(const float* matrix, cudaStream_t s) {
  cudaMemcpyToSymbolAsync(g_dct64, matrix, sizeof(float) * 64 * 64, 0, cudaMemcpyHostToDevice, s);
}

void upload_render_constants(const float* opsin_m, const float* opsin_bias,
                             const float* opsin_bias_cbrt, cudaStream_t s) {
  cudaMemcpyToSymbolAsync(c_opsin_m, opsin_m, sizeof(float) * 9, 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_opsin_bias, opsin_bias, sizeof(float) * 3, 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_opsin_bias_cbrt, opsin_bias_cbrt, sizeof(float) * 3, 0,
                          cudaMemcpyHostToDevice, s);
}

}  // namespace jpxlg
