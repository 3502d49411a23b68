// jpxlg_common.cuh — device helpers shared by the sm_103a kernels of the
// lossy VarDCT pixel path: exact-parity cube roots, mirroring, the transform
// table, the DCT butterflies and the error word.
//
// Everything here is compiled with -fmad=false: a*b+c always rounds twice,
// exactly as the Rust reference (which never contracts), and __fmaf_rn is
// written out exactly where the reference calls mul_add.
#pragma once
#include <cstdint>
#include <type_traits>

#include <cuda_runtime.h>

#include "jpxlg_defs.cuh"

namespace jpxlg {

// ---- mirroring (18181-1 5.2 Mirror1D) ---------------------------------------
__device__ __forceinline__ int mirror1d(int c, int size) {
  // Bounded: a coordinate at most a few samples outside needs at most a few
  // reflections even for a one-sample plane.
  for (int i = 0; i < 64; ++i) {
    if (c < 0) c = -c - 1;
    else if (c >= size) c = 2 * size - 1 - c;
    else return c;
  }
  return 0;
}

// ---- exact-parity cube roots -----------------------------------------------
// The reference has two cube roots, each f64 iteration rounded once to f32:
// jpxl-core simd.rs:36 (estimate + 2 Halley steps) and jpxl-perceptual
// color.rs:46 (estimate + 4 Newton steps).  Both land within ~2^-24 ulp of the
// exact cube root, i.e. they return the correctly rounded cube root unless
// the exact root lies within that distance of a rounding midpoint.  The fast
// paths below find the correctly rounded root in f32 arithmetic (an estimate,
// then a double-float residual that places the exact root to within 2^-17.7
// ulp from the short path's estimate, 2^-20 ulp from the wide one's); where
// the root lies within 2^-17 ulp of a midpoint, or the input is outside the
// paths' ranges, the reference's own f64 iteration runs, so the result is the
// reference's bit for bit either way (test_gpu_sweeps.py compares them for
// every float).

static __device__ __noinline__ float cbrt_core_f64(float value) {
  const uint32_t B1 = 709958130u, B2 = 642849266u;
  uint32_t bits = __float_as_uint(value);
  uint32_t magnitude = bits & 0x7fffffffu;
  if (magnitude == 0 || magnitude >= 0x7f800000u) return value;
  uint32_t estimate;
  if (magnitude < 0x00800000u) {
    float scaled = value * 16777216.0f;
    estimate = (__float_as_uint(scaled) & 0x7fffffffu) / 3u + B2;
  } else {
    estimate = magnitude / 3u + B1;
  }
  double x = (double)value;
  double t = (double)__uint_as_float((bits & 0x80000000u) | estimate);
  for (int i = 0; i < 2; ++i) {
    double r = (t * t) * t;
    t = (t * ((x + x) + r)) / ((x + r) + r);
  }
  return (float)t;
}

static __device__ __noinline__ float cbrt_perceptual_f64(float value) {
  double x = (double)value;
  double a = fabs(x);
  unsigned long long ab = (unsigned long long)__double_as_longlong(a);
  double y = __longlong_as_double((long long)(ab / 3ull + (0x2A9F7893ull << 32)));
  for (int i = 0; i < 4; ++i) y -= (((y * y) * y) - a) / ((3.0 * y) * y);
  float root = (float)y;
  float signed_root = x < 0.0 ? -root : root;
  if (value == 0.0f || !isfinite(value)) return value;
  return signed_root;
}

// Correctly rounded cbrt of a > 0 in [2^-90, 2^90]; sets *ok = false where
// the decision is not certain to 2^-17 ulp.
__device__ __forceinline__ float cbrt_cr_fast(float a, bool* ok) {
  float y = cbrtf(a);
  uint32_t yb = __float_as_uint(y);
  float p = y * y;
  float e1 = __fmaf_rn(y, y, -p);   // y*y = p + e1 exactly
  float q = p * y;
  float e2 = __fmaf_rn(p, y, -q);   // p*y = q + e2 exactly
  float e3 = e1 * y;                // e1*y, rounded (relative 2^-48 of y^3)
  float d = (q - a) + (e2 + e3);    // y^3 - a; q - a is exact (Sterbenz)
  int e = (int)((yb >> 23) & 0xffu) - 127;
  float inv_ulp = __uint_as_float((uint32_t)(127 + 23 - e) << 23);  // 2^(23-e)
  // (cbrt(a) - y) in ulps of y.  The quotient needs ~2^-20 relative accuracy
  // only (|delta| < 2.5 against a 2^-17 decision margin), so the fast
  // division (at most 2 ulp off) serves.
  float delta = __fdividef(-d, 3.0f * p) * inv_ulp;
  float k = rintf(delta);
  float frac = fabsf(delta - k);
  *ok = frac < 0.5f - 7.62939453125e-06f && fabsf(delta) < 2.5f;  // 2^-17
  int ki = (int)k;
  uint32_t mant = yb & 0x7fffffu;
  if ((ki < 0 && mant < (uint32_t)(-ki)) || (ki > 0 && mant + (uint32_t)ki > 0x7fffffu))
    *ok = false;  // the step would cross a binade, where the ulp changes
  return __uint_as_float(yb + ki);
}

// Everything the short path leaves: the wide range, then the reference's own
// iteration (the metric's or the codec's).
template <bool kMetric>
static __device__ __noinline__ float cbrt_general(float v) {
  const float a = fabsf(v);
  if (a >= 8.0e-28f && a <= 1.2e27f) {
    bool ok;
    const float r = cbrt_cr_fast(a, &ok);
    if (ok) return copysignf(r, v);
  }
  return kMetric ? cbrt_perceptual_f64(v) : cbrt_core_f64(v);
}

// Correctly rounded cbrt of v in [2^-10, 2^10] (where an opsin mix of
// in-gamut light lies: 0.0038 to 1.004).  The estimate y = 2^(log2(a) / 3)
// is within 2^-20.5 of the root: log2 loses 2^-22.6 of at most 10, a third of
// it by ln 2 is 2^-21.4, and the product and the power add 2^-21.6.  The
// residual a - y^3 is formed to 2^-48 of a; the correction from it, with its
// second-order term, is at most as large as the estimate's error and loses
// seven times 2^-24 of itself (d, p, 3p, two for the reciprocal, d1, d2), so
// that it places the root to 2^-41.7 of itself, 2^-17.7 ulp below a power of
// two.  z is the nearest float to y plus the correction; it is certain unless
// the remainder is within 2^-17 ulp of half an ulp, or z a power of two (where
// the ulp changes).
// Measured against a library root with its residual, by itself: XYB of a
// 4096x3072 frame 122 -> 102 us, colour output of a 2048x2048 one 77 -> 71.
template <bool kMetric>
__device__ __forceinline__ float cbrt_of(float v) {
  float t, y, r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(v));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(t * 0.333333343f));
  const float p = y * y;
  const float e1 = __fmaf_rn(y, y, -p);  // y*y = p + e1 exactly
  const float q = p * y;
  const float e2 = __fmaf_rn(p, y, -q);  // p*y = q + e2 exactly
  const float d = (v - q) - __fmaf_rn(e1, y, e2);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(3.0f * p));
  const float d1 = d * r;                                       // (a - y^3) / 3y^2
  const float d2 = __fmaf_rn(-d1 * d1, 3.0f * y * r, d1);       // - d1^2 / y
  const float z = y + d2;
  const float rest = d2 - (z - y);  // exact: |d2| < y
  const uint32_t zb = __float_as_uint(z);
  const float half = __uint_as_float(zb & 0x7f800000u) * 5.9604644775390625e-08f;  // 2^-24
  if (v >= 0.0009765625f && v <= 1024.0f && (zb & 0x7fffffu) != 0u &&
      fabsf(rest) < half * 0.9999847412109375f)  // 1 - 2^-16
    return z;
  return cbrt_general<kMetric>(v);
}

// jpxl-core simd.rs:36 reproducible_cbrt, bit for bit.
__device__ __forceinline__ float cbrt_core(float v) { return cbrt_of<false>(v); }

// jpxl-perceptual color.rs:46 reproducible_cbrt, bit for bit.
__device__ __forceinline__ float cbrt_perceptual(float v) { return cbrt_of<true>(v); }

// ---- SSIMULACRA2 positive XYB (jpxl-perceptual color.rs:66) ------------------
// Opsin mix without FMA, the metric's reproducible cube root, then
// [14x + 0.42, y + 0.01, b - y + 0.55].
__device__ __forceinline__ void positive_xyb(float r, float g, float b, float* o) {
  float lm = 0.3f * r + 0.622f * g + 0.078f * b + 0.0037930734f;
  float mm = 0.23f * r + 0.692f * g + 0.078f * b + 0.0037930734f;
  float sm = 0.2434227f * r + 0.2047674f * g + 0.5518099f * b + 0.0037930734f;
  float lg = cbrt_perceptual(lm) - 0.1559542f;
  float mg = cbrt_perceptual(mm) - 0.1559542f;
  float sg = cbrt_perceptual(sm) - 0.1559542f;
  float x = 0.5f * (lg - mg);
  float y = 0.5f * (lg + mg);
  o[0] = x * 14.0f + 0.42f;
  o[1] = y + 0.01f;
  o[2] = (sg - y) + 0.55f;
}

// ---- paired f32 arithmetic (sm_100 family) ----------------------------------
// Two f32 lanes in one 64-bit register (lane 0 in the low word).  Each lane
// of add/sub.rn.f32x2 rounds exactly as the scalar f32 operation.
//
// Products need care: the assembler fuses a paired multiply with a following
// paired add into one rounding, whatever the rounding modifier or -fmad
// setting (measured on sm_103a: mul.rn.f32x2 then add.rn.f32x2 differed
// from the scalar mul-then-add in about one result in nine, and so did
// fma.rn.f32x2(a, b, -0.0) with the -0.0 as an immediate).  f2_mul is
// therefore fma.rn.f32x2(a, b, z) with z = (-0.0, -0.0) supplied at run time
// (a kernel argument), which the assembler cannot see through: one rounding
// of a*b, signed zeros included, exactly the scalar product.
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_pack(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float f2_lo(f2 v) {
  float a;
  asm("mov.b64 {%0, _}, %1;" : "=f"(a) : "l"(v));
  return a;
}
__device__ __forceinline__ float f2_hi(f2 v) {
  float b;
  asm("mov.b64 {_, %0}, %1;" : "=f"(b) : "l"(v));
  return b;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) {
  f2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// a * b per lane; nz must be the run-time pair (-0.0f, -0.0f).
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b, f2 nz) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(nz));
  return d;
}
// a * b + c per lane with one rounding (the paired __fmaf_rn).
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// ---- double-float (f32 pair) sums --------------------------------------------
// Products of two f32 are split exactly (two_prod); sums keep hi + lo to
// about 2^-46 per addition, so a sum over n terms lies within
// n * 2^-46 * sum|t| of the exact sum, at f32 issue rates (GB300's FP64
// rate is a small fraction of its FP32 rate).  hi + lo converts to f64
// exactly.
struct DF {
  float hi, lo;
};
__device__ __forceinline__ DF df_two_prod(float a, float b) {
  float p = a * b;
  return {p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ DF df_add(DF a, DF b) {
  float s = a.hi + b.hi;
  float bb = s - a.hi;
  float e = (a.hi - (s - bb)) + (b.hi - bb);
  e = e + (a.lo + b.lo);
  float h = s + e;
  return {h, e - (h - s)};
}
// Fixed-order butterfly over a warp; every lane ends with the same sum.
__device__ __forceinline__ DF df_warp_sum(DF v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    DF w{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
    v = df_add(v, w);
  }
  return v;
}
__device__ __forceinline__ double df_value(DF v) { return (double)v.hi + (double)v.lo; }

// ---- reconstruct.rs:50 bias_adjust ------------------------------------------
// q -> q * bias for |q| <= 1, else q - 0.145 / q.  The expression is odd in q
// under round-to-nearest, so |q| < kBiasQuotN reads 0.145f / |q| from a table
// that the host fills with the same IEEE division, and the sign is applied
// last; larger |q| divide.
constexpr int kBiasQuotN = 256;
extern __device__ float g_bias_quot[kBiasQuotN];

__device__ __forceinline__ float bias_adjust_q(int32_t q, float bias) {
  const float f = (float)q;
  if (q >= -1 && q <= 1) return f * bias;
  const int32_t aq = q < 0 ? -q : q;
  const float af = (float)aq;
  const float t = aq < kBiasQuotN ? __ldg(&g_bias_quot[aq]) : 0.145f / af;
  const float r = af - t;
  return q < 0 ? -r : r;
}

// ---- DCT butterflies (jpxl-core dct.rs:235-465) -----------------------------
// Orthonormal DCT-IV leaves live in constant memory (filled by the host from
// the reference's first-row magnitudes); loops over them are unrolled, so
// every coefficient is a constant-bank operand.
extern __constant__ float c_iv4[16];
extern __constant__ float c_iv8[64];
extern __constant__ float c_iv16[256];

constexpr float kSqrtHalf = 0.707106769f;
constexpr float kCosPi8 = 0.9238795f;
constexpr float kSinPi8 = 0.38268343f;

template <int M>
__device__ __forceinline__ float iv_coef(int u, int n) {
  if constexpr (M == 4) return c_iv4[u * 4 + n];
  else if constexpr (M == 8) return c_iv8[u * 8 + n];
  else return c_iv16[u * 16 + n];
}

template <int M>
__device__ __forceinline__ void dct_iv(float* v) {
  if constexpr (M == 2) {
    float x0 = v[0], x1 = v[1];
    v[0] = kCosPi8 * x0 + kSinPi8 * x1;
    v[1] = kSinPi8 * x0 - kCosPi8 * x1;
  } else {
    float x[M];
#pragma unroll
    for (int i = 0; i < M; ++i) x[i] = v[i];
#pragma unroll
    for (int u = 0; u < M; ++u) {
      float acc = 0.0f;
#pragma unroll
      for (int n = 0; n < M; ++n) acc = acc + iv_coef<M>(u, n) * x[n];
      v[u] = acc;
    }
  }
}

__device__ __forceinline__ void dct_ii_2(float* v) {
  float x0 = v[0], x1 = v[1];
  v[0] = (x0 + x1) * kSqrtHalf;
  v[1] = (x0 - x1) * kSqrtHalf;
}

template <int N>
__device__ __forceinline__ void dct_ii(float* v) {
  if constexpr (N == 1) {
  } else if constexpr (N == 2) {
    dct_ii_2(v);
  } else {
    constexpr int H = N / 2;
    float even[H], odd[H];
#pragma unroll
    for (int k = 0; k < H; ++k) {
      even[k] = v[k] + v[N - 1 - k];
      odd[k] = v[k] - v[N - 1 - k];
    }
    dct_ii<H>(even);
    dct_iv<H>(odd);
#pragma unroll
    for (int k = 0; k < H; ++k) {
      v[2 * k] = even[k] * kSqrtHalf;
      v[2 * k + 1] = odd[k] * kSqrtHalf;
    }
  }
}

template <int N>
__device__ __forceinline__ void dct_iii(float* v) {
  if constexpr (N == 1) {
  } else if constexpr (N == 2) {
    dct_ii_2(v);
  } else {
    constexpr int H = N / 2;
    float even[H], odd[H];
#pragma unroll
    for (int k = 0; k < H; ++k) {
      even[k] = v[2 * k] * kSqrtHalf;
      odd[k] = v[2 * k + 1] * kSqrtHalf;
    }
    dct_iii<H>(even);
    dct_iv<H>(odd);
#pragma unroll
    for (int k = 0; k < H; ++k) {
      v[k] = even[k] + odd[k];
      v[N - 1 - k] = even[k] - odd[k];
    }
  }
}

// dct.rs:731/749: normative scaling after the butterfly.  The factors are
// 1/sqrtf(N) and sqrtf(N) in f32, as the reference computes them.
template <int N>
__device__ __forceinline__ void dct_1d(float* v) {
  dct_ii<N>(v);
  const float f = 1.0f / __fsqrt_rn((float)N);
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] *= f;
}
template <int N>
__device__ __forceinline__ void idct_1d(float* v) {
  dct_iii<N>(v);
  const float f = __fsqrt_rn((float)N);
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] *= f;
}

// ---- one DCT shared by a group of warps -------------------------------------
// A 1-D transform of N points falls apart into dot products: with
// i = (2u + 1) 2^t, the odd half of level t of the recursion is dct_iv of
// N >> (t + 1) points, each output of which is independent of the others.
// N / 4 "shares" of four outputs each cover a transform: shares
// 0 .. N/8 - 1 the odd half of level 0, the next N/16 level 1, and so on; the
// last one holds levels of two points and the final pair.  A warp takes one
// share of 32 (or 2 x 16) columns, so a 32-point transform is a few hundred
// instructions in each of eight warps instead of fifteen hundred in one, and
// no warp's code is long.  The operations and their order are those of dct_ii
// and dct_iii above.

// Scaling by sqrt(1/2) once per level, as the recursion applies it.
template <int T>
__device__ __forceinline__ float scale_half(float v) {
#pragma unroll
  for (int i = 0; i < T; ++i) v = v * kSqrtHalf;
  return v;
}

// acc[i] = sum over n of iv<M>(u0 + i, n) x[n], n in order from 0.
template <int M>
__device__ __forceinline__ void iv_dot4(int u0, const float* x, float* acc) {
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] = 0.0f;
#pragma unroll
  for (int n = 0; n < M; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = acc[i] + iv_coef<M>(u0 + i, n) * x[n];
}

// Forward: share `g` of the N-point transform of get(0 .. N-1); put(index,
// value) receives its four outputs, scaled as dct_1d.
template <int N, typename Get, typename Put>
__device__ __forceinline__ void dct_share(int g, Get get, Put put) {
  const float f = 1.0f / __fsqrt_rn((float)N);
  float e[N / 2];  // the running even half, from level 1 on
  if (g < N / 8) {
    float d[N / 2], acc[4];
#pragma unroll
    for (int n = 0; n < N / 2; ++n) d[n] = get(n) - get(N - 1 - n);
    iv_dot4<N / 2>(4 * g, d, acc);
#pragma unroll
    for (int i = 0; i < 4; ++i) put(2 * (4 * g + i) + 1, scale_half<1>(acc[i]) * f);
    return;
  }
#pragma unroll
  for (int n = 0; n < N / 2; ++n) e[n] = get(n) + get(N - 1 - n);
  g -= N / 8;
  if (N >= 16 && g < N / 16) {
    float d[N / 4], acc[4];
#pragma unroll
    for (int n = 0; n < N / 4; ++n) d[n] = e[n] - e[N / 2 - 1 - n];
    iv_dot4<N / 4>(4 * g, d, acc);
#pragma unroll
    for (int i = 0; i < 4; ++i) put(2 * (2 * (4 * g + i) + 1), scale_half<2>(acc[i]) * f);
    return;
  }
#pragma unroll
  for (int n = 0; n < N / 4; ++n) e[n] = e[n] + e[N / 2 - 1 - n];
  g -= N / 16;
  if constexpr (N == 32) {
    if (g < 1) {
      float d[4], acc[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) d[n] = e[n] - e[7 - n];
      iv_dot4<4>(0, d, acc);
#pragma unroll
      for (int i = 0; i < 4; ++i) put(4 * (2 * i + 1), scale_half<3>(acc[i]) * f);
      return;
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) e[n] = e[n] + e[7 - n];
  }
  // four points left: dct_ii<4>
  constexpr int T = N == 32 ? 3 : 2;  // levels above
  float odd[2] = {e[0] - e[3], e[1] - e[2]};
  dct_iv<2>(odd);
  float even[2] = {e[0] + e[3], e[1] + e[2]};
  dct_ii_2(even);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    put((N / 4) * (2 * k), scale_half<T + 1>(even[k]) * f);
    put((N / 4) * (2 * k + 1), scale_half<T + 1>(odd[k]) * f);
  }
}

// Levels of odd halves of two and more points below an N-point transform.
__host__ __device__ constexpr int dct_levels(int n) { return n <= 4 ? 1 : 1 + dct_levels(n / 2); }

// Inverse, first half: share `g`'s dot products from get(0 .. N-1) into
// put(row, value): the odd half of level t at rows N - (N >> t) ..., the last
// pair in rows N - 2, N - 1.  N = 8, 16, 32.
template <int N, typename Get, typename Put>
__device__ __forceinline__ void idct_share(int g, Get get, Put put) {
  auto level = [&](auto lt, int share) {
    constexpr int t = decltype(lt)::value, M = N >> (t + 1);
    float x[M], acc[4];
#pragma unroll
    for (int n = 0; n < M; ++n) x[n] = scale_half<t + 1>(get((2 * n + 1) << t));
    iv_dot4<M>(4 * share, x, acc);
#pragma unroll
    for (int i = 0; i < 4; ++i) put(N - (N >> t) + 4 * share + i, acc[i]);
  };
  if (g < N / 8) {
    level(std::integral_constant<int, 0>{}, g);
    return;
  }
  g -= N / 8;
  if constexpr (N >= 16) {
    if (g < N / 16) {
      level(std::integral_constant<int, 1>{}, g);
      return;
    }
    g -= N / 16;
  }
  if constexpr (N == 32) {
    if (g < 1) {
      level(std::integral_constant<int, 2>{}, 0);
      return;
    }
  }
  constexpr int T = dct_levels(N);
  float odd[2] = {scale_half<T>(get(N / 4)), scale_half<T>(get(3 * N / 4))};
  dct_iv<2>(odd);
  float even[2] = {scale_half<T>(get(0)), scale_half<T>(get(N / 2))};
  dct_ii_2(even);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    put(N - 4 + k, odd[k]);
    put(N - 2 + k, even[k]);
  }
}

// Inverse, second half: outputs k and N - 1 - k (k < N / 2) from the rows of
// idct_share, scaled as idct_1d.
template <int N, typename Get>
__device__ __forceinline__ void idct_pair(int k, Get get, float* lo, float* hi) {
  constexpr int kLevels = dct_levels(N);
  int at[kLevels];  // position within the half of level t
  at[0] = k;
#pragma unroll
  for (int t = 1; t < kLevels; ++t) {
    const int m = N >> (t + 1);
    at[t] = at[t - 1] < m ? at[t - 1] : 2 * m - 1 - at[t - 1];
  }
  // from the last pair outwards
  float even = get(N - 2 + at[kLevels - 1]);
#pragma unroll
  for (int t = kLevels - 1; t >= 1; --t) {
    const float odd = get(N - (N >> t) + at[t]);
    even = at[t - 1] < (N >> (t + 1)) ? even + odd : even - odd;
  }
  const float odd = get(at[0]), f = __fsqrt_rn((float)N);
  *lo = (even + odd) * f;
  *hi = (even - odd) * f;
}

}  // namespace jpxlg
