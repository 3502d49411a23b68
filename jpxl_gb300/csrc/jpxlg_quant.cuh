// jpxlg_quant.cuh — the HF quantizer shared by the encoder's kernels
// (jpxl-encode-policy quantize.rs): clamp_round, the nearest-reconstruction
// choice and the residual bit proxy.
#pragma once
#include "jpxlg_common.cuh"

namespace jpxlg {

// 1 - the reference's per-channel quant bias (color.rs:591), defined in k_encode.cu.
extern __constant__ float c_quant_bias[3];

// quantize.rs:1720 clamp_round: v +- 0.5 then truncate; false = Err.
__device__ __forceinline__ bool clamp_round(float v, int32_t* out) {
  if (!isfinite(v)) return false;
  float adjusted = signbit(v) ? v - 0.5f : v + 0.5f;
  if (!(fabsf(adjusted) < 2147483648.0f)) return false;
  int32_t q = (int32_t)adjusted;
  if ((q < 0 ? -q : q) > (1 << 20)) return false;
  *out = q;
  return true;
}

__device__ __forceinline__ float bias_adjust(int32_t q, float bias) { return bias_adjust_q(q, bias); }

// quantize.rs:1400 HfQuantizer::choose (nearest reconstruction, ties to the
// smaller magnitude) with step = scale * matrix and the zero threshold
// 0.5 * bias * step, both formed as quantize.rs:334 forms them, as it stands:
// candidates {0, e-1, e, e+1} around e = clamp_round(target / step), of which
// only e and its neighbour on the target's side can win, reconstruction
// levels increasing with q.  Out of line: choose below takes it for quotients
// beyond its table, for steps that are not positive and finite and for
// targets that are not finite, where the error conditions are decided.
static __device__ __noinline__ int32_t choose_general(float target, float step, float bias,
                                                      uint32_t* err, float* recon) {
  *recon = 0.0f;
  if (!(isfinite(step) && step > 0.0f)) {
    raise_error(err, kDevBadStep);
    return 0;
  }
  if (fabsf(target) <= 0.5f * bias * step) return 0;
  int32_t e;
  if (!clamp_round(target / step, &e)) {
    raise_error(err, kDevQuantRange);
    return 0;
  }
  const float re = bias_adjust(e, bias) * step;
  const int32_t nb = re < target ? e + 1 : e - 1;
  const float rn = bias_adjust(nb, bias) * step;
  // Candidates in the reference's update rule: q = 0 first (its level is 0,
  // error |target|), then the pair in increasing q; |q| > 2^20 is outside
  // its range.
  int32_t best = 0;
  float best_err = fabsf(target);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int32_t cand = (i == 0) == (e < nb) ? e : nb;
    const float r = (i == 0) == (e < nb) ? re : rn, er = fabsf(r - target);
    if (abs(cand) <= (1 << 20) &&
        (er < best_err || (er == best_err && abs(cand) < abs(best)))) {
      best = cand;
      best_err = er;
      *recon = r;
    }
  }
  return best;
}

__device__ __forceinline__ uint32_t residual_bits(int32_t q) {
  if (q == 0) return 0;
  uint32_t aq = (uint32_t)(q < 0 ? -q : q);
  return (32u - __clz(aq)) + 1u;
}

// Entry e of channel c: bias_adjust (reconstruct.rs:50, channel c's bias) at
// e - 1, e and e + 1 (0 at -1), and their residual bits in the fourth word's
// bytes, from the host (upload_dct_constants).
constexpr int kLevelN = 1024;  // a power of two
extern __device__ float4 g_levels[3][kLevelN];

// 1 / step to an ulp, for the choice's centre.
__device__ __forceinline__ float approx_rcp(float step) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(step));
  return r;
}

// choose_general for channel c on a table entry, without branches, so that
// several choices overlap; ok false: choose_general decides.  rstep is within
// a few ulps of 1 / step.
//
// Everything in it is odd in the target (ties go to the smaller magnitude on
// either side), so it works on a = |target|.  The levels around a are those
// of the floor and the ceiling of a / step: a level lies at most 0.08 steps
// below its integer.  The centre e, a / step rounded with an error of a few
// 2^-24 of it (2^23 + it leaves its integer in the low bits), is one of the
// two; the level of e tells which, and one table entry holds the other's
// level too.  The lower level wins ties; zero, a third candidate, never
// beats a lower level above it (that level lies below 2a), and the threshold
// test decides zero against the first.
struct Choice {
  float4 v;
  int e, place;  // q's magnitude is e - 1 + place, 0 under the threshold
  float level;   // its level times step
  bool zero, ok;
  __device__ __forceinline__ Choice(int c, float target, float step, float rstep) {
    const float a = fabsf(target), va = a * rstep;
    ok = va < (float)kLevelN - 0.5f && step > 0.0f && step < __int_as_float(0x7f800000);
    e = __float_as_int(va + 8388608.0f) & (kLevelN - 1);
    v = __ldg(&g_levels[c][e]);
    const float re = v.y * step;
    const bool up = re < a;  // e is the floor
    const float ro = (up ? v.z : v.x) * step;
    const float lo = up ? re : ro, hi = up ? ro : re;
    const bool upper = fabsf(hi - a) < fabsf(lo - a);
    place = (up ? 1 : 0) + (upper ? 1 : 0);
    level = upper ? hi : lo;
    zero = a <= 0.5f * c_quant_bias[c] * step;
  }
  __device__ __forceinline__ uint32_t bits() const {
    return zero ? 0u : (__float_as_uint(v.w) >> (8 * place)) & 0xffu;
  }
  __device__ __forceinline__ int32_t q(float target) const {
    const int m = zero ? 0 : e - 1 + place;
    return target < 0.0f ? -m : m;
  }
  __device__ __forceinline__ float recon(float target) const {
    const float r = zero ? 0.0f : level;
    return target < 0.0f ? 0.0f - r : r;  // +0 for zero
  }
};

// The choice of N targets, each with its own step.
template <int N>
__device__ __forceinline__ void choose_n(int c, const float* target, const float* step,
                                         uint32_t* err, int32_t* q, float* recon) {
  bool ok = true;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const Choice ch(c, target[i], step[i], approx_rcp(step[i]));
    ok = ok && ch.ok;
    q[i] = ch.q(target[i]);
    recon[i] = ch.recon(target[i]);
  }
  if (!ok)
#pragma unroll 1
    for (int i = 0; i < N; ++i)
      q[i] = choose_general(target[i], step[i], c_quant_bias[c], err, &recon[i]);
}
__device__ __forceinline__ int32_t choose(int c, float target, float step, uint32_t* err,
                                          float* recon) {
  int32_t q;
  choose_n<1>(c, &target, &step, err, &q, recon);
  return q;
}

}  // namespace jpxlg
