// k_ssim.cu — sm_103a kernels of SSIMULACRA2 (jpxl-perceptual) besides the
// blur (k_blur.cu):
//   S1, S2 k_pyramid       pyramid.rs:19 2x2 means, edge replicated, and
//                          color.rs:66 positive XYB (reproducible cube root)
//   S5 k_score_finish      the partial rows' sums per scale and quantity, norms,
//                          108 weights, remap (ssimulacra2.rs:509/:531)
//
// The per-strip partial sums that S5 folds come from k_blur_cols (f32 per
// 32 rows of a column, double-float above that, fixed order).
#include <algorithm>
#include <cstdint>

#include "jpxlg_common.cuh"
#include "jpxlg_internal.h"
#include "jpxlg_kernels.h"

namespace jpxlg {

// S1 — the pyramid of one frame in one launch: a CTA takes a 64 x 64 tile
// of the source, whose 2x2 means at every level (edge replicated,
// pyramid.rs:19) depend on that tile alone, and keeps each level in shared
// memory for the next; only the levels' positive XYB (S2) goes to memory.
// Bound by the cube roots (issue slots of the ALU and FMA pipes).  Measured
// at 2048x2048: 24.5 us for levels 1..5 against 39.9 us in five launches; with
// level 0, 4096x3072: 154 us (182 in six launches; 189 at four CTAs an SM).
constexpr int kPyrTile = 64;
constexpr int kPyrThreads = 256;

__global__ void __launch_bounds__(kPyrThreads, 6) k_pyramid(const float* __restrict__ rgb, int w,
                                                         int h, PyramidOut out, int n) {
  __shared__ float lev[3][kPyrTile / 2][kPyrTile / 2 + 1];
  __shared__ float lev2[3][kPyrTile / 4][kPyrTile / 4 + 1];
  const int t = threadIdx.x;
  const int x0 = blockIdx.x * kPyrTile, y0 = blockIdx.y * kPyrTile;
  const size_t plane = (size_t)w * h;
  auto put = [](float* dst, size_t np, size_t p, const float* v) {
    float o[3];
    positive_xyb(v[0], v[1], v[2], o);
    dst[p] = o[0];
    dst[np + p] = o[1];
    dst[2 * np + p] = o[2];
  };
  if (out.xyb[0]) {
    for (int i = t; i < kPyrTile * kPyrTile; i += kPyrThreads) {
      const int gx = x0 + i % kPyrTile, gy = y0 + i / kPyrTile;
      if (gx >= w || gy >= h) continue;
      const size_t p = (size_t)gy * w + gx;
      const float v[3] = {rgb[p], rgb[plane + p], rgb[2 * plane + p]};
      put(out.xyb[0], plane, p, v);
    }
  }
  // Level 1 from the source.
  int lw = (w + 1) / 2, lh = (h + 1) / 2;
  if (n > 1)
    for (int i = t; i < kPyrTile * kPyrTile / 4; i += kPyrThreads) {
      const int lx = i % (kPyrTile / 2), ly = i / (kPyrTile / 2);
      const int gx = x0 / 2 + lx, gy = y0 / 2 + ly;
      if (gx >= lw || gy >= lh) continue;
      const int sx0 = 2 * gx, sx1 = min(2 * gx + 1, w - 1);
      const size_t ra = (size_t)(2 * gy) * w, rb = (size_t)min(2 * gy + 1, h - 1) * w;
      float v[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float* p = rgb + plane * c;
        v[c] = (p[ra + sx0] + p[ra + sx1] + p[rb + sx0] + p[rb + sx1]) * 0.25f;
        lev[c][ly][lx] = v[c];
      }
      put(out.xyb[1], (size_t)lw * lh, (size_t)gy * lw + gx, v);
    }
  // The smaller levels from the one before, which alternates between the two
  // shared tiles.
  for (int s = 2; s < n; ++s) {
    __syncthreads();
    const int pw = lw, ph = lh, side = kPyrTile >> s;
    lw = (lw + 1) / 2;
    lh = (lh + 1) / 2;
    const int bx = x0 >> s, by = y0 >> s;
    if (t < side * side) {
      const int lx = t % side, ly = t / side, gx = bx + lx, gy = by + ly;
      if (gx < lw && gy < lh) {
        const int a0 = 2 * lx, a1 = min(2 * gx + 1, pw - 1) - 2 * bx;
        const int b0 = 2 * ly, b1 = min(2 * gy + 1, ph - 1) - 2 * by;
        float v[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (s & 1) {
            v[c] = (lev2[c][b0][a0] + lev2[c][b0][a1] + lev2[c][b1][a0] + lev2[c][b1][a1]) * 0.25f;
            lev[c][ly][lx] = v[c];
          } else {
            v[c] = (lev[c][b0][a0] + lev[c][b0][a1] + lev[c][b1][a0] + lev[c][b1][a1]) * 0.25f;
            lev2[c][ly][lx] = v[c];
          }
        }
        put(out.xyb[s], (size_t)lw * lh, (size_t)gy * lw + gx, v);
      }
    }
  }
}

void launch_pyramid(const float* rgb, int w, int h, const PyramidOut& out, int n, cudaStream_t s) {
  const dim3 grid((w + kPyrTile - 1) / kPyrTile, (h + kPyrTile - 1) / kPyrTile);
  k_pyramid<<<grid, kPyrThreads, 0, s>>>(rgb, w, h, out, n);
}

// S5 — ssimulacra2.rs:391 WEIGHTS (the metric's data table), :509
// weighted_error, :531 remap; pool.rs:60 norms.
__constant__ double c_weights[108] = {
    0.0, 0.0007376606707406586, 0.0, 0.0, 0.0007793481682867309, 0.0, 0.0,
    0.0004371155730107379, 0.0, 1.1041726426657346, 0.00066284834129271, 0.00015231632783718752,
    0.0, 0.0016406437456599754, 0.0, 1.8422455520539298, 11.441172603757666, 0.0,
    0.0007989109436015163, 0.000176816438078653, 0.0, 1.8787594979546387, 10.94906990605142, 0.0,
    0.0007289346991508072, 0.9677937080626833, 0.0, 0.00014003424285435884, 0.9981766977854967,
    0.00031949755934435053, 0.0004550992113792063, 0.0, 0.0, 0.0013648766163243398, 0.0, 0.0,
    0.0, 0.0, 0.0, 7.466890328078848, 0.0, 17.445833984131262, 0.0006235601634041466, 0.0, 0.0,
    6.683678146179332, 0.00037724407979611296, 1.027889937768264, 225.20515300849274, 0.0, 0.0,
    19.213238186143016, 0.0011401524586618361, 0.001237755635509985, 176.39317598450694, 0.0,
    0.0, 24.43300999870476, 0.28520802612117757, 0.0004485436923833408, 0.0, 0.0, 0.0,
    34.77906344483772, 44.835625328877896, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0,
    0.0008680556573291698, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0005313191874358747, 0.0,
    0.00016533814161379112, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0004179171803251336,
    0.0017290828234722833, 0.0, 0.0020827005846636437, 0.0, 0.0, 8.826982764996862,
    23.19243343998926, 0.0, 95.1080498811086, 0.9863978034400682, 0.9834382792465353,
    0.0012286405048278493, 171.2667255897307, 0.9807858872435379, 0.0, 0.0, 0.0,
    0.0005130064588990679, 0.0, 0.00010854057858411537};

struct FinishArgs {
  int nscales;
  int ctas[6];
  long long pixels[6];
};

constexpr int kReduceThreads = 256;

// S5 — one CTA per (quantity, scale): thread t sums the quantity's tile rows
// t, t + 256, ... of the scale in order in double-float, then the threads'
// sums meet in a fixed tree (warps, then warps in order).  The total goes to
// row 0 of the scale's partial rows, column k (only this CTA reads that
// column).  Deterministic for a given frame size; every load of a scale is
// in flight at once instead of behind one CTA's sequential chains.
//
// The CTA that finishes last (`ticket`, zeroed by the blur before) goes on to
// the norms, weights and remap of the 6 x 18 totals, a thread per term.
// Bound by the latency of its double-precision chain (two square roots, the
// weighted sum, one power): 3 + 13.6 us at 64x64 as two launches whose second
// took a channel's six terms in one thread, 12.5 us in one (13 by itself, 17 at
// 2048x2048, from a cold cache).
__global__ void __launch_bounds__(kReduceThreads) k_score_finish(DF* __restrict__ partials,
                                                                 FinishArgs fa,
                                                                 uint32_t* __restrict__ ticket,
                                                                 double* __restrict__ out,
                                                                 double* __restrict__ score,
                                                                 double* __restrict__ raw) {
  __shared__ DF wsum[kReduceThreads / 32];
  __shared__ double wterm[108];
  __shared__ bool last;
  const int k = blockIdx.x, s = blockIdx.y, t = threadIdx.x;
  size_t base = 0;
  for (int i = 0; i < s; ++i) base += fa.ctas[i];
  DF acc{0.0f, 0.0f};
#pragma unroll 4
  for (int i = t; i < fa.ctas[s]; i += kReduceThreads)
    acc = df_add(acc, partials[(base + i) * 18 + k]);
  const DF w = df_warp_sum(acc);
  if ((t & 31) == 0) wsum[t >> 5] = w;
  __syncthreads();
  if (t == 0) {
    DF tot = wsum[0];
    for (int i = 1; i < kReduceThreads / 32; ++i) tot = df_add(tot, wsum[i]);
    partials[base * 18 + k] = tot;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x * gridDim.y - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // ssimulacra2.rs:509 weighted error: weight i belongs to channel c, scale
  // sc, norm nn, map m with i = ((c * scales + sc) * 2 + nn) * 3 + m; the norm
  // itself is pool.rs:60's (mean, or fourth root of the mean).
  if (t < 3 * fa.nscales * 6) {
    const int m = t % 3, nn = (t / 3) % 2, c = t / 6 / fa.nscales, sc = t / 6 % fa.nscales;
    size_t b = 0;
    for (int i = 0; i < sc; ++i) b += fa.ctas[i];
    const float2 p = __ldcg(reinterpret_cast<const float2*>(partials) + b * 18 + c * 6 + 2 * m + nn);
    const double inv = 1.0 / (double)(fa.pixels[sc] > 0 ? fa.pixels[sc] : 1);
    double term = inv * df_value(DF{p.x, p.y});
    if (nn) term = sqrt(sqrt(term));
    out[2 + (sc * 3 + c) * 6 + nn * 3 + m] = term;
    wterm[t] = c_weights[t] * fabs(term);
  }
  __syncthreads();
  if (t >= 32) return;
  double part = 0.0;
  for (int i = t; i < 3 * fa.nscales * 6; i += 32) part += wterm[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (t != 0) return;
  const double err = part;
  double sc = err * 0.9562382616834844;
  sc = 6.248496625763138e-5 * sc * sc * sc + 2.326765642916932 * sc -
       0.020884521182843837 * sc * sc;
  const double value = sc > 0.0 ? 100.0 - 10.0 * pow(sc, 0.6276336467831387) : 100.0;
  out[0] = value;
  out[1] = err;
  if (score) *score = value;
  if (raw) *raw = err;
}

int launch_score_finish(DF* partials, const int* ctas_per_scale, int nscales,
                        const int* pixels_per_scale, void* carry, double* out, double* score,
                        double* raw, cudaStream_t s) {
  FinishArgs fa;
  fa.nscales = nscales;
  for (int i = 0; i < 6; ++i) {
    fa.ctas[i] = i < nscales ? ctas_per_scale[i] : 0;
    fa.pixels[i] = i < nscales ? pixels_per_scale[i] : 0;
  }
  k_score_finish<<<dim3(18, nscales), kReduceThreads, 0, s>>>(partials, fa, blur_ticket(carry), out,
                                                              score, raw);
  return 1;
}


}  // namespace jpxlg
