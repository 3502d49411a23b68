// k_blur.cu — SSIMULACRA2's Gaussian (jpxl-perceptual blur.rs) evaluated to
// the reference's f32 outputs, and the candidate side of one scale.
//
// blur.rs runs along every row, then along every column of that result,
// three f64 two-pole resonators (feedback 2 cos(k pi / 10) and -1, k = 1, 3,
// 5) fed with s_j = f32(x[j-6] + x[j+4]), and rounds their summed output to
// f32 once per sample (blur.rs:164 step, :414 horizontal_padded, :574
// vertical_row).  Split s_j = (x[j-6] + x[j+4]) + e_j, with e_j the rounding
// error of the f32 pair sum (exact in f32).  The resonators fed with the
// exact pair sums have a finite response: the 9-tap symmetric FIR
// FIR_j = sum_d tap_d x[j+d], |d| <= 4 (the fifth harmonics cancel).  Fed
// with the e's they ring without damping for the rest of the line: R_j.  So
//
//     output_j = f32(FIR_j + R_j)
//
// up to the reference's own f64 noise (~1e-16 relative).  R is a size- and
// content-dependent ripple of order 1e-7 of the signal; a plain f32 FIR
// misses it and lands tens of ulps away, which SSIMULACRA2's variance
// differences (sigma - mu^2 with C2 = 0.0009) amplify into score errors of
// a tenth of a point on large near-identical pairs.  Here FIR_j is a
// double-float dot product (exact pair sums, exact products, compensated
// accumulation; taps as hi + lo from the f64 recursion's impulse response)
// and R_j comes from f32 resonators (R's own relative error of 1e-6 is far
// below an output ulp); one final f32 addition rounds FIR_j + R_j.
//
// Lines are split into segments.  Each segment runs its resonators from
// rest; a scan over the segments (after L steps the state is M^L times the
// entry state plus the segment's own response, M the resonator's 2x2 step
// matrix) gives each segment its entry state; each segment adds the
// homogeneous response of that state to its R from rest, and the FIR
// outputs, independent of one another, are formed in parallel.  Arithmetic
// is paired (two f32 lanes per instruction, each rounded as the scalar
// operation): rows two at a time in the row pass, columns two at a time in
// the column pass.
//   B1 k_blur_rows<NQ>     one CTA per row pair, channel and quantity (x, x*x
//                          and r*x, rounded to f32 as blur.rs:395 forms them);
//                          one segment per thread, the scan across the CTA's
//                          threads
//   B2 k_blur_cols<NQ>     one CTA per 64-row segment of a 32-column strip
//                          and channel: the ripple from rest per column and
//                          quantity in four quarters, the chained scan over
//                          the strip's segments (each column waits,
//                          boundedly, for the previous segment's published
//                          state; CTAs take their segments in the order they
//                          start), then the outputs; NQ = 2 writes mu and
//                          sigma11 (reference.rs:90), NQ = 3 evaluates
//                          pool.rs:248's per-pixel terms on the blurred mu2,
//                          sigma22, sigma12 and writes one row of partial
//                          sums per 32 x 32 tile
// Each kernel runs every scale of the pyramid in one launch: a scale's CTAs
// follow the larger scale's, so that the small scales' chains fill the last
// waves instead of running alone behind launch gaps.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "jpxlg_common.cuh"
#include "jpxlg_internal.h"
#include "jpxlg_kernels.h"

namespace jpxlg {

struct BlurConsts {
  float a[3], b[3];    // MUL_IN and MUL_PREV (blur.rs:41/:47) in f32, for the ripple
  float th[5], tl[5];  // FIR taps (centre, +-1 .. +-4) as hi + lo
  // U[k][n] = sin((n+1) w_k) / sin(w_k), w_k = (2k+1) pi / 10: M_k^n is
  // [[U[n], -U[n-1]], [U[n-1], -U[n-2]]] (period 20 in n; U[-1] = 0).
  float U[3][20];
};
__constant__ BlurConsts c_blur;

// The constants as lane pairs for the paired forms, and the pair (+0, +0)
// for negations.
struct BlurPairs {
  f2 a[3], b[3], th[5], tl[5], nth[5], ntl[5], z;  // nth, ntl: the taps negated
  f2 U[3][24];  // BlurConsts::U, its first four entries again past the end
};
__constant__ BlurPairs c_blur2;

// blur.rs:41 / :47.
static const double kMulIn[3] = {0.05529523572608661, -0.05883668702694998,
                                 0.012955819110517063};
static const double kMulPrev[3] = {1.902113032590307, 1.1755705045849463,
                                   1.2246467991473532e-16};

void upload_blur_consts(cudaStream_t s) {
  BlurConsts bc;
  for (int k = 0; k < 3; ++k) {
    bc.a[k] = (float)kMulIn[k];
    bc.b[k] = (float)kMulPrev[k];
  }
  // Tap d: the f64 recursion's response at output p + d to a unit sample at
  // p, the sample entering as the right (x[j+4]) and later the left
  // (x[j-6]) member of the pair sums.
  for (int d = 0; d <= 4; ++d) {
    double prev[3] = {0, 0, 0}, prev2[3] = {0, 0, 0}, out = 0.0;
    const int p = 16;
    for (int j = 0; j <= p + d; ++j) {
      const double s = (j + 4 == p ? 1.0 : 0.0) + (j - 6 == p ? 1.0 : 0.0);
      double o[3];
      for (int k = 0; k < 3; ++k) o[k] = s * kMulIn[k] + kMulPrev[k] * prev[k] - prev2[k];
      for (int k = 0; k < 3; ++k) {
        prev2[k] = prev[k];
        prev[k] = o[k];
      }
      out = (o[0] + o[1]) + o[2];
    }
    bc.th[d] = (float)out;
    bc.tl[d] = (float)(out - (double)bc.th[d]);
  }
  for (int k = 0; k < 3; ++k) {
    const double w = (2 * k + 1) * M_PI / 10.0;
    for (int m = 0; m < 20; ++m) bc.U[k][m] = (float)(std::sin((m + 1) * w) / std::sin(w));
  }
  cudaMemcpyToSymbolAsync(c_blur, &bc, sizeof(bc), 0, cudaMemcpyHostToDevice, s);
  BlurPairs bp;
  auto pair = [](float v) {
    uint32_t u;
    std::memcpy(&u, &v, 4);
    return ((unsigned long long)u << 32) | u;
  };
  for (int k = 0; k < 3; ++k) {
    bp.a[k] = pair(bc.a[k]);
    bp.b[k] = pair(bc.b[k]);
  }
  for (int d = 0; d < 5; ++d) {
    bp.th[d] = pair(bc.th[d]);
    bp.tl[d] = pair(bc.tl[d]);
    bp.nth[d] = pair(-bc.th[d]);
    bp.ntl[d] = pair(-bc.tl[d]);
  }
  for (int k = 0; k < 3; ++k)
    for (int m = 0; m < 24; ++m) bp.U[k][m] = pair(bc.U[k][m % 20]);
  bp.z = 0ull;
  cudaMemcpyToSymbolAsync(c_blur2, &bp, sizeof(bp), 0, cudaMemcpyHostToDevice, s);
}

// M_k^steps for the three resonators (row-major 2x2 acting on (o[j], o[j-1])),
// by repeated squaring in f64.
static void resonator_power(long long steps, float out[3][4]) {
  for (int k = 0; k < 3; ++k) {
    double r[4] = {1, 0, 0, 1};
    double m[4] = {kMulPrev[k], -1.0, 1.0, 0.0};
    long long e = steps;
    while (e > 0) {
      if (e & 1) {
        const double t[4] = {r[0] * m[0] + r[1] * m[2], r[0] * m[1] + r[1] * m[3],
                             r[2] * m[0] + r[3] * m[2], r[2] * m[1] + r[3] * m[3]};
        for (int i = 0; i < 4; ++i) r[i] = t[i];
      }
      const double t[4] = {m[0] * m[0] + m[1] * m[2], m[0] * m[1] + m[1] * m[3],
                           m[2] * m[0] + m[3] * m[2], m[2] * m[1] + m[3] * m[3]};
      for (int i = 0; i < 4; ++i) m[i] = t[i];
      e >>= 1;
    }
    for (int i = 0; i < 4; ++i) out[k][i] = (float)r[i];
  }
}

__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// The ripple's input at output j: what rounding added to the pair sum,
// f32(x[j-6] + x[j+4]) - (x[j-6] + x[j+4]) (two_sum's error with its sign
// turned).
__device__ __forceinline__ float pair_error(float left, float right) {
  float s, e;
  two_sum(left, right, s, e);
  return -e;
}

// ---- paired forms --------------------------------------------------------

__device__ __forceinline__ void two_sum2(f2 a, f2 b, f2& s, f2& e) {
  s = f2_add(a, b);
  const f2 bb = f2_sub(s, a);
  e = f2_add(f2_sub(a, f2_sub(s, bb)), f2_sub(b, bb));
}

// pair_error on two lanes: f32(l + r) - (l + r), i.e. two_sum's error negated
// term by term (negation commutes with rounding).
__device__ __forceinline__ f2 pair_error2(f2 l, f2 r) {
  const f2 s = f2_add(l, r);
  const f2 bb = f2_sub(s, l);
  return f2_add(f2_sub(f2_sub(s, bb), l), f2_sub(bb, r));
}

// The ripple: three resonators fed with the pair-sum rounding errors.
struct Ripple2 {
  f2 p[3], q[3];  // o[j], o[j-1]
};

__device__ __forceinline__ f2 ripple_step2(Ripple2& r, f2 e, f2 nz) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const f2 o = f2_sub(f2_add(f2_mul(e, c_blur2.a[k], nz), f2_mul(c_blur2.b[k], r.p[k], nz)),
                        r.q[k]);
    r.q[k] = r.p[k];
    r.p[k] = o;
  }
  return f2_add(f2_add(r.p[0], r.p[1]), r.p[2]);
}

// The double-float FIR on two lanes.  The low word is kept negated (cn = -c,
// exact since rounding is symmetric) so that every product error comes from
// one FMA with a negated tap: fma(-t, u, t*u rounded) = -(t*u - its rounding).
__device__ __forceinline__ f2 fir_exact2(f2 m4, f2 m3, f2 m2, f2 m1, f2 c0, f2 p1, f2 p2, f2 p3,
                                         f2 p4, f2 rip, f2 nz) {
  f2 S = f2_mul(c_blur2.th[0], c0, nz);
  f2 cn = f2_fma(c_blur2.ntl[0], c0, f2_fma(c_blur2.nth[0], c0, S));
  const f2 lo[4] = {m1, m2, m3, m4}, hi[4] = {p1, p2, p3, p4};
#pragma unroll
  for (int d = 1; d <= 4; ++d) {
    f2 u, ul;
    two_sum2(lo[d - 1], hi[d - 1], u, ul);
    const f2 p = f2_mul(c_blur2.th[d], u, nz);
    const f2 rn = f2_fma(c_blur2.nth[d], u, p);  // -(th*u - p)
    f2 q;
    two_sum2(S, p, S, q);
    cn = f2_sub(cn, q);
    cn = f2_add(cn, rn);
    cn = f2_fma(c_blur2.nth[d], ul, cn);
    cn = f2_fma(c_blur2.ntl[d], u, cn);
  }
  return f2_add(S, f2_sub(rip, cn));
}

// The homogeneous response at distance i + 1 of the entry state (p, q) =
// (o[j0-1], o[j0-2]): the sum over the resonators of U[i+1] p - U[i] q.
// `u` is the table's column i.
__device__ __forceinline__ f2 ripple_hom2(int u, const f2* ep, const f2* eq, f2 nz) {
  f2 hom = f2_sub(f2_mul(c_blur2.U[0][u + 1], ep[0], nz), f2_mul(c_blur2.U[0][u], eq[0], nz));
#pragma unroll
  for (int k = 1; k < 3; ++k)
    hom = f2_add(hom, f2_sub(f2_mul(c_blur2.U[k][u + 1], ep[k], nz),
                             f2_mul(c_blur2.U[k][u], eq[k], nz)));
  return hom;
}

// ---------------------------------------------------------------------------
// The cross-segment state of the column pass: a 64-byte header (the launch's
// epoch and the work counter), then per scale [nch][nseg][NQ][2][w] words of
// 16 bytes.  A word carries three of the six states of a column's ripple
// after the segment and, in its fourth place, the epoch it was published in:
// it is stored and loaded as one 128-bit access, so a reader that finds this
// launch's epoch has the states too, with no flag, fence or reset.  Every
// fourth place holds an epoch whatever the frame's size was, the epoch grows
// by one per launch, and the buffer starts out zeroed with epoch 0, so no
// stale word can carry the current one.
// ---------------------------------------------------------------------------

// counter: the column pass's segments handed out.  ticket: the score's CTAs
// that have finished.  Both are zeroed by the row pass of every blur, so that
// whatever an earlier call left in them (calls that raced on one buffer lose
// counts) ends with that call.
struct ScanHeader {
  uint32_t epoch, counter, ticket;
  uint32_t pad[13];
};
static_assert(sizeof(ScanHeader) == 64, "scan header");

uint32_t* blur_ticket(void* carry) { return &static_cast<ScanHeader*>(carry)->ticket; }

cudaError_t blur_disturb(void* carry, cudaStream_t s) {
  ScanHeader* const h = static_cast<ScanHeader*>(carry);
  return cudaMemsetAsync(&h->counter, 0x35, sizeof h->counter + sizeof h->ticket, s);
}

__device__ __forceinline__ void scan_store(uint4* p, float a, float b, float c, uint32_t tag) {
  const unsigned long long lo =
      ((unsigned long long)__float_as_uint(b) << 32) | __float_as_uint(a);
  const unsigned long long hi = ((unsigned long long)tag << 32) | __float_as_uint(c);
  asm volatile(
      "{\n.reg .b128 v;\nmov.b128 v, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], v;\n}" ::"l"(p),
      "l"(lo), "l"(hi)
      : "memory");
}

// True when the word carries `tag`; a, b, c receive its states.
__device__ __forceinline__ bool scan_load(const uint4* p, uint32_t tag, float* a, float* b,
                                          float* c) {
  unsigned long long lo, hi;
  asm volatile(
      "{\n.reg .b128 v;\nld.relaxed.gpu.global.b128 v, [%2];\nmov.b128 {%0, %1}, v;\n}"
      : "=l"(lo), "=l"(hi)
      : "l"(p)
      : "memory");
  *a = __uint_as_float((uint32_t)lo);
  *b = __uint_as_float((uint32_t)(lo >> 32));
  *c = __uint_as_float((uint32_t)hi);
  return (uint32_t)(hi >> 32) == tag;
}

// ---------------------------------------------------------------------------
// B1 — rows, two at a time (the lanes).
// ---------------------------------------------------------------------------

constexpr int kRowThreads = 128;  // one segment each
constexpr int kRowLevels = 7;     // log2(kRowThreads): Kogge-Stone levels
constexpr int kRowChunk = 4;      // outputs per trip of the FIR loop

struct RowScale {
  const float* x;  // [3][h][w]
  const float* r;  // [3][h][w] (NQ == 3: the reference side of r*x)
  float* out;      // [nch][NQ][h][pitch]
  int w, h, pitch, seg, pairs, first;  // pairs: row pairs; first: the scale's first CTA
  bool vec;                            // rows start on 16-byte boundaries
  f2 pw[kRowLevels][3][4];             // M_k^(seg * 2^l), as lane pairs
};
struct RowArgs {
  RowScale s[kMaxScales];
  ScanHeader* scan;
  int n, c0;
  float nz;  // -0.0f
};

// One CTA per quantity (x, x*x, r*x) of a row pair and channel: its line is
// formed once, as the samples arrive, and the five CTAs that an SM holds at
// 2048 columns are in different phases (loading, walking, scanning, FIR), so
// one's latency hides behind another's FIR.
// Bound: the FMA pipe.  A pair of outputs takes 77 paired operations of FIR,
// 20 of ripple and 13 of homogeneous response, two pipe cycles each.  A
// thread's outputs are consecutive, so four FIRs share twelve line reads.
// Measured, all scales: 2048x2048 353 -> 279 us (six launches of one 128-thread
// CTA per row pair and channel before, its three quantities one after
// another), 4096x3072 907 -> 783 us; 0.57 of the pipe's 160 and 480 us.
template <int NQ>
__global__ void __launch_bounds__(kRowThreads, 5) k_blur_rows(const __grid_constant__ RowArgs a) {
  extern __shared__ __align__(16) f2 bsm2[];
  __shared__ f2 carry[6][kRowThreads];
  const int t = threadIdx.x;
  // The column pass that follows starts a new epoch and work count, and the
  // score's end a new count of its CTAs.
  if (blockIdx.x == 0 && t == 0) {
    atomicAdd(&a.scan->epoch, 1u);
    a.scan->counter = 0;
    a.scan->ticket = 0;
  }
  int si = 0;
  while (si + 1 < a.n && (int)blockIdx.x >= a.s[si + 1].first) ++si;
  const RowScale& sc = a.s[si];
  const int w = sc.w, h = sc.h, seg = sc.seg;
  const int item = (int)blockIdx.x - sc.first;
  // quantity q: 0 x, 1 x*x, 2 r*x
  const int q = item % NQ, chp = item / NQ;
  const int ch = chp / sc.pairs, y0 = 2 * (chp - ch * sc.pairs), c = a.c0 + ch;
  const bool two = y0 + 1 < h;
  f2* const xl = bsm2;                      // the line at i - 10, both rows
  f2* const rip = bsm2 + ((w + 21) & ~1);   // [pitch]: the ripple, then the outputs
  const size_t n = (size_t)w * h;
  const f2 nz = f2_pack(a.nz, a.nz);
  {
    const float* x0 = sc.x + n * c + (size_t)y0 * w;
    const float* x1 = two ? x0 + w : x0;
    const bool other = NQ == 3 && q == 2;
    const float* r0 = (other ? sc.r : sc.x) + n * c + (size_t)y0 * w;
    const float* r1 = two ? r0 + w : r0;
    auto put = [&](float a0, float a1, float b0, float b1, f2& dst) {
      const f2 v = f2_pack(a0, a1);
      dst = q == 0 ? v : f2_mul(f2_pack(b0, b1), v, nz);
    };
    if (t < 20) xl[t < 10 ? t : w + t] = 0ull;  // zero outside the line
    if (sc.vec) {
      // 16-byte loads, up to eight in flight per thread.
      auto put4 = [&](int i, float4 a0, float4 a1, float4 b0, float4 b1) {
        f2* d = xl + i + 10;
        put(a0.x, a1.x, b0.x, b1.x, d[0]);
        put(a0.y, a1.y, b0.y, b1.y, d[1]);
        put(a0.z, a1.z, b0.z, b1.z, d[2]);
        put(a0.w, a1.w, b0.w, b1.w, d[3]);
      };
      auto ld4 = [](const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); };
      const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (!other) {
#pragma unroll 4
        for (int i = 4 * t; i < w; i += 4 * kRowThreads) {
          const float4 v0 = ld4(x0 + i), v1 = two ? ld4(x1 + i) : zero;
          put4(i, v0, v1, v0, v1);
        }
      } else {
#pragma unroll 2
        for (int i = 4 * t; i < w; i += 4 * kRowThreads)
          put4(i, ld4(x0 + i), two ? ld4(x1 + i) : zero, ld4(r0 + i), two ? ld4(r1 + i) : zero);
      }
    } else if (!other) {
#pragma unroll 8
      for (int i = t; i < w; i += kRowThreads) {
        const float v0 = __ldg(x0 + i), v1 = two ? __ldg(x1 + i) : 0.0f;
        put(v0, v1, v0, v1, xl[i + 10]);
      }
    } else {
#pragma unroll 4
      for (int i = t; i < w; i += kRowThreads)
        put(__ldg(x0 + i), two ? __ldg(x1 + i) : 0.0f, __ldg(r0 + i), two ? __ldg(r1 + i) : 0.0f,
            xl[i + 10]);
    }
  }
  __syncthreads();
  const int j0 = min(t * seg, w), j1 = min(j0 + seg, w);
  // (1) the segment's ripple from rest, recorded.
  Ripple2 rp;
#pragma unroll
  for (int k = 0; k < 3; ++k) rp.p[k] = rp.q[k] = 0ull;
  // blur.rs:414 starts the recursion four samples before the line, fed
  // with 0 + x[0..3]: no rounding, so no ripple, for finite samples, and
  // NaN through the whole line for a non-finite one.
  if (t == 0)
#pragma unroll 1
    for (int j = -4; j < 0; ++j) ripple_step2(rp, pair_error2(xl[j + 4], xl[j + 14]), nz);
#pragma unroll 4
  for (int j = j0; j < j1; ++j) rip[j] = ripple_step2(rp, pair_error2(xl[j + 4], xl[j + 14]), nz);
  // (2) inclusive scan over segments: S_t = sum_{u <= t} A^(t-u) B_u, per lane
  // of the pairs and per resonator.  Warp k scans resonator k by itself, a
  // lane holding segments lane + 32 m, so no level needs a barrier.
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    carry[2 * k][t] = rp.p[k];
    carry[2 * k + 1][t] = rp.q[k];
  }
  __syncthreads();
  if (t < 96) {
    const int k = t >> 5, lane = t & 31;
    const unsigned full = 0xffffffffu;
    const int live = (w + seg - 1) / seg;  // segments with samples
    f2 p[4], qv[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      p[m] = carry[2 * k][lane + 32 * m];
      qv[m] = carry[2 * k + 1][lane + 32 * m];
    }
    auto level = [&](int l, const f2* op, const f2* oq, auto from) {
      const f2 m0 = sc.pw[l][k][0], m1 = sc.pw[l][k][1], m2 = sc.pw[l][k][2],
               m3 = sc.pw[l][k][3];
#pragma unroll
      for (int m = 0; m < 4; ++m)
        if (from(m)) {
          p[m] = f2_add(p[m], f2_add(f2_mul(m0, op[m], nz), f2_mul(m1, oq[m], nz)));
          qv[m] = f2_add(qv[m], f2_add(f2_mul(m2, op[m], nz), f2_mul(m3, oq[m], nz)));
        }
    };
#pragma unroll 1
    for (int l = 0; l < 5 && (1 << l) < live; ++l) {
      const int d = 1 << l, src = (lane - d) & 31;
      f2 op[4], oq[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        op[m] = __shfl_sync(full, p[m], src);
        oq[m] = __shfl_sync(full, qv[m], src);
      }
      if (lane < d)
#pragma unroll
        for (int m = 3; m >= 1; --m) {
          op[m] = op[m - 1];
          oq[m] = oq[m - 1];
        }
      level(l, op, oq, [&](int m) { return m > 0 || lane >= d; });
    }
    if (live > 32) {
      const f2 op[4] = {0, p[0], p[1], p[2]}, oq[4] = {0, qv[0], qv[1], qv[2]};
      level(5, op, oq, [](int m) { return m >= 1; });
    }
    if (live > 64) {
      const f2 op[4] = {0, 0, p[0], p[1]}, oq[4] = {0, 0, qv[0], qv[1]};
      level(6, op, oq, [](int m) { return m >= 2; });
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      carry[2 * k][lane + 32 * m] = p[m];
      carry[2 * k + 1][lane + 32 * m] = qv[m];
    }
  }
  __syncthreads();
  // (3) the outputs of the thread's own samples: the ripple is its
  // response from rest plus the entry state's homogeneous response.
  f2 ep[3] = {0, 0, 0}, eq[3] = {0, 0, 0};
  if (t > 0)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      ep[k] = carry[2 * k][t - 1];
      eq[k] = carry[2 * k + 1][t - 1];
    }
  auto ripple = [&](int j, int u) -> f2 {
    const f2 r = rip[j];
    return t > 0 ? f2_add(r, ripple_hom2(u, ep, eq, nz)) : r;
  };
  int j = j0, u = 0;  // u: (j - j0) mod 20
#pragma unroll 1
  for (; j + kRowChunk <= j1; j += kRowChunk) {
    f2 v[kRowChunk + 8];
#pragma unroll
    for (int i = 0; i < kRowChunk + 8; ++i) v[i] = xl[j + 6 + i];
#pragma unroll
    for (int m = 0; m < kRowChunk; ++m)
      rip[j + m] = fir_exact2(v[m], v[m + 1], v[m + 2], v[m + 3], v[m + 4], v[m + 5], v[m + 6],
                              v[m + 7], v[m + 8], ripple(j + m, u + m), nz);
    u = u + kRowChunk >= 20 ? u + kRowChunk - 20 : u + kRowChunk;
  }
#pragma unroll 1
  for (; j < j1; ++j) {
    f2 v[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) v[i] = xl[j + 6 + i];
    rip[j] = fir_exact2(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], ripple(j, u), nz);
    u = u + 1 >= 20 ? 0 : u + 1;
  }
  __syncthreads();
  // (4) both rows to memory, four columns at a time (rows of `out` are
  // 16-byte aligned; the columns past w are padding nobody reads).
  float* o0 = sc.out + ((size_t)(ch * NQ + q) * h + y0) * sc.pitch;
  for (int i = 4 * t; i < w; i += 4 * kRowThreads) {
    const ulonglong2 u0 = *reinterpret_cast<const ulonglong2*>(rip + i);
    const ulonglong2 u1 = *reinterpret_cast<const ulonglong2*>(rip + i + 2);
    *reinterpret_cast<float4*>(o0 + i) =
        make_float4(f2_lo(u0.x), f2_lo(u0.y), f2_lo(u1.x), f2_lo(u1.y));
    if (two)
      *reinterpret_cast<float4*>(o0 + sc.pitch + i) =
          make_float4(f2_hi(u0.x), f2_hi(u0.y), f2_hi(u1.x), f2_hi(u1.y));
  }
}

// ---------------------------------------------------------------------------
// B2 — columns (and the candidate's per-pixel terms).
// ---------------------------------------------------------------------------

constexpr int kColW = 32;            // columns per strip
constexpr int kTileH = 32;           // rows per output tile (one row of partial sums)
constexpr int kColT = 2 * kTileH;    // rows per segment
constexpr int kQuarter = kColT / 4;  // rows per ripple walk
constexpr int kColThreads = 256;
constexpr uint32_t kColWaitLimit = 1u << 20;  // polls of a predecessor's words (about a second)

struct ColScale {
  const float* hpl;  // [nch][NQ][h][pitch] row-pass planes
  uint4* states;     // [nch][nseg][NQ][2][w] published states
  float* mu;         // NQ == 2: [3][h][w] outputs
  float* s11;
  const float* mu1;  // NQ == 3: reference mu, sigma11, positive XYB; candidate XYB
  const float* s11r;
  const float* rx;
  const float* cx;
  DF* partial;  // NQ == 3: [tile rows][strips][18]
  int w, h, pitch, nseg, strips, first;
};
struct ColArgs {
  ColScale s[kMaxScales];
  ScanHeader* scan;
  uint32_t* err;  // the context's device error word
  int n, c0, nch, items;  // items: segments of all scales
  float nz;
  float pw[3][4];  // M_k^kTileH
};

template <int NQ>
struct ColSmem {
  float tile[NQ][kColT + 10][kColW];  // rows r0-6 .. r0+kColT+3
  float rp[NQ][kColT][kColW];         // the ripple from rest, a quarter at a time
  // Each quarter's end state from rest; once the segment's entry is known,
  // each quarter's entry state (read by the outputs as lane pairs).
  float state[4][NQ][6][kColW];
  DF red[2][kColThreads / 32][6];
  int item;
};

// Reduces six double-float sums over the 16 lanes of a half warp in the
// order of an xor butterfly (distances 8, 4, 2, 1; df_add is symmetric), each
// step handing half of the remaining quantities to the partner lane: seven
// additions instead of six butterflies' twenty-four.  Returns this lane's
// total; *k is its quantity.
__device__ __forceinline__ DF half_warp_sum6(DF* v, int lane, int* k) {
  const unsigned full = 0xffffffffu;
  auto swap = [&](DF x, int o) {
    return DF{__shfl_xor_sync(full, x.hi, o), __shfl_xor_sync(full, x.lo, o)};
  };
  const bool h8 = lane & 8, h4 = lane & 4, h2 = lane & 2;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const DF keep = h8 ? v[i + 3] : v[i], send = h8 ? v[i] : v[i + 3];
    v[i] = df_add(keep, swap(send, 8));
  }
  const DF keep = h4 ? v[2] : v[0], send = h4 ? v[0] : v[2];
  const DF w0 = df_add(keep, swap(send, 4));
  const DF w1 = df_add(v[1], swap(v[1], 4));
  DF x = df_add(h2 ? w1 : w0, swap(h2 ? w0 : w1, 2));
  x = df_add(x, swap(x, 1));
  *k = (h8 ? 3 : 0) + (h2 ? 1 : (h4 ? 2 : 0));
  return x;
}

// Bound: the FMA pipe, as the row pass (the same FIR and ripple), plus the
// per-pixel terms.  A 64-row segment reads 74 rows for its 64 (42 for 32
// before), a strip's chain has half the links, a link is one 128-bit word per
// column instead of a flag behind fences and barriers, the walks and FIRs run
// on column pairs, and four consecutive rows a thread share twelve tile reads
// and their quarter's entry states.
// The planes read only by the terms are prefetched into L2 by the CTA that
// will read them (294 -> 283 us).
// Measured, all scales: 2048x2048 470 -> 283 us (six launches of 32-row
// segments before: the 1024-column scale alone took 91 us, 32 links of a
// chain at 2.8 us each), 4096x3072 1157 -> 804 us.
template <int NQ>
__global__ void __launch_bounds__(kColThreads, 3) k_blur_cols(const __grid_constant__ ColArgs a) {
  extern __shared__ __align__(16) unsigned char col_smem[];
  ColSmem<NQ>& sm = *reinterpret_cast<ColSmem<NQ>*>(col_smem);
  const int t = threadIdx.x;
  // Items in the order CTAs start (segments slowest within a scale), so that
  // the segment a CTA waits for belongs to a CTA that has already started.
  if (t == 0) sm.item = (int)atomicAdd(&a.scan->counter, 1u);
  const uint32_t epoch = a.scan->epoch;
  __syncthreads();
  const int gitem = sm.item;
  // A count past the last segment: another call runs on this buffer at the
  // same time.  The scores are spoilt, the accesses stay inside it.
  if (gitem >= a.items) return;
  int si = 0;
  while (si + 1 < a.n && gitem >= a.s[si + 1].first) ++si;
  const ColScale& sc = a.s[si];
  const int w = sc.w, h = sc.h;
  const int item = gitem - sc.first, per_sg = sc.strips * a.nch;
  const int sg = item / per_sg, ch = (item - sg * per_sg) / sc.strips, sx = item % sc.strips;
  const int c = a.c0 + ch;
  const int x0 = sx * kColW, r0 = sg * kColT;
  const size_t n = (size_t)w * h;
  if (NQ == 3) {
    // The reference's and the candidate's planes, read only at the end, on
    // their way from memory meanwhile.
    static_assert(kColThreads == 4 * kColT, "one 128-byte line per thread");
    const int k = t & 3, gy = r0 + (t >> 2);
    const float* src = k == 0 ? sc.mu1 : (k == 1 ? sc.s11r : (k == 2 ? sc.rx : sc.cx));
    if (gy < h) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + (size_t)c * n + (size_t)gy * w + x0));
  }
  {
    // 16 bytes at a time (rows of the planes are padded to 16-byte pitch);
    // rows outside the plane and columns past the pitch read as zero.
    const float* H = sc.hpl + (size_t)ch * NQ * h * sc.pitch;
    constexpr int kVec = kColW / 4;
    for (int i = t; i < NQ * (kColT + 10) * kVec; i += kColThreads) {
      const int vx = i % kVec, ly = (i / kVec) % (kColT + 10), q = i / (kVec * (kColT + 10));
      const int gy = r0 - 6 + ly, gx = x0 + 4 * vx;
      const bool in = gy >= 0 && gy < h && gx < sc.pitch;
      const float* src = H + ((size_t)q * h + (in ? gy : 0)) * sc.pitch + (in ? gx : 0);
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sm.tile[q][ly][4 * vx]);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
                   "r"(in ? 16 : 0)
                   : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  __syncthreads();
  const f2 nz = f2_pack(a.nz, a.nz);
  // The ripple in four quarters per column pair and quantity: each quarter
  // walks from rest, recording R from rest and its end state.
  if (t < 4 * NQ * (kColW / 2)) {
    const int wx = 2 * (t % (kColW / 2)), wq = (t / (kColW / 2)) % NQ, wh = t / (NQ * (kColW / 2));
    Ripple2 st;
#pragma unroll
    for (int k = 0; k < 3; ++k) st.p[k] = st.q[k] = 0ull;
    auto at = [&](int r) { return *reinterpret_cast<const f2*>(&sm.tile[wq][r][wx]); };
#pragma unroll 8
    for (int r = wh * kQuarter; r < (wh + 1) * kQuarter; ++r)
      *reinterpret_cast<f2*>(&sm.rp[wq][r][wx]) =
          ripple_step2(st, pair_error2(at(r), at(r + 10)), nz);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      *reinterpret_cast<f2*>(&sm.state[wh][wq][2 * k][wx]) = st.p[k];
      *reinterpret_cast<f2*>(&sm.state[wh][wq][2 * k + 1][wx]) = st.q[k];
    }
  }
  __syncthreads();
  // The chained scan over the column's segments, one thread per column and
  // quantity: the entry state is the previous segment's inclusive state (for
  // the first segment, the state blur.rs:574 reaches over its four warm-up
  // rows, fed with 0 + rows 0..3: zero ripple for finite samples).  A tile of
  // 32 rows takes its entry through M^kTileH plus its own response from rest,
  // M^kQuarter times its first quarter's end state plus its second's.  Every
  // wait is bounded; one that runs out raises kDevBlurTimeout.
  if (t < NQ * kColW) {
    const int sq = t / kColW, sl = t % kColW, sxc = x0 + sl;
    float p1[2][3], q1[2][3], bp[2][3], bq[2][3];
    float u0[3], u1[3], u2[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      u0[k] = c_blur.U[k][kQuarter % 20];
      u1[k] = c_blur.U[k][(kQuarter - 1) % 20];
      u2[k] = c_blur.U[k][(kQuarter - 2) % 20];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        p1[i][k] = sm.state[2 * i][sq][2 * k][sl];
        q1[i][k] = sm.state[2 * i][sq][2 * k + 1][sl];
        bp[i][k] = (u0[k] * p1[i][k] - u1[k] * q1[i][k]) + sm.state[2 * i + 1][sq][2 * k][sl];
        bq[i][k] = (u1[k] * p1[i][k] - u2[k] * q1[i][k]) + sm.state[2 * i + 1][sq][2 * k + 1][sl];
      }
    }
    const bool live = sxc < w;
    uint4* const mine =
        sc.states + (((size_t)(ch * sc.nseg + sg) * NQ + sq) * 2) * w + (live ? sxc : 0);
    float sp[3] = {0.0f, 0.0f, 0.0f}, sqq[3] = {0.0f, 0.0f, 0.0f};
    if (sg == 0) {
#pragma unroll
      for (int k = 0; k < 3; ++k)
        for (int i = 0; i < 4 && i < h; ++i) {
          const float e = pair_error(0.0f, sm.tile[sq][6 + i][sl]);
          const float o = (e * c_blur.a[k] + c_blur.b[k] * sp[k]) - sqq[k];
          sqq[k] = sp[k];
          sp[k] = o;
        }
    } else if (live) {
      const uint4* prev = mine - (size_t)NQ * 2 * w;
      bool got = false;
      for (uint32_t it = 0; it < kColWaitLimit; ++it) {
        const bool g0 = scan_load(prev, epoch, &sp[0], &sqq[0], &sp[1]);
        const bool g1 = scan_load(prev + w, epoch, &sqq[1], &sp[2], &sqq[2]);
        got = g0 && g1;
        if (got) break;
        __nanosleep(20);
      }
      if (!got) {
        raise_error(a.err, kDevBlurTimeout);
#pragma unroll
        for (int k = 0; k < 3; ++k) sp[k] = sqq[k] = 0.0f;
      }
    }
    // inclusive states after the segment's two tiles
    float ip[2][3], iq[2][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float* m = a.pw[k];
      ip[0][k] = (m[0] * sp[k] + m[1] * sqq[k]) + bp[0][k];
      iq[0][k] = (m[2] * sp[k] + m[3] * sqq[k]) + bq[0][k];
      ip[1][k] = (m[0] * ip[0][k] + m[1] * iq[0][k]) + bp[1][k];
      iq[1][k] = (m[2] * ip[0][k] + m[3] * iq[0][k]) + bq[1][k];
    }
    if (live) {
      scan_store(mine, ip[1][0], iq[1][0], ip[1][1], epoch);
      scan_store(mine + w, iq[1][1], ip[1][2], iq[1][2], epoch);
    }
    // Each quarter's entry state: its tile's entry for the first quarter,
    // M^kQuarter times it plus the first quarter's end state for the second.
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float ep = i == 0 ? sp[k] : ip[0][k], eq = i == 0 ? sqq[k] : iq[0][k];
        sm.state[2 * i][sq][2 * k][sl] = ep;
        sm.state[2 * i][sq][2 * k + 1][sl] = eq;
        sm.state[2 * i + 1][sq][2 * k][sl] = (u0[k] * ep - u1[k] * eq) + p1[i][k];
        sm.state[2 * i + 1][sq][2 * k + 1][sl] = (u1[k] * ep - u2[k] * eq) + q1[i][k];
      }
  }
  __syncthreads();
  // Outputs: columns 2j, 2j+1 (the lanes) of four rows.  A warp's two halves
  // take the same rows of two quarters, so that both read one U entry.
  const int lane = t & 31, warp = t >> 5;
  const int jp = lane & 15, quarter = 2 * (warp >> 2) + (lane >> 4), ir = 4 * (warp & 3);
  const int rr = quarter * kQuarter + ir;
  const int lx = 2 * jp, gx = x0 + lx;
  const bool pairs = (w & 1) == 0;  // rows of the w-pitched planes hold aligned pairs
  f2 val[NQ][4];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    f2 v[12], ep[3], eq[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      ep[k] = *reinterpret_cast<const f2*>(&sm.state[quarter][q][2 * k][lx]);
      eq[k] = *reinterpret_cast<const f2*>(&sm.state[quarter][q][2 * k + 1][lx]);
    }
#pragma unroll
    for (int i = 0; i < 12; ++i) v[i] = *reinterpret_cast<const f2*>(&sm.tile[q][rr + 2 + i][lx]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const f2 rip = f2_add(*reinterpret_cast<const f2*>(&sm.rp[q][rr + i][lx]),
                            ripple_hom2(ir + i, ep, eq, nz));
      val[q][i] = fir_exact2(v[i], v[i + 1], v[i + 2], v[i + 3], v[i + 4], v[i + 5], v[i + 6],
                             v[i + 7], v[i + 8], rip, nz);
    }
  }
  // Partial sums: each thread's rows in pairs, then lanes and warps in
  // double-float, in one fixed order.
  DF acc2[6];
#pragma unroll
  for (int hr = 0; hr < 2; ++hr) {
    float acc[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int i = 2 * hr; i < 2 * hr + 2; ++i) {
      const int gy = r0 + rr + i;
      if (gy >= h || gx >= w) continue;
      const bool second = gx + 1 < w;
      const size_t p = (size_t)c * n + (size_t)gy * w + gx;
      if (NQ == 2) {
        if (pairs) {
          *reinterpret_cast<f2*>(sc.mu + p) = val[0][i];
          *reinterpret_cast<f2*>(sc.s11 + p) = val[1][i];
        } else {
          sc.mu[p] = f2_lo(val[0][i]);
          sc.s11[p] = f2_lo(val[1][i]);
          if (second) {
            sc.mu[p + 1] = f2_hi(val[0][i]);
            sc.s11[p + 1] = f2_hi(val[1][i]);
          }
        }
      } else {
        float pf[4][2];
        const float* src[4] = {sc.mu1, sc.s11r, sc.rx, sc.cx};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (pairs) {
            const float2 v2 = __ldg(reinterpret_cast<const float2*>(src[k] + p));
            pf[k][0] = v2.x;
            pf[k][1] = v2.y;
          } else {
            pf[k][0] = __ldg(src[k] + p);
            pf[k][1] = second ? __ldg(src[k] + p + 1) : 0.0f;
          }
        }
        // pool.rs:248 accumulate_scalar, in the reference's operation order.
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (e == 1 && !second) break;
          const float m1 = pf[0][e];
          const float m2 = e ? f2_hi(val[0][i]) : f2_lo(val[0][i]);
          const float v11 = pf[1][e];
          const float s22 = e ? f2_hi(val[1][i]) : f2_lo(val[1][i]);
          const float s12 = e ? f2_hi(val[NQ - 1][i]) : f2_lo(val[NQ - 1][i]);
          const float mu11 = m1 * m1, mu22 = m2 * m2, mu12 = m1 * m2;
          const float md = m1 - m2;
          const float num_m = 1.0f - md * md;
          const float num_s = 2.0f * (s12 - mu12) + 0.0009f;
          const float den_s = (v11 - mu11) + (s22 - mu22) + 0.0009f;
          const float d = fmaxf(1.0f - (num_m * num_s) / den_s, 0.0f);
          const float d2 = d * d;
          // (1 + |i2-m2|) / (1 + |i1-m1|) - 1 as a difference over the
          // denominator (within the 0.01-point contract the fast division, at
          // most 2 ulp off, serves; identical images give a zero numerator).
          const float a1 = fabsf(pf[2][e] - m1), a2 = fabsf(pf[3][e] - m2);
          const float d1 = __fdividef(a2 - a1, 1.0f + a1);
          const float art = fmaxf(d1, 0.0f), lost = fmaxf(-d1, 0.0f);
          const float art2 = art * art, lost2 = lost * lost;
          acc[0] += d;
          acc[1] += d2 * d2;
          acc[2] += art;
          acc[3] += art2 * art2;
          acc[4] += lost;
          acc[5] += lost2 * lost2;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const DF v{acc[k], 0.0f};
      acc2[k] = hr == 0 ? v : df_add(acc2[k], v);
    }
  }
  if (NQ == 3) {
    int k;
    const DF tot = half_warp_sum6(acc2, lane, &k);
    // the four rows' place among its tile's eight
    const int tl = quarter >> 1, slot = 4 * (quarter & 1) + (warp & 3);
    if ((lane & 1) == 0) sm.red[tl][slot][k] = tot;
    __syncthreads();
    const int tr = 2 * sg + t / 6;
    if (t < 12 && tr * kTileH < h) {
      DF s = sm.red[t / 6][0][t % 6];
      for (int i = 1; i < kColThreads / 32; ++i) s = df_add(s, sm.red[t / 6][i][t % 6]);
      sc.partial[((size_t)tr * sc.strips + sx) * 18 + c * 6 + t % 6] = s;
    }
  }
}

// ---------------------------------------------------------------------------
// Launches.
// ---------------------------------------------------------------------------

namespace {

int row_seg(int w) {
  int seg = (w + kRowThreads - 1) / kRowThreads;
  return seg | 1;  // odd: the threads' shared-memory strides fall on distinct banks
}

int blur_pitch(int w) { return (w + 3) & ~3; }

f2 lane_pair(float v) {
  uint32_t u;
  std::memcpy(&u, &v, 4);
  return ((unsigned long long)u << 32) | u;
}

// Bytes of the row pass's line and ripple.
size_t row_smem(int w) { return ((size_t)((w + 21) & ~1) + blur_pitch(w)) * sizeof(f2); }

// Rows of scales [0, n), then their columns.
template <int NQ>
void launch_blur(const BlurScale* scales, int n, int c0, int nch, float* hpl, void* carry,
                 uint32_t* err, cudaStream_t s, ScaleHook hook, void* user) {
  RowArgs ra;
  ColArgs ca;
  ra.scan = ca.scan = static_cast<ScanHeader*>(carry);
  ra.n = ca.n = n;
  ra.c0 = ca.c0 = c0;
  ra.nz = ca.nz = -0.0f;
  ca.nch = nch;
  ca.err = err;
  resonator_power(kTileH, ca.pw);
  uint4* states = reinterpret_cast<uint4*>(ca.scan + 1);
  int rows = 0, cols = 0;
  for (int i = 0; i < n; ++i) {
    const BlurScale& b = scales[i];
    RowScale& r = ra.s[i];
    ColScale& c = ca.s[i];
    r.x = b.x;
    r.r = b.r;
    r.out = hpl;
    r.w = c.w = b.w;
    r.h = c.h = b.h;
    r.pitch = c.pitch = blur_pitch(b.w);
    r.seg = row_seg(b.w);
    r.pairs = (b.h + 1) / 2;
    r.first = rows;
    r.vec = b.w % 4 == 0 && ((uintptr_t)b.x & 15) == 0 && ((uintptr_t)b.r & 15) == 0;
    rows += r.pairs * nch * NQ;
    for (int l = 0; l < kRowLevels; ++l) {
      float m[3][4];
      resonator_power((long long)r.seg << l, m);
      for (int k = 0; k < 3; ++k)
        for (int e = 0; e < 4; ++e) r.pw[l][k][e] = lane_pair(m[k][e]);
    }
    c.hpl = hpl;
    hpl += (size_t)nch * NQ * r.pitch * b.h;
    c.states = states;
    c.mu = b.mu;
    c.s11 = b.s11;
    c.mu1 = b.mu;
    c.s11r = b.s11;
    c.rx = b.r;
    c.cx = b.x;
    c.partial = b.partial;
    c.nseg = (b.h + kColT - 1) / kColT;
    c.strips = (b.w + kColW - 1) / kColW;
    c.first = cols;
    cols += c.strips * c.nseg * nch;
    states += (size_t)nch * c.nseg * NQ * 2 * b.w;
  }
  ca.items = cols;
  if (hook) hook(user, 0);
  // scale 0 has the longest lines
  k_blur_rows<NQ><<<rows, kRowThreads, row_smem(scales[0].w), s>>>(ra);
  if (hook) hook(user, 1);
  if (hook) hook(user, 2);
  k_blur_cols<NQ><<<cols, kColThreads, sizeof(ColSmem<NQ>), s>>>(ca);
  if (hook) hook(user, 3);
}

template <typename F>
cudaError_t allow_smem(F* kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace

cudaError_t configure_blur_kernels() {
  cudaError_t e;
  if ((e = allow_smem(k_blur_rows<2>, row_smem(kBlurMaxWidth))) != cudaSuccess) return e;
  if ((e = allow_smem(k_blur_rows<3>, row_smem(kBlurMaxWidth))) != cudaSuccess) return e;
  if ((e = allow_smem(k_blur_cols<2>, sizeof(ColSmem<2>))) != cudaSuccess) return e;
  return allow_smem(k_blur_cols<3>, sizeof(ColSmem<3>));
}

int blur_partial_rows(int w, int h) {
  return ((w + kColW - 1) / kColW) * ((h + kTileH - 1) / kTileH);
}

size_t blur_plane_floats(int w, int h) { return (size_t)blur_pitch(w) * h; }

size_t blur_carry_bytes(int w, int h, int nch) {
  return (size_t)nch * ((h + kColT - 1) / kColT) * 3 * 2 * w * sizeof(uint4);
}

void launch_ref_moments(const BlurScale* scales, int n, float* hpl, void* carry, uint32_t* err,
                        cudaStream_t s) {
  launch_blur<2>(scales, n, 0, 3, hpl, carry, err, s, nullptr, nullptr);
}

int launch_score_scales(const BlurScale* scales, int n, int c0, int nch, float* hpl, void* carry,
                        uint32_t* err, cudaStream_t s, ScaleHook hook, void* user) {
  launch_blur<3>(scales, n, c0, nch, hpl, carry, err, s, hook, user);
  return 2;
}

}  // namespace jpxlg
