// k_encode.cu — sm_103a kernels of the encoder's transform path:
//   K1 k_srgb_to_xyb       RGB8/RGB16 -> LUT -> linear -> XYB planes
//   K2 k_precondition      12 fused Jacobi steps of the inverse Gaborish
//   K3 k_fdct8, k_fdct_sq<N>  gather + DCT_2D + LF samples + luma quantization
//   K4 k_cfl_*             chroma-from-luma factor estimation, and with it
//   K5                     X/B quantization against reconstructed luma
// Each kernel restates the reference arithmetic it replaces (cited per
// kernel) in the reference's operation order; the build uses -fmad=false.
#include <algorithm>
#include <cstdint>
#include <cstring>

#include "jpxlg_common.cuh"
#include "jpxlg_internal.h"
#include "jpxlg_kernels.h"
#include "jpxlg_quant.cuh"

namespace jpxlg {

__constant__ float c_iv4[16];
__constant__ float c_iv8[64];
__constant__ float c_iv16[256];
__constant__ float c_scale_f[32];  // [lf count 1,2,4,8][c < 8]

// ---------------------------------------------------------------------------
// K1 — jpxl-encode-policy source.rs:226 (RGB8) / :355 (RGB16): code point ->
// linear through the host-built table, then jpxl-core color.rs:84 opsin mix
// (no FMA), reproducible cube root, opponent rotation.
// ---------------------------------------------------------------------------

__device__ __forceinline__ void xyb_of(float r, float g, float b, float* x, float* y, float* s) {
  float lm = 0.3f * r + 0.622f * g + 0.078f * b + 0.0037930734f;
  float mm = 0.23f * r + 0.692f * g + 0.078f * b + 0.0037930734f;
  float sm = 0.2434227f * r + 0.2047674f * g + 0.5518099f * b + 0.0037930734f;
  float lg = cbrt_core(lm) - 0.1559542f;
  float mg = cbrt_core(mm) - 0.1559542f;
  float sg = cbrt_core(sm) - 0.1559542f;
  *x = 0.5f * (lg - mg);
  *y = 0.5f * (lg + mg);
  *s = sg;
}

// Bound: the latency of the reads and the table (32 registers, so that eight
// CTAs cover it).  A byte image's table is copied to shared memory, a deeper
// one's is read in memory (a byte per code point beside the curve, in shared
// memory, measured 38 us against 40 at 2048x2048 and was not kept).
// Measured: 4096x3072 16-bit 122 -> 79 us, 2048x2048 45.5 -> 34.
template <typename T>
__global__ void __launch_bounds__(256, 8) k_srgb_to_xyb(const T* __restrict__ rgb, size_t n,
                                                     const float* __restrict__ lut,
                                                     float* __restrict__ px,
                                                     float* __restrict__ py,
                                                     float* __restrict__ pb,
                                                     uint32_t* __restrict__ not_gray,
                                                     uint32_t global_scale,
                                                     float* __restrict__ mul_table) {
  constexpr bool kByte = sizeof(T) == 1;
  // The transform's table of HF multipliers, where it follows: the last CTA's
  // threads, beside its pixels (a launch of its own cost 2.9 us).
  if (mul_table && blockIdx.x == gridDim.x - 1) fill_mul_table(global_scale, mul_table);
  __shared__ float slut[kByte ? 256 : 1];
  if (kByte) {
    slut[threadIdx.x] = __ldg(lut + threadIdx.x);
    __syncthreads();
  }
  auto light = [&](uint32_t code) { return kByte ? slut[code] : __ldg(&lut[code]); };
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  bool color = false;
#pragma unroll 2
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    uint32_t cr = rgb[3 * i], cg = rgb[3 * i + 1], cb = rgb[3 * i + 2];
    color |= (cr != cg) || (cg != cb);
    float x, y, b;
    xyb_of(light(cr), light(cg), light(cb), &x, &y, &b);
    px[i] = x;
    py[i] = y;
    pb[i] = b;
  }
  if (__any_sync(0xffffffffu, color) && (threadIdx.x & 31) == 0) atomicOr(not_gray, 1u);
}

void launch_srgb_to_xyb(const void* rgb, int bits, size_t n, const float* lut, float* x, float* y,
                        float* b, uint32_t* not_gray, uint32_t global_scale, float* mul_table,
                        int num_sms, cudaStream_t s) {
  const int blocks = (int)std::max<size_t>(
      1, std::min<size_t>((n + 255) / 256, (size_t)num_sms * 16));
  if (bits == 8)
    k_srgb_to_xyb<uint8_t><<<blocks, 256, 0, s>>>((const uint8_t*)rgb, n, lut, x, y, b, not_gray,
                                                  global_scale, mul_table);
  else
    k_srgb_to_xyb<uint16_t><<<blocks, 256, 0, s>>>((const uint16_t*)rgb, n, lut, x, y, b,
                                                   not_gray, global_scale, mul_table);
}

// ---------------------------------------------------------------------------
// K2 — jpxl-encode vardct/gaborish.rs:218 precondition_xyb_planes: twelve
// Jacobi steps x <- x + (f - Kx) * (1/centre) (tail: / centre) against the
// encoder's non-FMA J.1 kernel.  All twelve steps run on one register-resident
// tile with a 12-sample halo, so the plane is read once and written once.
//
// Bit parity with the reference's position-dependent arithmetic:
//   * a pixel on the frame border sums its nine mirrored taps sequentially
//     (dy outer, dx inner), acc += w*s;
//   * an interior pixel in the SIMD groups of four that start at x = 1
//     (x - 1 < 4*floor((w-2)/4)) evaluates mid*c + (N+S+W+E)*e + (NW+NE+SW+SE)*k;
//   * remaining interior pixels sum the nine taps sequentially;
//   * the update multiplies by 1/centre for flat indices below 4*floor(n/4)
//     and divides by centre above.
// Border cells read their taps at mirrored frame coordinates, so no cell
// outside the frame is ever read after the load.
// ---------------------------------------------------------------------------

// Tiling.  A CTA owns a 128 x 128 tile of one plane with a 12-sample halo
// (104 x 104 outputs).  Lane l of warp v holds columns 4l .. 4l+3 of tile
// rows 8v .. 8v+7, and the source plane's, in registers for all twelve
// steps: west and east neighbours come from the adjacent lanes by shuffle,
// the rows above and below the warp's eight from the neighbouring warps
// through shared memory (double-buffered, one barrier per step).  Bound by
// the issue of its sums and products; sixteen warps of eight rows against
// thirty-two of four keep the source plane out of shared memory and halve
// the exchanged rows (4096 x 3072: 452 us, then 433; a wider choice of
// barriers, pairs of warps or rows at rest, gained nothing).  Every step updates the whole tile; a cell k samples from
// the tile's edge is exact for k steps, so after twelve the inner 104 x 104
// are, and no cell of the edge ring is ever read by one nearer the centre
// than itself.
//
// Two kinds of tile cover a frame: those whose haloed extent has no cell of
// another rule (kEdge false), and the ring of tiles around them (kEdge
// true).  A ring tile keeps each step's input in shared memory and, after
// the paired update of every cell, the CTA's threads share out the cells of
// another rule (frame border and columns past the groups of four: the
// sequential nine-tap sum; the last n % 4 cells of the plane: the division
// by the centre weight) and recompute them from their nine taps at mirrored
// frame coordinates (always among the cell's own 3 x 3 neighbourhood).  One
// launch holds both: the ring's CTAs first (they take longer), then the
// interior's, which fill the SMs around them.
constexpr int kPreOut = 104;                   // outputs across
constexpr int kPreHalo = 12;
constexpr int kPreW = kPreOut + 2 * kPreHalo;  // 128: 32 lanes x 4 columns
constexpr int kPreWarps = 16;                  // of ROWS = 2, 3, 4 or 8 rows
constexpr int kPreThreads = 32 * kPreWarps;
static_assert(kPreW == 128 && kPreHalo >= 12, "tile of the inverse Gaborish");
// Tile rows in shared memory are kPreP floats apart: 16-byte aligned for the
// rows' float4 accesses, and a column's 32 consecutive rows spread over 8
// banks for the ring's per-cell accesses (a pitch of 128 puts them all in
// one).
constexpr int kPreP = kPreW + 4;
// F (a ring tile's source, [H][kPreP]), then an interior tile's published
// rows [2 parities][kPreWarps][first, last][kPreW], or a ring tile's step
// inputs [2 parities][H][kPreP].
template <int ROWS>
struct PreTile {
  static constexpr int H = ROWS * kPreWarps;         // up to 128 rows
  static constexpr int kOut = H - 2 * kPreHalo;      // of them outputs
  static constexpr size_t kSmem = (size_t)3 * H * kPreP * sizeof(float);
};

struct EncKernel {
  float centre, edge, corner, inv_c;
};

// The tiles of a frame: a rectangle [fx0, fx1) x [fy0, fy1) of tiles with no
// cell of another rule (kEdge false) and the ring around it (kEdge true).
struct PreTiles {
  int tx, ty;  // tiles across and down
  int fx0, fx1, fy0, fy1;
};

// The update of the last n % 4 samples of the plane divides by the centre
// weight; out of line so that the division is not evaluated for every cell.
static __device__ __noinline__ float precondition_tail(float mm, float fv, float kx, float centre) {
  return mm + (fv - kx) / centre;
}

// The sums that take a neighbour one column over (pairs that straddle two
// registers' alignment) and the products run as two scalar operations: a
// paired sum of them costs register moves, a paired product a run-time
// addend of -0 and an operand's bank conflict (4096 x 3072: 433 us all
// paired, 396 all scalar, 388 mixed so).
__device__ __forceinline__ f2 f2_add_lanes(f2 a, f2 b) {
  return f2_pack(f2_lo(a) + f2_lo(b), f2_hi(a) + f2_hi(b));
}
__device__ __forceinline__ f2 f2_mul_lanes(f2 a, f2 b) {
  return f2_pack(f2_lo(a) * f2_lo(b), f2_hi(a) * f2_hi(b));
}

// The three rows around a row of four cells, as lane pairs.  Columns are
// paired (0, 1) and (2, 3); W*, C*, E* are the pairs one column to the
// left of pair 0, between the pairs, and one column to the right of pair 1.
struct PreRows {
  f2 Mn0, Mn1, Mm0, Mm1, Ms0, Ms1;
  f2 Wn, Cn, En, Wm, Cm, Em, Ws, Cs, Es;
};
__device__ __forceinline__ PreRows pre_rows(const float4& n, float nW, float nE, const float4& m,
                                            float mW, float mE, const float4& s, float sW,
                                            float sE) {
  PreRows q;
  q.Mn0 = f2_pack(n.x, n.y);
  q.Mn1 = f2_pack(n.z, n.w);
  q.Mm0 = f2_pack(m.x, m.y);
  q.Mm1 = f2_pack(m.z, m.w);
  q.Ms0 = f2_pack(s.x, s.y);
  q.Ms1 = f2_pack(s.z, s.w);
  q.Wn = f2_pack(nW, n.x);
  q.Cn = f2_pack(n.y, n.z);
  q.En = f2_pack(n.w, nE);
  q.Wm = f2_pack(mW, m.x);
  q.Cm = f2_pack(m.y, m.z);
  q.Em = f2_pack(m.w, mE);
  q.Ws = f2_pack(sW, s.x);
  q.Cs = f2_pack(s.y, s.z);
  q.Es = f2_pack(s.w, sE);
  return q;
}

// Interior rule: mm*c + (((N + S) + W) + E)*e + (((NW + NE) + SW) + SE)*k.
__device__ __forceinline__ void pre_kx_interior(const PreRows& q, f2 c2, f2 e2, f2 k2, f2& kxa,
                                                f2& kxb) {
  const f2 s1a = f2_add_lanes(f2_add_lanes(f2_add(q.Mn0, q.Ms0), q.Wm), q.Cm);
  const f2 s2a = f2_add_lanes(f2_add_lanes(f2_add_lanes(q.Wn, q.Cn), q.Ws), q.Cs);
  const f2 s1b = f2_add_lanes(f2_add_lanes(f2_add(q.Mn1, q.Ms1), q.Cm), q.Em);
  const f2 s2b = f2_add_lanes(f2_add_lanes(f2_add_lanes(q.Cn, q.En), q.Cs), q.Es);
  kxa = f2_add(f2_add(f2_mul_lanes(q.Mm0, c2), f2_mul_lanes(s1a, e2)), f2_mul_lanes(s2a, k2));
  kxb = f2_add(f2_add(f2_mul_lanes(q.Mm1, c2), f2_mul_lanes(s1b, e2)), f2_mul_lanes(s2b, k2));
}

// mm + (f - kx) * (1/c).
__device__ __forceinline__ float4 pre_update(const PreRows& q, const float4& f, f2 kxa, f2 kxb,
                                             f2 i2) {
  const f2 ya = f2_add(q.Mm0, f2_mul_lanes(f2_sub(f2_pack(f.x, f.y), kxa), i2));
  const f2 yb = f2_add(q.Mm1, f2_mul_lanes(f2_sub(f2_pack(f.z, f.w), kxb), i2));
  return make_float4(f2_lo(ya), f2_hi(ya), f2_lo(yb), f2_hi(yb));
}

// A ring tile's cell of another rule, found once: its tile position and the
// tile rows and columns of its mirrored taps (7 bits each) and its rule.
struct PreSpecial {
  uint32_t a;  // tx | xm << 7 | xp << 14 | ty << 21
  uint32_t b;  // ym | yp << 7 | seq << 14 | div << 15 | valid << 16
};
template <int H>
__device__ __forceinline__ PreSpecial pre_special(int ty, int tx, int cx, int cy, int gx0, int gy0,
                                                  int w, int h, bool seq, bool div) {
  auto clampt = [](int v, int n) { return min(max(v, 0), n - 1); };
  const int xm = clampt(mirror1d(cx - 1, w) - gx0, kPreW),
            xp = clampt(mirror1d(cx + 1, w) - gx0, kPreW);
  const int ym = clampt(mirror1d(cy - 1, h) - gy0, H), yp = clampt(mirror1d(cy + 1, h) - gy0, H);
  return {(uint32_t)tx | (uint32_t)xm << 7 | (uint32_t)xp << 14 | (uint32_t)ty << 21,
          (uint32_t)ym | (uint32_t)yp << 7 | (uint32_t)seq << 14 | (uint32_t)div << 15 | 1u << 16};
}
// Its update from the step's input S into Sn.
__device__ __forceinline__ void pre_special_step(const PreSpecial& c, const float* S, const float* F,
                                                 float* Sn, const EncKernel& k) {
  const int tx = c.a & 127, xm = (c.a >> 7) & 127, xp = (c.a >> 14) & 127, y0 = (c.a >> 21) * kPreP;
  const int ym = (c.b & 127) * kPreP, yp = ((c.b >> 7) & 127) * kPreP;
  const float nw = S[ym + xm], nn = S[ym + tx], ne = S[ym + xp];
  const float ww = S[y0 + xm], mm = S[y0 + tx], ee = S[y0 + xp];
  const float sw = S[yp + xm], ss = S[yp + tx], se = S[yp + xp];
  float kx;
  if (!((c.b >> 14) & 1u)) {
    kx = mm * k.centre + (nn + ss + ww + ee) * k.edge + (nw + ne + sw + se) * k.corner;
  } else {
    // nine taps in order: dy = -1, 0, 1 outer, dx inner
    float acc = 0.0f;
    acc += k.corner * nw;
    acc += k.edge * nn;
    acc += k.corner * ne;
    acc += k.edge * ww;
    acc += k.centre * mm;
    acc += k.edge * ee;
    acc += k.corner * sw;
    acc += k.edge * ss;
    acc += k.corner * se;
    kx = acc;
  }
  const float fv = F[y0 + tx];
  Sn[y0 + tx] = ((c.b >> 15) & 1u) ? precondition_tail(mm, fv, kx, k.centre)
                                    : mm + (fv - kx) * k.inv_c;
}

// The cells of another rule in a ring tile with frame origin (gx0, gy0):
// the special rows (frame row 0 and rows [rb, h)) across the tile's
// in-frame columns, then the special columns (0 and [cb, w)) down its other
// in-frame rows; rb and cb as the reference's groups of four and division
// tail place them.
template <int H>
struct PreRingCells {
  int cx0, ncin, rB0, nr0, nrin, cB0, nrow_cells, count, groups;
  bool r0, c0;
  size_t bulk;
  __device__ __forceinline__ PreSpecial special(int i, int w, int h, int gx0, int gy0) const {
    int ty, tx;
    if (i < nrow_cells) {
      const int rr = i / ncin;
      tx = cx0 + (i - rr * ncin);
      ty = r0 ? (rr == 0 ? -gy0 : rB0 + rr - 1) : rB0 + rr;
    } else {
      const int j = i - nrow_cells;
      const int ci = j / nrin;
      ty = nr0 + (j - ci * nrin);
      tx = c0 ? (ci == 0 ? -gx0 : cB0 + ci - 1) : cB0 + ci;
    }
    const int cx = gx0 + tx, cy = gy0 + ty;
    const bool border = cx == 0 || cx == w - 1 || cy == 0 || cy == h - 1;
    return pre_special<H>(ty, tx, cx, cy, gx0, gy0, w, h, border || cx - 1 >= 4 * groups,
                       (size_t)cy * w + cx >= bulk);
  }
};
template <int H>
__device__ __forceinline__ PreRingCells<H> pre_ring_cells(int w, int h, int gx0, int gy0) {
  PreRingCells<H> g;
  const size_t plane = (size_t)w * h;
  g.groups = (w >= 3 && h >= 3) ? (w - 2) / 4 : 0;
  g.bulk = plane - plane % 4;
  const int bulk_row = (int)(g.bulk / (size_t)w);
  const int rb = max(g.bulk == plane ? h - 1 : min(h - 1, bulk_row), 1);
  const int cb = max(min(w - 1, 4 * g.groups + 1), 1);
  g.cx0 = max(0, -gx0);
  g.ncin = max(0, min(kPreW, w - gx0) - g.cx0);
  const int ry0 = max(0, -gy0), ry1 = min(H, h - gy0), cx1 = g.cx0 + g.ncin;
  g.r0 = -gy0 >= ry0 && -gy0 < ry1;
  g.rB0 = max(ry0, rb - gy0);
  const int nsr = (g.r0 ? 1 : 0) + max(0, ry1 - g.rB0);
  g.nr0 = max(ry0, 1 - gy0);
  g.nrin = max(0, min(ry1, rb - gy0) - g.nr0);
  g.c0 = -gx0 >= g.cx0 && -gx0 < cx1;
  g.cB0 = max(g.cx0, cb - gx0);
  const int nsc = (g.c0 ? 1 : 0) + max(0, cx1 - g.cB0);
  g.nrow_cells = nsr * g.ncin;
  g.count = g.nrow_cells + nsc * g.nrin;
  return g;
}

__device__ __forceinline__ int pre_clamp(int c, int size) { return min(max(c, 0), size - 1); }

// One tile: item is the tile's index among the interior tiles (row-major
// over the rectangle) or among the ring tiles.
template <int ROWS, bool kEdge>
__device__ __forceinline__ void precondition_tile(const float* __restrict__ in,
                                                  float* __restrict__ out, int w, int h,
                                                  const EncKernel& k, const PreTiles& pt,
                                                  int item) {
  extern __shared__ __align__(16) float pre_smem[];
  constexpr int H = PreTile<ROWS>::H;
  float* const F = pre_smem;               // [H][kPreP]
  float* const xb = pre_smem + H * kPreP;  // published rows, or the ring's step inputs
  const size_t plane = (size_t)w * h;
  in += plane * blockIdx.z;
  out += plane * blockIdx.z;
  int tile_x, tile_y;
  if (!kEdge) {
    const int nfx = pt.fx1 - pt.fx0;
    tile_y = pt.fy0 + item / nfx;
    tile_x = pt.fx0 + item % nfx;
  } else {
    // Ring tiles: the rows above the rectangle, the rows below it, then the
    // tiles left and right of it on its rows.
    int i = item;
    const int top = pt.fy0 * pt.tx, bottom = (pt.ty - pt.fy1) * pt.tx;
    if (i < top) {
      tile_y = i / pt.tx;
      tile_x = i - tile_y * pt.tx;
    } else if (i < top + bottom) {
      i -= top;
      tile_y = pt.fy1 + i / pt.tx;
      tile_x = i - (tile_y - pt.fy1) * pt.tx;
    } else {
      i -= top + bottom;
      const int side = pt.fx0 + (pt.tx - pt.fx1);
      tile_y = pt.fy0 + i / side;
      const int c = i - (tile_y - pt.fy0) * side;
      tile_x = c < pt.fx0 ? c : pt.fx1 + (c - pt.fx0);
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tx0 = tile_x * kPreOut, ty0 = tile_y * PreTile<ROWS>::kOut;
  const int gx0 = tx0 - kPreHalo, gy0 = ty0 - kPreHalo;
  const int lx = 4 * lane, ly = ROWS * warp;  // the thread's first column and row in the tile
  const int gx = gx0 + lx, gy = gy0 + ly;  // ... in the frame
  // Load: tiles inside the frame with 16-byte aligned rows take 16-byte
  // loads; others clamp each coordinate (cells outside the frame are never
  // read by a cell inside it, so their values do not matter).
  const bool vec = gx0 >= 0 && gy0 >= 0 && gx0 + kPreW <= w && gy0 + H <= h && (w % 4) == 0 &&
                   ((reinterpret_cast<uintptr_t>(in) & 15) == 0);
  float4 X[ROWS];
  if (vec) {
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
      X[r] = __ldg(reinterpret_cast<const float4*>(in + (size_t)(gy + r) * w + gx));
  } else {
    const int c0 = pre_clamp(gx, w), c1 = pre_clamp(gx + 1, w), c2 = pre_clamp(gx + 2, w),
              c3 = pre_clamp(gx + 3, w);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const float* row = in + (size_t)pre_clamp(gy + r, h) * w;
      X[r] = make_float4(__ldg(row + c0), __ldg(row + c1), __ldg(row + c2), __ldg(row + c3));
    }
  }
  const f2 c2 = f2_pack(k.centre, k.centre), e2 = f2_pack(k.edge, k.edge);
  const f2 k2 = f2_pack(k.corner, k.corner), i2 = f2_pack(k.inv_c, k.inv_c);
  const unsigned full = 0xffffffffu;
  if (!kEdge) {
    float4 Fr[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) Fr[r] = X[r];
    // The rows just above and below the warp's: the last row of the warp
    // above and the first of the warp below (the tile's edge rows for the
    // first and last warps, never read by an exact cell).
    const int row_up = (2 * max(warp - 1, 0) + 1) * kPreW + lx;
    const int row_down = (2 * min(warp + 1, kPreWarps - 1)) * kPreW + lx;
#pragma unroll 1
    for (int it = 0; it < 12; ++it) {
      float* const S = xb + (it & 1) * (kPreWarps * 2 * kPreW);
      *reinterpret_cast<float4*>(S + (2 * warp) * kPreW + lx) = X[0];
      *reinterpret_cast<float4*>(S + (2 * warp + 1) * kPreW + lx) = X[ROWS - 1];
      __syncthreads();
      float4 prev = *reinterpret_cast<const float4*>(S + row_up);
      float pW = __shfl_up_sync(full, prev.w, 1), pE = __shfl_down_sync(full, prev.x, 1);
      float mW = __shfl_up_sync(full, X[0].w, 1), mE = __shfl_down_sync(full, X[0].x, 1);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const float4 nxt =
            r < ROWS - 1 ? X[r + 1 < ROWS ? r + 1 : r] : *reinterpret_cast<const float4*>(S + row_down);
        const float sW = __shfl_up_sync(full, nxt.w, 1), sE = __shfl_down_sync(full, nxt.x, 1);
        const float4 f = Fr[r];
        f2 kxa, kxb;
        const PreRows q = pre_rows(prev, pW, pE, X[r], mW, mE, nxt, sW, sE);
        pre_kx_interior(q, c2, e2, k2, kxa, kxb);
        const float4 y = pre_update(q, f, kxa, kxb, i2);
        prev = X[r];
        pW = mW;
        pE = mE;
        X[r] = y;
        mW = sW;
        mE = sE;
      }
    }
  } else {
    // Ring tiles keep the step's input in shared memory and write the
    // step's output to the other buffer; each thread first finds its cells
    // of another rule (at most two, as a rule none).
    const PreRingCells<H> rc = pre_ring_cells<H>(w, h, gx0, gy0);
    PreSpecial mine[2] = {{0u, 0u}, {0u, 0u}};
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int i = threadIdx.x + s * kPreThreads;
      if (i < rc.count) mine[s] = rc.special(i, w, h, gx0, gy0);
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      *reinterpret_cast<float4*>(F + (ly + r) * kPreP + lx) = X[r];
      *reinterpret_cast<float4*>(xb + (ly + r) * kPreP + lx) = X[r];
    }
    const int row_up = max(ly - 1, 0) * kPreP + lx;
    // Rows wholly outside the frame are read by no cell inside it (64 x 64:
    // half of the tile; 30 us with them, 23 without).
    const bool live = gy + ROWS - 1 >= 0 && gy < h;
#pragma unroll 1
    for (int it = 0; it < 12; ++it) {
      const float* const S = xb + (it & 1) * (H * kPreP);
      float* const Sn = xb + ((it + 1) & 1) * (H * kPreP);
      __syncthreads();
      // A warp whose rows have all left the exact region [1 + it,
      // H - 1 - it) rests; its rows in the step buffers are read only by
      // cells that are no longer exact either.
      if (live && !(ly + ROWS - 1 < 1 + it || ly >= H - 1 - it)) {
        float4 prev = *reinterpret_cast<const float4*>(S + row_up);
        float4 cur = *reinterpret_cast<const float4*>(S + ly * kPreP + lx);
        float pW = __shfl_up_sync(full, prev.w, 1), pE = __shfl_down_sync(full, prev.x, 1);
        float mW = __shfl_up_sync(full, cur.w, 1), mE = __shfl_down_sync(full, cur.x, 1);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const float4 nxt =
              *reinterpret_cast<const float4*>(S + min(ly + r + 1, H - 1) * kPreP + lx);
          const float sW = __shfl_up_sync(full, nxt.w, 1), sE = __shfl_down_sync(full, nxt.x, 1);
          const float4 f = *reinterpret_cast<const float4*>(F + (ly + r) * kPreP + lx);
          f2 kxa, kxb;
          const PreRows q = pre_rows(prev, pW, pE, cur, mW, mE, nxt, sW, sE);
          pre_kx_interior(q, c2, e2, k2, kxa, kxb);
          *reinterpret_cast<float4*>(Sn + (ly + r) * kPreP + lx) = pre_update(q, f, kxa, kxb, i2);
          prev = cur;
          pW = mW;
          pE = mE;
          cur = nxt;
          mW = sW;
          mE = sE;
        }
      }
      __syncthreads();
      if (mine[0].b) pre_special_step(mine[0], S, F, Sn, k);
      if (mine[1].b) pre_special_step(mine[1], S, F, Sn, k);
      // More cells than two per thread (none for frames at least 4 samples wide).
      if (rc.count > 2 * kPreThreads) {
        const PreRingCells<H> more = pre_ring_cells<H>(w, h, gx0, gy0);
        for (int i = threadIdx.x + 2 * kPreThreads; i < more.count; i += kPreThreads)
          pre_special_step(more.special(i, w, h, gx0, gy0), S, F, Sn, k);
      }
    }
    __syncthreads();
    // Twelve steps end in buffer 0; each thread reads back its own rows.
#pragma unroll
    for (int r = 0; r < ROWS; ++r) X[r] = *reinterpret_cast<const float4*>(xb + (ly + r) * kPreP + lx);
  }
  // The inner rows and columns: lanes 3 .. 28 of rows 12 .. H - 13.
  const int oh = kPreHalo / 4;
  if (lane >= oh && lane < 32 - oh) {
    const bool vec_out =
        gx + 3 < w && (w % 4) == 0 && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      if (ly + r < kPreHalo || ly + r >= H - kPreHalo || gy + r >= h) continue;
      float* row = out + (size_t)(gy + r) * w;
      if (vec_out) {
        *reinterpret_cast<float4*>(row + gx) = X[r];
      } else {
        if (gx < w) row[gx] = X[r].x;
        if (gx + 1 < w) row[gx + 1] = X[r].y;
        if (gx + 2 < w) row[gx + 2] = X[r].z;
        if (gx + 3 < w) row[gx + 3] = X[r].w;
      }
    }
  }
}

// Both kinds of tile in one launch: the ring tiles at blockIdx.x < nedge,
// then the interior tiles.
template <int ROWS>
__global__ void __launch_bounds__(kPreThreads, 1) k_precondition(const float* __restrict__ in,
                                                              float* __restrict__ out, int w,
                                                              int h, EncKernel k, PreTiles pt,
                                                              int nedge) {
  const int i = (int)blockIdx.x;
  if (i < nedge) precondition_tile<ROWS, true>(in, out, w, h, k, pt, i);
  else precondition_tile<ROWS, false>(in, out, w, h, k, pt, i - nedge);
}

template <int ROWS>
static int precondition_rows(const float* in, float* out, int w, int h, cudaStream_t s) {
  using Tile = PreTile<ROWS>;
  const float w1 = 0.115169525f, w2 = 0.061248592f;
  // gaborish.rs:31 GaborKernel::new, normalised without FMA.
  float unnorm = 1.0f + 4.0f * w1 + 4.0f * w2;
  float scale = 1.0f / unnorm;
  EncKernel k{scale, w1 * scale, w2 * scale, 1.0f / scale};
  PreTiles pt{(w + kPreOut - 1) / kPreOut, (h + Tile::kOut - 1) / Tile::kOut, 0, 0, 0, 0};
  // Columns and rows of cells with another rule: 0, [cb, w) and 0, [rb, h)
  // (the frame border, the columns past the groups of four, the rows of
  // the division tail).  A tile is in the rectangle when its haloed extent
  // [t*104 - 12, t*104 + 116), down [t*kOut - 12, (t+1)*kOut + 12), lies inside
  // [1, cb) and [1, rb).
  const long long n = (long long)w * h;
  const int groups = (w >= 3 && h >= 3) ? (w - 2) / 4 : 0;
  const int cb = std::max(std::min(w - 1, 4 * groups + 1), 1);
  const int row_end = n % 4 == 0 ? h - 1 : (int)std::min<long long>(h - 1, (n - n % 4) / w);
  const int rb = std::max(row_end, 1);
  const int reach = kPreW - kPreHalo, reach_y = Tile::H - kPreHalo;
  const int fx1 = cb >= reach ? std::min((cb - reach) / kPreOut + 1, pt.tx) : 0;
  const int fy1 = rb >= reach_y ? std::min((rb - reach_y) / Tile::kOut + 1, pt.ty) : 0;
  if (fx1 > 1 && fy1 > 1) {
    pt.fx0 = 1;
    pt.fx1 = fx1;
    pt.fy0 = 1;
    pt.fy1 = fy1;
  }
  const int nfast = (pt.fx1 - pt.fx0) * (pt.fy1 - pt.fy0);
  const int nedge = pt.tx * pt.ty - nfast;
  k_precondition<ROWS><<<dim3(nedge + nfast, 1, 3), kPreThreads, Tile::kSmem, s>>>(in, out, w, h, k,
                                                                                  pt, nedge);
  return 1;
}

// Rows per lane: the fewest with which every tile still has an SM of its own,
// else eight.  A short tile computes more cells per output but ends sooner
// (64x64: 24.5 us with eight rows, 18.3 with four, 14.2 with two; 501x333:
// 30.7, 20.2 with four); beyond a tile to an SM the work is the time, and
// choosing rows to fill the last round better gained nothing (1920x1080 with
// seven: 81.8 us, 81.0 with eight).
int launch_precondition(const float* in, float* out, int w, int h, int num_sms, cudaStream_t s) {
  auto fits = [&](int outs) {
    const long long across = (w + kPreOut - 1) / kPreOut, down = (h + outs - 1) / outs;
    return 3 * across * down <= num_sms;
  };
  if (fits(PreTile<2>::kOut)) return precondition_rows<2>(in, out, w, h, s);
  if (fits(PreTile<3>::kOut)) return precondition_rows<3>(in, out, w, h, s);
  if (fits(PreTile<4>::kOut)) return precondition_rows<4>(in, out, w, h, s);
  return precondition_rows<8>(in, out, w, h, s);
}

// ---------------------------------------------------------------------------
// Shared quantization rules (jpxl-encode-policy quantize.rs)
// ---------------------------------------------------------------------------

constexpr float kQuantBiasX = 1.0f - 0.054650073f, kQuantBiasY = 1.0f - 0.0700545f,
                kQuantBiasB = 1.0f - 0.049935103f;
__constant__ float c_quant_bias[3] = {kQuantBiasX, kQuantBiasY, kQuantBiasB};

__device__ float g_bias_quot[kBiasQuotN];
__device__ float4 g_levels[3][kLevelN];

// quantize.rs:199 LfQuantizer::quantize with extra_precision 0.
__device__ __forceinline__ int32_t lf_quantize(float target, float m, uint32_t* err) {
  if (!(isfinite(m) && m > 0.0f)) {
    raise_error(err, kDevBadStep);
    return 0;
  }
  float scaled = target * 1.0f / m;
  int32_t q;
  if (!clamp_round(scaled, &q)) {
    raise_error(err, kDevQuantRange);
    return 0;
  }
  return q;
}

// ---------------------------------------------------------------------------
// K3 — forward transform of every square varblock (policy lib.rs:3008
// gather_square with edge replication; forward.rs:451 forward_dct_rc =
// dct.rs:956 DCT_2D), LF samples (lib.rs:3100 lf_samples_of; forward.rs:779
// lf_from_llf_into), and the luma half of lib.rs:3237
// quantize_square_varblock: LF quantize + reconstruct, HF choose +
// reconstruct.
//
// 8 x 8: eight lanes per block, four blocks per warp; lane j transforms
// column j, then (through shared memory, its own warp only) row j, ending
// with column j of the coefficient matrix, which it writes to column bx*8+j
// of the coefficient image.  The three channels go together: their loads are
// in flight at once and no barrier of the block is needed.
// FROM_IMAGE: the split-precision forward transform has written all three
// channels' coefficients already.
// ---------------------------------------------------------------------------

template <bool FROM_IMAGE>
__global__ void __launch_bounds__(128) k_fdct8(EncArgs a, const uint32_t* __restrict__ list,
                                               int count) {
  __shared__ float T[16][3][8][9];
  const int g = threadIdx.x / 8, j = threadIdx.x % 8;
  const int vi = blockIdx.x * 16 + g;
  const bool active = vi < count;
  const uint32_t packed = list[active ? vi : count - 1];  // idle lanes repeat the last block
  const int bx = packed & 0xffff, by = packed >> 16;
  const int x0 = bx * 8, y0 = by * 8;
  const Geo& geo = a.geo;
  const size_t plane = (size_t)geo.w * geo.h;
  const size_t cplane = (size_t)geo.W8 * geo.H8;
  const size_t cell0 = (size_t)y0 * geo.W8 + x0 + j;
  const float mul =
      hf_multiplier(a.mul_table, a.qs.global_scale, a.hf_mul[(size_t)by * geo.bw + bx]);
  float v[3][8];
  if constexpr (FROM_IMAGE) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (c == 1 || k == 0) v[c][k] = a.coeff[cplane * c + cell0 + (size_t)k * geo.W8];
  } else {
    const int xx = min(x0 + j, geo.w - 1);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = 0; r < 8; ++r)
        v[c][r] = a.pre[plane * c + (size_t)min(y0 + r, geo.h - 1) * geo.w + xx];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      dct_1d<8>(v[c]);
#pragma unroll
      for (int r = 0; r < 8; ++r) T[g][c][r][j] = v[c][r];
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int k = 0; k < 8; ++k) v[c][k] = T[g][c][j][k];
      dct_1d<8>(v[c]);
    }
    if (active)
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < 8; ++k) a.coeff[cplane * c + cell0 + (size_t)k * geo.W8] = v[c][k];
  }
  if (!active) return;
  // LF samples of all three channels (a 1 x 1 inverse: the coefficient) and
  // the luma LF quantization.
  if (j == 0) {
    const size_t bplane = (size_t)geo.bw * geo.bh, bi = (size_t)by * geo.bw + bx;
    const float sf2 = c_scale_f[0] * c_scale_f[0];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float lf = v[c][0] / sf2;
      a.lfs[bplane * c + bi] = lf;
      if (c == 1) {
        const int32_t q = lf_quantize(lf, a.qs.m_dc[1], a.err);
        a.lfq[bplane + bi] = q;
        a.dylf[bi] = a.qs.m_dc[1] * (float)q / 1.0f;
      }
    }
  }
  // Luma HF: cells (k, j) of column j; the LLF cell stays zero: level 0, from
  // a target under every threshold.
  if (j == 0) v[1][0] = 0.0f;
  const float scale = mul * a.qs.qm[1];
  const float* m = a.dq + kDequantTableFloats + dq_offset(dq_slot(0));
  // Through this lane's own column of T, so that the choice is not inlined
  // twice.
#pragma unroll
  for (int k = 0; k < 8; ++k) T[g][1][j][k] = v[1][k];
#pragma unroll 1
  for (int k0 = 0; k0 < 8; k0 += 4) {
    float target[4], step[4], recon[4];
    int32_t q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      target[i] = T[g][1][j][k0 + i];
      step[i] = scale * __ldg(&m[(k0 + i) * 8 + j]);
    }
    choose_n<4>(1, target, step, a.err, q, recon);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const size_t ci = cell0 + (size_t)(k0 + i) * geo.W8;
      a.qcoeff[cplane + ci] = q[i];
      a.dyhf[ci] = recon[i];
    }
  }
}

// K3, N = 16 and 32 — the same block by N / 4 warps, a share of each column
// per warp and the three channels together through each phase: the split of
// k_render_rect, for the same reason (the luma stage at 1920x1080: 47 us, now
// 34; at 64x64 14.9, now 13.3).
template <int N, bool FROM_IMAGE = false>
__global__ void __launch_bounds__(8 * N) k_fdct_sq(EncArgs a, const uint32_t* __restrict__ list,
                                                   int count) {
  constexpr int kShares = N / 4, VPB = 32 / N, n = N / 8;
  constexpr int kRows = FROM_IMAGE ? 1 : N;
  __shared__ float A[VPB][3][kRows][N + 1], B[VPB][3][kRows][N + 1];
  __shared__ float LL[VPB][3][16];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int g = lane / N, j = lane % N;
  const int vi = blockIdx.x * VPB + g;
  const bool active = vi < count;
  const uint32_t packed = list[active ? vi : count - 1];  // an idle half repeats the last block
  const int bx = packed & 0xffff, by = packed >> 16;
  const int x0 = bx * 8, y0 = by * 8;
  const Geo& geo = a.geo;
  const size_t plane = (size_t)geo.w * geo.h;
  const size_t cplane = (size_t)geo.W8 * geo.H8;
  const float mul =
      hf_multiplier(a.mul_table, a.qs.global_scale, a.hf_mul[(size_t)by * geo.bw + bx]);
  float target[4];
  if constexpr (FROM_IMAGE) {
    // The split-precision forward transform has written all three channels'
    // coefficients.
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = 4 * warp + i;
      target[i] = a.coeff[cplane + (size_t)(y0 + k) * geo.W8 + x0 + j];
      if (k < n && j < n)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          LL[g][c][k * n + j] = a.coeff[cplane * c + (size_t)(y0 + k) * geo.W8 + x0 + j];
    }
    __syncthreads();
  } else {
    const int xx = min(x0 + j, geo.w - 1);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = 4 * warp + i;
        A[g][c][r][j] = a.pre[plane * c + (size_t)min(y0 + r, geo.h - 1) * geo.w + xx];
      }
    __syncthreads();
#pragma unroll 1
    for (int c = 0; c < 3; ++c)
      dct_share<N>((warp + 3 * c) % kShares, [&](int i) { return A[g][c][i][j]; },
                   [&](int k, float v) { B[g][c][k][j] = v; });
    __syncthreads();
#pragma unroll 1
    for (int c = 0; c < 3; ++c)
      dct_share<N>((warp + 3 * c) % kShares, [&](int i) { return B[g][c][j][i]; },
                   [&](int k, float v) { A[g][c][k][j] = v; });
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = 4 * warp + i;
      target[i] = A[g][1][k][j];
      if (k < n && j < n)
#pragma unroll
        for (int c = 0; c < 3; ++c) LL[g][c][k * n + j] = A[g][c][k][j];
      if (active)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          a.coeff[cplane * c + (size_t)(y0 + k) * geo.W8 + x0 + j] = A[g][c][k][j];
    }
  }
  // Luma HF: cells (k, j) of column j; the n x n LLF corner stays zero.
  if (active) {
    const float scale = mul * a.qs.qm[1];
    const float* m = a.dq + kDequantTableFloats + dq_offset(dq_slot(N == 16 ? 4 : 5));
    float step[4], recon[4];
    int32_t q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = 4 * warp + i;
      step[i] = scale * __ldg(&m[k * N + j]);
      // the LLF corner: level 0, from a target under every threshold
      if (k < n && j < n) target[i] = 0.0f;
    }
    choose_n<4>(1, target, step, a.err, q, recon);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const size_t ci = (size_t)(y0 + 4 * warp + i) * geo.W8 + x0 + j;
      a.qcoeff[cplane + ci] = q[i];
      a.dyhf[ci] = recon[i];
    }
  }
  // LF samples of all three channels: IDCT_2D of the n x n LLF corner over its
  // scale factors (one lane per column, then per row) and the luma LF quantization, by the warp that holds the corner.
  if (warp != 0) return;
  __syncwarp();
  const int lg = lane / (3 * n), c = lane / n % 3, k = lane % n;
  const int lv = blockIdx.x * VPB + lg;
  const bool on = lane < VPB * 3 * n && lv < count;
  const float* sf = &c_scale_f[(n == 2 ? 1 : 2) * 8];
  float v[n];
  if (on) {
#pragma unroll
    for (int r = 0; r < n; ++r) v[r] = LL[lg][c][r * n + k] / (sf[r] * sf[k]);
    idct_1d<n>(v);
#pragma unroll
    for (int r = 0; r < n; ++r) LL[lg][c][r * n + k] = v[r];
  }
  __syncwarp();
  if (!on) return;
#pragma unroll
  for (int r = 0; r < n; ++r) v[r] = LL[lg][c][k * n + r];
  idct_1d<n>(v);
  const uint32_t pk = list[lv];
  const size_t bplane = (size_t)geo.bw * geo.bh;
#pragma unroll
  for (int r = 0; r < n; ++r) {
    const size_t bi = (size_t)((pk >> 16) + r) * geo.bw + (pk & 0xffff) + k;
    a.lfs[bplane * c + bi] = v[r];
    if (c == 1) {
      const int32_t lq = lf_quantize(v[r], a.qs.m_dc[1], a.err);
      a.lfq[bplane + bi] = lq;
      a.dylf[bi] = a.qs.m_dc[1] * (float)lq / 1.0f;
    }
  }
}

// ---------------------------------------------------------------------------
// K4 — chroma-from-luma estimation (policy lib.rs:3437 estimate_cfl).
//
// Decisions depend on f64 regression sums that the reference accumulates in
// one fixed sequential order.  The kernels sum in a fixed tree order instead
// and bound the difference: both orders lie within n*u*sum|t| of the exact
// sum (u = 2^-53), which bounds how far the least-squares seed
// round((s_yc/s_yy - base)*84) and the energy comparisons that confirm it
// can move.  Where the seed is more than that bound away from a decision
// boundary the tree result is the reference's; otherwise the tile (or the
// frame-wide LF pair) is recomputed sequentially in the reference's own
// order.  Residual bit costs are integer sums, exact in any order.
// ---------------------------------------------------------------------------

struct RegSums {
  double s_yy, s_yc, s_cc, a_yc;
  double n;
};

// quantize.rs:1640 best_factor on given sums; *robust = the result is
// certainly the one the reference's sequential sums give (bound `slack` on
// the absolute error of each sum, relative to its magnitude sum).
__device__ int best_factor(const RegSums& s, float base, double slack_yy, double slack_yc,
                           double slack_cc, bool* robust) {
  *robust = true;
  if (s.s_yy <= 0.0) {
    // s_yy is a sum of squares: the reference's is <= 0 only when every term
    // is zero, which the tree sum sees identically.
    return 0;
  }
  const double cf = 84.0;
  double k_ls = s.s_yc / s.s_yy;
  double star = (k_ls - (double)base) * cf;
  double centre_d = round(star);
  // Error of star from the sum differences (first order), with margin.
  double dk = (slack_yc + fabs(k_ls) * slack_yy) / s.s_yy;
  double dstar = cf * dk * 1.01 + 1e-12 * (1.0 + fabs(star));
  // Energy comparisons between neighbouring candidates are decided by
  // |j + 0.5 - star| * 2 s_yy / 84^2 against the f64 rounding of the
  // energies themselves (a few ulps of s_cc + 2|k s_yc| + k^2 s_yy).
  double kk = fabs(k_ls) + 2.0;
  double e_round = 8.0 * 1.1102230246251565e-16 *
                   (s.s_cc + slack_cc + 2.0 * kk * (fabs(s.s_yc) + slack_yc) + kk * kk * (s.s_yy + slack_yy));
  double tie = e_round * cf * cf / (2.0 * s.s_yy);
  double frac = star - floor(star);
  double dist = fabs(frac - 0.5);
  if (dist <= dstar + tie || !isfinite(star)) *robust = false;
  long long centre = (long long)centre_d;
  // candidates centre-2..centre+2 clamped to [-128,127], then 0; with a
  // robust star the nearest candidate wins outright.
  int best = 0;
  double best_e = 0.0;
  bool have = false;
  auto consider = [&](int cand) {
    double k = (double)((float)base + (float)cand / 84.0f);
    double e = s.s_cc - 2.0 * k * s.s_yc + k * k * s.s_yy;
    int ac = cand < 0 ? -cand : cand, ab = best < 0 ? -best : best;
    if (!have || e < best_e || (e == best_e && ac < ab)) {
      have = true;
      best = cand;
      best_e = e;
    }
  };
  for (int d = -2; d <= 2; ++d) {
    long long c = centre + d;
    c = c < -128 ? -128 : (c > 127 ? 127 : c);
    consider((int)c);
  }
  consider(0);
  return best;
}

// best_factor by eight lanes (a lane per candidate; `sub` is the lane's place
// among them, the group aligned): the candidates' energies are independent,
// and the choice goes over them in the same order afterwards.
__device__ __forceinline__ int best_factor_lanes(unsigned mask, int sub, const RegSums& s,
                                                 float base, double slack_yy, double slack_yc,
                                                 double slack_cc, bool* robust) {
  int star_cand = 0;
  *robust = true;
  double energy = 0.0;
  if (s.s_yy > 0.0) {
    const double cf = 84.0;
    const double k_ls = s.s_yc / s.s_yy;
    const double star = (k_ls - (double)base) * cf;
    const double dk = (slack_yc + fabs(k_ls) * slack_yy) / s.s_yy;
    const double dstar = cf * dk * 1.01 + 1e-12 * (1.0 + fabs(star));
    const double kk = fabs(k_ls) + 2.0;
    const double e_round = 8.0 * 1.1102230246251565e-16 *
                           (s.s_cc + slack_cc + 2.0 * kk * (fabs(s.s_yc) + slack_yc) +
                            kk * kk * (s.s_yy + slack_yy));
    const double tie = e_round * cf * cf / (2.0 * s.s_yy);
    const double dist = fabs((star - floor(star)) - 0.5);
    if (dist <= dstar + tie || !isfinite(star)) *robust = false;
    long long c = (long long)round(star) + (sub - 2);
    c = c < -128 ? -128 : (c > 127 ? 127 : c);
    star_cand = sub < 5 ? (int)c : 0;
    const double k = (double)((float)base + (float)star_cand / 84.0f);
    energy = s.s_cc - 2.0 * k * s.s_yc + k * k * s.s_yy;
  }
  int best = 0;
  double best_e = 0.0;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    const int cand = __shfl_sync(mask, star_cand, i, 8);
    const double e = __shfl_sync(mask, energy, i, 8);
    const int ac = cand < 0 ? -cand : cand, ab = best < 0 ? -best : best;
    if (i == 0 || e < best_e || (e == best_e && ac < ab)) {
      best = cand;
      best_e = e;
    }
  }
  return s.s_yy > 0.0 ? best : 0;  // as best_factor: all terms zero
}

__device__ __forceinline__ uint32_t factor_bits(int32_t f) {
  if (f == 0) return 0;
  uint32_t af = (uint32_t)(f < 0 ? -f : f);
  return (32u - __clz(af)) + 2u;
}

// One CTA per 64x64 tile, from the coefficients to the quantized chroma:
// (1) the HF regression sums (X and B against source Y) in double-float;
// (2) the seeds; (3) the residual bit costs of the candidate windows and the
// choice; (4) K5, the X and B cells against the chosen factors.  X, Y and B
// arrive once, by cp.async, and stay in shared memory; the reconstructed luma
// of (3) and (4) takes Y's place behind (1) and arrives while (2) runs.  The
// steps' latencies (the seeds' f64 chain above all) hide behind the SM's
// other tiles.
// Bound: issue slots and, with 32 warps to an SM, the steps' latencies.  Three
// planes instead of four let an SM hold four tiles; a cell whose candidates
// all fall under the zero threshold (most of a photograph's chroma) skips its
// ten quantizer choices.  Measured, with the LF chain beside it: 4096x3072
// 452 us, then 280 (one kernel), 255 (skips), 226 (four tiles); 1920x1080 66,
// then 57, 51.
// Where every tile has an SM of its own the CTA's own chain is the time, and
// 512 threads shorten it (64x64: 32.5 us, 28.5 with 512); beyond that CTAs of
// 256 hide one another's chains (2048x2048 at three to an SM: 109 against 118).
constexpr int kCflSide = 64;
template <int THREADS>
struct CflSmem {
  float p[3][kCflSide][kCflSide];        // X, Y, B coefficients; Y, then reconstructed luma
  float step[2][64], rstep[2][64];       // baseline quantizer, DCT8x8 cells
  float half[2][64];                     // its zero threshold, -1 for a step out of range
  float mul[64];                         // hf multiplier of each 8x8 block's varblock
  uint8_t lg[64];                        // log2 of its side in blocks
  DF part[THREADS / 32][8];
  uint32_t bits[THREADS / 32][8];
  int seed[2], factor[2];
};

// Eight double-float sums over a warp in the order of an xor butterfly, each
// step handing half of the remaining quantities to the partner lane.  Every
// fourth lane ends with the total of quantity *q = lane >> 2.
__device__ __forceinline__ DF warp_sum8(DF* v, int lane, int* q) {
  const unsigned full = 0xffffffffu;
  auto swap = [&](DF x, int o) {
    return DF{__shfl_xor_sync(full, x.hi, o), __shfl_xor_sync(full, x.lo, o)};
  };
  int base = 0;
#pragma unroll
  for (int o = 16, n = 4; o >= 4; o >>= 1, n >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const DF keep = up ? v[i + n] : v[i], send = up ? v[i] : v[i + n];
      v[i] = df_add(keep, swap(send, o));
    }
    base += up ? n : 0;
  }
  DF x = v[0];
  x = df_add(x, swap(x, 2));
  x = df_add(x, swap(x, 1));
  *q = base;
  return x;
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 4 : 1)
    k_cfl_tile(const __grid_constant__ EncArgs a) {
  extern __shared__ __align__(16) unsigned char cfl_smem[];
  auto& sm = *reinterpret_cast<CflSmem<THREADS>*>(cfl_smem);
  const Geo& geo = a.geo;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int tx = blockIdx.x, ty = blockIdx.y, tile = ty * geo.tw + tx;
  const size_t cplane = (size_t)geo.W8 * geo.H8;
  const int px0 = tx * kCflSide, py0 = ty * kCflSide;
  const int pw = min(kCflSide, geo.W8 - px0), ph = min(kCflSide, geo.H8 - py0);
  const size_t origin = (size_t)py0 * geo.W8 + px0;
  auto fetch = [&](const float* plane, float(&to)[kCflSide][kCflSide]) {
    for (int i = t; i < kCflSide * kCflSide / 4; i += THREADS) {
      const int x = 4 * (i % (kCflSide / 4)), y = i / (kCflSide / 4);
      if (x >= pw || y >= ph) continue;
      const float* src = plane + origin + (size_t)y * geo.W8 + x;
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&to[y][x]);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    }
  };
  for (int c = 0; c < 3; ++c) fetch(a.coeff + cplane * c, sm.p[c]);
  // Each block's varblock (square, naturally aligned: its origin is the
  // block position with the low bits cleared).
  if (t < 64) {
    const int bx = px0 / 8 + t % 8, by = py0 / 8 + t / 8;
    int l = 0;
    float mul = 1.0f;
    if (bx < geo.bw && by < geo.bh) {
      const int sel = a.block_map[(size_t)by * geo.bw + bx] & 0x1f;
      l = sel == 0 ? 0 : (sel == 4 ? 1 : 2);
      const int clear = ~((1 << l) - 1);
      mul = hf_multiplier(a.mul_table, a.qs.global_scale,
                          a.hf_mul[(size_t)(by & clear) * geo.bw + (bx & clear)]);
    }
    sm.lg[t] = (uint8_t)l;
    sm.mul[t] = mul;
  }
  // Baseline steps of the 64 folded cells and their reciprocals.
  if (t >= 128 && t < 256) {
    const int ch = (t - 128) / 64, cell = t % 64;
    const float scale = a.base_mul * a.qs.qm[ch == 0 ? 0 : 2];
    const float st = scale * a.dq[(ch == 0 ? 0 : 2) * kDequantTableFloats + cell];
    sm.step[ch][cell] = st;
    sm.rstep[ch][cell] = 1.0f / st;
    sm.half[ch][cell] = st > 0.0f && st < __int_as_float(0x7f800000)
                            ? 0.5f * c_quant_bias[ch == 0 ? 0 : 2] * st
                            : -1.0f;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const bool on = *a.not_gray != 0u && a.cfl_enabled;
  // Thread t covers column t % 64 of rows t / 64, t / 64 + kStep, ...
  const int col = t % kCflSide, row0 = t / kCflSide;
  constexpr int kStep = THREADS / kCflSide;
  int seed[2] = {0, 0};
  if (on) {
    // (1) s_yy, s_yx, s_xx, s_yb, s_bb, sum|yx|, sum|yb|, count.
    DF v[8] = {};
    if (col < pw)
#pragma unroll 2
      for (int row = row0; row < ph; row += kStep) {
        const int l = sm.lg[(row >> 3) * 8 + (col >> 3)], mask = (8 << l) - 1;
        if ((col & mask) < (1 << l) && (row & mask) < (1 << l)) continue;  // LLF
        const float x = sm.p[0][row][col], y = sm.p[1][row][col], b = sm.p[2][row][col];
        v[0] = df_add(v[0], df_two_prod(y, y));
        v[1] = df_add(v[1], df_two_prod(y, x));
        v[2] = df_add(v[2], df_two_prod(x, x));
        v[3] = df_add(v[3], df_two_prod(y, b));
        v[4] = df_add(v[4], df_two_prod(b, b));
        v[5].hi += fabsf(y * x);
        v[6].hi += fabsf(y * b);
        v[7].hi += 1.0f;
      }
    int q;
    const DF w = warp_sum8(v, lane, &q);
    if ((lane & 3) == 0) sm.part[warp][q] = w;
    __syncthreads();
    fetch(a.dyhf, sm.p[1]);
    // (2) Eight lanes for X's seed, eight for B's; a seed the bound cannot
    // settle is recomputed from the tile's coefficients in the reference's
    // order (varblocks in raster order of their origins within the tile,
    // then coefficient rows and columns).
    if (warp == 0) {
      DF sum = sm.part[0][lane & 7];
      for (int i = 1; i < THREADS / 32; ++i) sum = df_add(sum, sm.part[i][lane & 7]);
      const double value = df_value(sum);
      auto total = [&](int k) { return __shfl_sync(0xffffffffu, value, k); };
      const int ch = lane >> 3 & 1;
      const double t0 = total(0), t1 = total(1), t2 = total(2), t3 = total(3), t4 = total(4),
                   t5 = total(5), t6 = total(6), t7 = total(7);
      RegSums r{t0, ch ? t3 : t1, ch ? t4 : t2, ch ? t6 : t5, t7};
      // Distance of the double-float tree sum and of the reference's
      // sequential f64 sum from the exact sum, relative to sum|t| (the |t|
      // sums are f32 estimates; the factor 2 covers their error).
      const double gam = 2.0 * (r.n + 64.0) * (2.2737367544323206e-13 + 1.1102230246251565e-16);
      bool robust;
      int sd = best_factor_lanes(0xffffffffu, lane & 7, r, ch ? 1.0f : 0.0f, gam * r.s_yy,
                                 gam * r.a_yc, gam * r.s_cc, &robust);
      if (!(r.n > 0.0)) sd = 0;
      else if (!robust && (lane & 7) == 0 && lane < 16) {
        atomicAdd(a.cfl_fallbacks, 1u);
        RegSums e{0, 0, 0, 0, 0};
        for (int by = 0; by < ph / 8; ++by)
          for (int bx = 0; bx < pw / 8; ++bx) {
            const uint8_t m = a.block_map[(size_t)(py0 / 8 + by) * geo.bw + px0 / 8 + bx];
            if (!(m & 0x80)) continue;
            const int nb = 1 << sm.lg[by * 8 + bx], side = nb * 8;
            for (int row = 0; row < side; ++row)
              for (int cc = (row < nb ? nb : 0); cc < side; ++cc) {
                const double y = (double)a.coeff[cplane + origin + (size_t)(by * 8 + row) * geo.W8 +
                                                 bx * 8 + cc];
                const double c = (double)sm.p[ch ? 2 : 0][by * 8 + row][bx * 8 + cc];
                e.s_yy += y * y;
                e.s_yc += y * c;
                e.s_cc += c * c;
                e.n += 1.0;
              }
          }
        bool unused;
        sd = e.n > 0 ? best_factor(e, ch ? 1.0f : 0.0f, 0, 0, 0, &unused) : 0;
      }
      if ((lane & 7) == 0 && lane < 16) sm.seed[ch] = sd;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    seed[0] = sm.seed[0];
    seed[1] = sm.seed[1];
  } else {
    fetch(a.dyhf, sm.p[1]);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
  }
  // (3) Residual bits of every candidate through the DCT8x8 baseline quantizer
  // (cells folded onto the 8x8 grid, lib.rs:3585), then the choice.
  // lib.rs:3735 factor_candidates(seed, -128, 127): seed-1, seed, seed+1
  // clamped and de-duplicated, then 0 if absent (every thread forms both).
  if (seed[0] != 0 || seed[1] != 0) {
    int cands[2][4], ncand[2];
#pragma unroll
    for (int ch = 0; ch < 2; ++ch) {
      int nc = 0;
      for (int d = -1; d <= 1; ++d) {
        int v = min(max(seed[ch] + d, -128), 127);
        bool dup = false;
        for (int i = 0; i < nc; ++i) dup |= cands[ch][i] == v;
        if (!dup) cands[ch][nc++] = v;
      }
      bool has0 = false;
      for (int i = 0; i < nc; ++i) has0 |= cands[ch][i] == 0;
      if (!has0) cands[ch][nc++] = 0;
      ncand[ch] = nc;
    }
    uint32_t bits[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
    float kx[4], kb[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      kx[i] = 0.0f + (float)cands[0][i < ncand[0] ? i : 0] / 84.0f;
      kb[i] = 1.0f + (float)cands[1][i < ncand[1] ? i : 0] / 84.0f;
    }
    // lanes by frequency: a warp takes the same four of eight columns of each
    // block, so that its cells fall under the threshold together
    const int col = t % 8 * 8 + t / 8 % 8;
    if (col < pw)
#pragma unroll 1
      for (int row = row0; row < ph; row += kStep) {
        const int l = sm.lg[(row >> 3) * 8 + (col >> 3)], mask = (8 << l) - 1;
        if ((col & mask) < (1 << l) && (row & mask) < (1 << l)) continue;  // LLF
        const int cell8 = ((row & mask) >> l) * 8 + ((col & mask) >> l);
        const float x = sm.p[0][row][col], b = sm.p[2][row][col], dy = sm.p[1][row][col];
        const float step_x = sm.step[0][cell8], rstep_x = sm.rstep[0][cell8];
        const float step_b = sm.step[1][cell8], rstep_b = sm.rstep[1][cell8];
        auto cost = [&](int ch, float v, const float* k, float step, float rstep, float half) {
          bool ok = true;
          uint32_t n[4];
          float target[4];
          bool zeros = true;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            target[c] = v - k[c] * dy;
            zeros = zeros && fabsf(target[c]) <= half;
          }
          if (zeros) return;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const Choice q(ch, target[c], step, rstep);
            ok = ok && q.ok;
            n[c] = q.bits();
          }
          if (!ok)
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              float rc;
              n[c] = residual_bits(
                  choose_general(target[c], step, c_quant_bias[ch], a.err, &rc));
            }
#pragma unroll
          for (int c = 0; c < 4; ++c) bits[ch / 2][c] += n[c];
        };
        if (seed[0] != 0) cost(0, x, kx, step_x, rstep_x, sm.half[0][cell8]);
        if (seed[1] != 0) cost(2, b, kb, step_b, rstep_b, sm.half[1][cell8]);
      }
    // Integer sums, exact in any order.  A tile holds at most 4096 cells of at
    // most 22 bits, so 32 bits suffice.
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const uint32_t v = __reduce_add_sync(0xffffffffu, bits[q / 4][q % 4]);
      if (lane == 0) sm.bits[warp][q] = v;
    }
    __syncthreads();
    if (lane == 0 && warp < 2) {
      const int ch = warp;
      uint32_t tot[4];
      for (int c = 0; c < 4; ++c) {
        tot[c] = 0;
        for (int i = 0; i < THREADS / 32; ++i) tot[c] += sm.bits[i][ch * 4 + c];
      }
      int result = 0;
      if (seed[ch] != 0) {
        // lib.rs:3966 refine_hf_factor: cost(0) first, then each non-zero
        // candidate needs residual + factor bits strictly below (ties to the
        // smaller magnitude).
        unsigned long long best_cost = 0;
        for (int c = 0; c < ncand[ch]; ++c)
          if (cands[ch][c] == 0) best_cost = tot[c];
        int best_f = 0;
        for (int c = 0; c < ncand[ch]; ++c) {
          int f = cands[ch][c];
          if (f == 0) continue;
          unsigned long long fb = factor_bits(f);
          unsigned long long cutoff = best_cost > fb ? best_cost - fb : 0;
          if (tot[c] > cutoff) continue;
          unsigned long long cost = tot[c] + fb;
          int af = f < 0 ? -f : f, ab = best_f < 0 ? -best_f : best_f;
          if (cost < best_cost || (cost == best_cost && af < ab)) {
            best_cost = cost;
            best_f = f;
          }
        }
        result = best_f;
      }
      sm.factor[ch] = result;
    }
  } else if (t < 2) {
    sm.factor[t] = 0;
  }
  __syncthreads();
  if (t < 2) (t == 0 ? a.cfl_x : a.cfl_b)[tile] = (int8_t)sm.factor[t];
  // (4) K5 — the HF half of lib.rs:3237 quantize_square_varblock for chroma:
  // targets c - k*dY (no FMA), nearest choice; the LLF corners stay zero.
  if (col >= pw) return;
  const float k_x = 0.0f + (float)sm.factor[0] / 84.0f, k_b = 1.0f + (float)sm.factor[1] / 84.0f;
  const float qm_x = a.qs.qm[0], qm_b = a.qs.qm[2];
#pragma unroll 2
  for (int row = row0; row < ph; row += kStep) {
    const int blk = (row >> 3) * 8 + (col >> 3);
    const int l = sm.lg[blk], mask = (8 << l) - 1, k = row & mask, j = col & mask;
    int32_t qx = 0, qb = 0;
    if (!(k < (1 << l) && j < (1 << l))) {
      const float mul = sm.mul[blk], dy = sm.p[1][row][col];
      const float* m = a.dq + dq_offset(l) + (k << (3 + l)) + j;  // slots 0, 1, 2: the squares
      const float step_x = mul * qm_x * __ldg(m);
      const float step_b = mul * qm_b * __ldg(m + 2 * kDequantTableFloats);
      const float vx = sm.p[0][row][col] - k_x * dy, vb = sm.p[2][row][col] - k_b * dy;
      const float inf = __int_as_float(0x7f800000);
      const bool zeros = step_x > 0.0f && step_x < inf && step_b > 0.0f && step_b < inf &&
                         fabsf(vx) <= 0.5f * c_quant_bias[0] * step_x &&
                         fabsf(vb) <= 0.5f * c_quant_bias[2] * step_b;
      if (!zeros) {
        const Choice cx(0, vx, step_x, approx_rcp(step_x)), cb(2, vb, step_b, approx_rcp(step_b));
        qx = cx.q(vx);
        qb = cb.q(vb);
        if (!(cx.ok && cb.ok)) {
          float rc;
          qx = choose_general(vx, step_x, c_quant_bias[0], a.err, &rc);
          qb = choose_general(vb, step_b, c_quant_bias[2], a.err, &rc);
        }
      }
    }
    const size_t ci = origin + (size_t)row * geo.W8 + col;
    a.qcoeff[ci] = qx;
    a.qcoeff[2 * cplane + ci] = qb;
  }
}

// Frame-wide LF pair (lib.rs:3831 refine_lf_factors) and the chroma LF in
// three kernels: the regression sums of every LF sample as per-CTA
// double-float partials across the GPU; the two seeds, which every CTA forms
// from the partials (with the sequential fallback in the reference's LF-group
// / band / varblock / cell order when a seed is not robust), and the residual
// bit costs of both candidate windows as per-CTA partials; the joint choice,
// which every CTA makes from those, and the LF half of lib.rs:3237 for X and
// B against it.  Forming a small sum again in each CTA costs less than the
// launches of single-CTA kernels between.
constexpr int kLfThreads = 256;

__device__ void lf_candidates(int seed, int* c, int* nc_out) {
  int nc = 0;
  for (int d = -1; d <= 1; ++d) {
    int v = min(max(seed + d, -128), 127);
    bool dup = false;
    for (int i = 0; i < nc; ++i) dup |= c[i] == v;
    if (!dup) c[nc++] = v;
  }
  bool has0 = false;
  for (int i = 0; i < nc; ++i) has0 |= c[i] == 0;
  if (!has0) c[nc++] = 0;
  *nc_out = nc;
}

__device__ __forceinline__ bool cfl_off(const EncArgs& a) {
  return *a.not_gray == 0u || !a.cfl_enabled;
}

// Partial sums per CTA: [kLfCtas][7] double-float (yy, yx, xx, yb, bb, |yx|, |yb|).
__global__ void __launch_bounds__(kLfThreads) k_cfl_lf_sums(EncArgs a, DF* part) {
  __shared__ DF s_w[kLfThreads / 32][7];
  if (cfl_off(a)) return;
  const size_t nb = (size_t)a.geo.bw * a.geo.bh;
  DF v[7] = {};
  for (size_t i = (size_t)blockIdx.x * kLfThreads + threadIdx.x; i < nb;
       i += (size_t)kLfCtas * kLfThreads) {
    const float y = a.lfs[nb + i], x = a.lfs[i], b = a.lfs[2 * nb + i];
    v[0] = df_add(v[0], df_two_prod(y, y));
    v[1] = df_add(v[1], df_two_prod(y, x));
    v[2] = df_add(v[2], df_two_prod(x, x));
    v[3] = df_add(v[3], df_two_prod(y, b));
    v[4] = df_add(v[4], df_two_prod(b, b));
    v[5].hi += fabsf(y * x);
    v[6].hi += fabsf(y * b);
  }
  const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
#pragma unroll
  for (int q = 0; q < 7; ++q) {
    DF t = df_warp_sum(v[q]);
    if (lane == 0) s_w[wid][q] = t;
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    DF t = s_w[0][threadIdx.x];
    for (int i = 1; i < kLfThreads / 32; ++i) t = df_add(t, s_w[i][threadIdx.x]);
    part[blockIdx.x * 7 + threadIdx.x] = t;
  }
}

// The seeds from the partial sums, by a whole CTA (all of it calls); the
// first CTA counts a fallback.
__device__ void cfl_lf_seeds(const EncArgs& a, const DF* part, int seeds[2]) {
  __shared__ double s_t[8];
  __shared__ int s_seed[2];
  const Geo& geo = a.geo;
  const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
  if (wid < 7) {
    DF t = part[lane * 7 + wid];
    for (int c = lane + 32; c < kLfCtas; c += 32) t = df_add(t, part[c * 7 + wid]);
    t = df_warp_sum(t);
    if (lane == 0) s_t[wid] = df_value(t);
  }
  __syncthreads();
  const size_t nb = (size_t)geo.bw * geo.bh;
  if (wid == 0) {
    const double* t = s_t;
    const double n = (double)nb;
    const double gam = 2.0 * (n + 64.0) * (2.2737367544323206e-13 + 1.1102230246251565e-16);
    const int ch = lane >> 3 & 1;
    const RegSums r{t[0], ch ? t[3] : t[1], ch ? t[4] : t[2], ch ? t[6] : t[5], n};
    bool robust;
    int seed = best_factor_lanes(0xffffffffu, lane & 7, r, ch ? 1.0f : 0.0f, gam * r.s_yy,
                                 gam * r.a_yc, gam * r.s_cc, &robust);
    if (__any_sync(0xffffffffu, !robust)) {
      if (blockIdx.x == 0 && lane == 0) atomicAdd(a.cfl_fallbacks, 1u);
      if ((lane & 7) == 0 && lane < 16) {
        RegSums e{0, 0, 0, 0, n};
        const int G = 256;
        const int gw = (geo.bw + G - 1) / G, gh = (geo.bh + G - 1) / G;
        for (int gy = 0; gy < gh; ++gy)
          for (int gx = 0; gx < gw; ++gx) {
            int by0 = gy * G, bx0 = gx * G;
            int gbh = min(G, geo.bh - by0), gbw = min(G, geo.bw - bx0);
            for (int trow = 0; trow < (gbh + 7) / 8; ++trow)
              for (int by = by0 + trow * 8; by < min(by0 + trow * 8 + 8, by0 + gbh); ++by)
                for (int bx = bx0; bx < bx0 + gbw; ++bx) {
                  uint8_t m = a.block_map[(size_t)by * geo.bw + bx];
                  if (!(m & 0x80)) continue;
                  int sel = m & 0x1f, nbk = sel == 0 ? 1 : (sel == 4 ? 2 : 4);
                  for (int i = 0; i < nbk * nbk; ++i) {
                    size_t bi = (size_t)(by + i / nbk) * geo.bw + bx + i % nbk;
                    double y = a.lfs[nb + bi], c = a.lfs[(ch ? 2 * nb : 0) + bi];
                    e.s_yy += y * y;
                    e.s_yc += y * c;
                    e.s_cc += c * c;
                  }
                }
          }
        bool unused;
        seed = best_factor(e, ch ? 1.0f : 0.0f, 0, 0, 0, &unused);
      }
    }
    if ((lane & 7) == 0 && lane < 16) s_seed[ch] = seed;
  }
  __syncthreads();
  seeds[0] = s_seed[0];
  seeds[1] = s_seed[1];
}

// Residual bits of every candidate per CTA: [kLfCtas][8] (X candidates 0..3,
// B candidates 0..3).  At most 2^16 * 22 bits per CTA fit in 32 bits for
// frames up to 2^28 LF samples.
__global__ void __launch_bounds__(kLfThreads) k_cfl_lf_bits(EncArgs a, const DF* sums,
                                                            int* seeds_out, uint32_t* part) {
  __shared__ uint32_t s_w[kLfThreads / 32][8];
  if (cfl_off(a)) return;
  const size_t nb = (size_t)a.geo.bw * a.geo.bh;
  int seeds[2];
  cfl_lf_seeds(a, sums, seeds);
  if (blockIdx.x == 0 && threadIdx.x < 2) seeds_out[threadIdx.x] = seeds[threadIdx.x];
  int cand[2][4], ncand[2];
  lf_candidates(seeds[0], cand[0], &ncand[0]);
  lf_candidates(seeds[1], cand[1], &ncand[1]);
  uint32_t bits[8] = {};
  float k[2][4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    k[0][c] = 0.0f + (float)cand[0][c < ncand[0] ? c : 0] / 84.0f;
    k[1][c] = 1.0f + (float)cand[1][c < ncand[1] ? c : 0] / 84.0f;
  }
  for (size_t i = (size_t)blockIdx.x * kLfThreads + threadIdx.x; i < nb;
       i += (size_t)kLfCtas * kLfThreads) {
    const float dy = a.dylf[i], x = a.lfs[i], b = a.lfs[2 * nb + i];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (c < ncand[0]) bits[c] += residual_bits(lf_quantize(x - k[0][c] * dy, a.qs.m_dc[0], a.err));
      if (c < ncand[1]) bits[4 + c] += residual_bits(lf_quantize(b - k[1][c] * dy, a.qs.m_dc[2], a.err));
    }
  }
  const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    uint32_t t = bits[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) s_w[wid][q] = t;
  }
  __syncthreads();
  if (threadIdx.x < 8) {
    uint32_t t = 0;
    for (int i = 0; i < kLfThreads / 32; ++i) t += s_w[i][threadIdx.x];
    part[blockIdx.x * 8 + threadIdx.x] = t;
  }
}

// The joint choice (every CTA, from the partial costs), then the LF half of
// lib.rs:3237 quantize_square_varblock for X and B: targets c - k_lf*dY_lf.
__global__ void __launch_bounds__(kLfThreads) k_cfl_lf_quant(EncArgs a, const int* seeds,
                                                             const uint32_t* part) {
  __shared__ unsigned long long s_cost[8];
  __shared__ int s_factor[2];
  const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
  if (!cfl_off(a)) {
    static_assert(kLfThreads / 32 == 8, "a warp per candidate cost");
    uint32_t t = 0;  // 2^16 x 22 bits per partial: a lane's four fit
    for (int c = lane; c < kLfCtas; c += 32) t += part[c * 8 + wid];
    unsigned long long v = t;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) s_cost[wid] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      int cand[2][4], ncand[2];
      lf_candidates(seeds[0], cand[0], &ncand[0]);
      lf_candidates(seeds[1], cand[1], &ncand[1]);
      const unsigned long long* cost0 = s_cost;
      const unsigned long long* cost1 = s_cost + 4;
      unsigned long long nx = 0, nbb = 0;
      for (int c = 0; c < ncand[0]; ++c) if (cand[0][c] == 0) { nx = cost0[c]; break; }
      for (int c = 0; c < ncand[1]; ++c) if (cand[1][c] == 0) { nbb = cost1[c]; break; }
      int bx = 0, bbf = 0;
      unsigned long long best = nx + nbb;
      for (int i = 0; i < ncand[0]; ++i)
        for (int j = 0; j < ncand[1]; ++j) {
          int fx = cand[0][i], fb = cand[1][j];
          unsigned long long c = cost0[i] + cost1[j];
          if (fx != 0 || fb != 0) c += 50ull + factor_bits(fx) + factor_bits(fb);
          int mag = abs(fx) + abs(fb), bmag = abs(bx) + abs(bbf);
          if (c < best || (c == best && mag < bmag)) {
            bx = fx;
            bbf = fb;
            best = c;
          }
        }
      s_factor[0] = bx;
      s_factor[1] = bbf;
    }
  } else if (threadIdx.x < 2) {
    s_factor[threadIdx.x] = 0;
  }
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x < 2) a.lf_factors[threadIdx.x] = s_factor[threadIdx.x];
  const float k_x = 0.0f + (float)s_factor[0] / 84.0f, k_b = 1.0f + (float)s_factor[1] / 84.0f;
  const size_t nb = (size_t)a.geo.bw * a.geo.bh;
  for (size_t i = (size_t)blockIdx.x * kLfThreads + threadIdx.x; i < nb;
       i += (size_t)gridDim.x * kLfThreads) {
    const float dy = a.dylf[i];
    a.lfq[i] = lf_quantize(a.lfs[i] - k_x * dy, a.qs.m_dc[0], a.err);
    a.lfq[2 * nb + i] = lf_quantize(a.lfs[2 * nb + i] - k_b * dy, a.qs.m_dc[2], a.err);
  }
}

int launch_fdct_luma(const EncArgs& a, const uint32_t* const* lists, const int* counts,
                     const cudaStream_t* s) {
  // square classes: 0 -> DCT8, 1 -> DCT16, 2 -> DCT32, each on its stream
  int k = 0;
  if (counts[0]) { k_fdct8<false><<<(counts[0] + 15) / 16, 128, 0, s[0]>>>(a, lists[0], counts[0]); ++k; }
  if (counts[1]) { k_fdct_sq<16><<<(counts[1] + 1) / 2, 128, 0, s[1]>>>(a, lists[1], counts[1]); ++k; }
  if (counts[2]) { k_fdct_sq<32><<<counts[2], 256, 0, s[2]>>>(a, lists[2], counts[2]); ++k; }
  return k;
}

int launch_luma_from_image(const EncArgs& a, const uint32_t* const* lists, const int* counts,
                           const cudaStream_t* s) {
  int k = 0;
  if (counts[0]) { k_fdct8<true><<<(counts[0] + 15) / 16, 128, 0, s[0]>>>(a, lists[0], counts[0]); ++k; }
  if (counts[1]) { k_fdct_sq<16, true><<<(counts[1] + 1) / 2, 128, 0, s[1]>>>(a, lists[1], counts[1]); ++k; }
  if (counts[2]) { k_fdct_sq<32, true><<<counts[2], 256, 0, s[2]>>>(a, lists[2], counts[2]); ++k; }
  return k;
}

int launch_cfl_chroma(const EncArgs& a, int* lf_seeds, void* lf_scratch, int num_sms, cudaStream_t s,
                      cudaStream_t lf_s) {
  const dim3 tiles(a.geo.tw, a.geo.th);
  if (a.geo.tw * a.geo.th <= num_sms)
    k_cfl_tile<512><<<tiles, 512, sizeof(CflSmem<512>), s>>>(a);
  else
    k_cfl_tile<256><<<tiles, 256, sizeof(CflSmem<256>), s>>>(a);
  DF* sums = (DF*)lf_scratch;
  uint32_t* bits = (uint32_t*)((char*)lf_scratch + kLfCtas * 7 * sizeof(DF));
  // The LF chain reads only the LF planes: on its own stream.
  k_cfl_lf_sums<<<kLfCtas, kLfThreads, 0, lf_s>>>(a, sums);
  k_cfl_lf_bits<<<kLfCtas, kLfThreads, 0, lf_s>>>(a, sums, lf_seeds, bits);
  const size_t nb = (size_t)a.geo.bw * a.geo.bh;
  const int ctas = (int)std::min<size_t>((nb + kLfThreads - 1) / kLfThreads, kLfCtas);
  k_cfl_lf_quant<<<ctas, kLfThreads, 0, lf_s>>>(a, lf_seeds, bits);
  return 4;
}

__global__ void __launch_bounds__(kMulTableN) k_mul_table(uint32_t global_scale, float* table) {
  fill_mul_table(global_scale, table);
}

void launch_mul_table(uint32_t global_scale, float* table, cudaStream_t s) {
  k_mul_table<<<1, kMulTableN, 0, s>>>(global_scale, table);
}

cudaError_t configure_encode_kernels() {
  auto allow = [](auto* kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  cudaError_t e;
  if ((e = allow(k_precondition<2>, PreTile<2>::kSmem)) != cudaSuccess) return e;
  if ((e = allow(k_precondition<3>, PreTile<3>::kSmem)) != cudaSuccess) return e;
  if ((e = allow(k_precondition<4>, PreTile<4>::kSmem)) != cudaSuccess) return e;
  if ((e = allow(k_precondition<8>, PreTile<8>::kSmem)) != cudaSuccess) return e;
  if ((e = allow(k_cfl_tile<256>, sizeof(CflSmem<256>))) != cudaSuccess) return e;
  return allow(k_cfl_tile<512>, sizeof(CflSmem<512>));
}

void upload_dct_constants(const float* iv4, const float* iv8, const float* iv16,
                          const float* scale_f, cudaStream_t s) {
  cudaMemcpyToSymbolAsync(c_iv4, iv4, sizeof(float) * 16, 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_iv8, iv8, sizeof(float) * 64, 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_iv16, iv16, sizeof(float) * 256, 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_scale_f, scale_f, sizeof(float) * 32, 0, cudaMemcpyHostToDevice, s);
  // 0.145f / q in IEEE single precision, as bias_adjust divides on the device.
  static float quot[kBiasQuotN];
  quot[0] = 0.0f;
  for (int q = 1; q < kBiasQuotN; ++q) quot[q] = 0.145f / (float)q;
  cudaMemcpyToSymbolAsync(g_bias_quot, quot, sizeof quot, 0, cudaMemcpyHostToDevice, s);
  // bias_adjust of q and its neighbours, evaluated as bias_adjust_q does.
  static const float bias[3] = {kQuantBiasX, kQuantBiasY, kQuantBiasB};
  static float4 levels[3][kLevelN];
  for (int c = 0; c < 3; ++c) {
    auto level = [&](int q) {
      return q <= 0 ? 0.0f : (q == 1 ? 1.0f * bias[c] : (float)q - 0.145f / (float)q);
    };
    for (int q = 0; q < kLevelN; ++q) {
        uint32_t packed = 0;
        for (int i = 0; i < 3; ++i) {
          uint32_t m = (uint32_t)std::max(q - 1 + i, 0), n = 0;
          while (m >> n) ++n;
          packed |= (n ? n + 1 : 0) << (8 * i);  // residual_bits
        }
        float w;
        std::memcpy(&w, &packed, sizeof w);
        levels[c][q] = make_float4(level(q - 1), level(q), level(q + 1), w);
    }
  }
  cudaMemcpyToSymbolAsync(g_levels, levels, sizeof levels, 0, cudaMemcpyHostToDevice, s);
}

}  // namespace jpxlg
