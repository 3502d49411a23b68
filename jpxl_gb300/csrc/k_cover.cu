// k_cover.cu — sm_103a kernel of the encoder's cover selection
// (jpxl-encode-policy lib.rs:5260 select_blocks, :5115 tile_region_with,
// :4909 block_cost_bounded, :4685 score_channel_lanes) for a fixed quantizer
// with adaptive quantization off and the Legacy rate model.
//
// C1 k_cover, one CTA per 32x32 region:
//   * the region's three planes into shared memory;
//   * the forward DCTs of its 1 + 4 + 16 square candidates, a warp per strip
//     of 32 columns (one channel, one row of blocks), which transforms the
//     columns, then the rows in place, without a CTA barrier;
//   * every candidate's non-LLF cells quantized (X and B against neutral
//     chroma-from-luma, B minus Y's reconstruction), a thread taking a cell's
//     three channels: residual bits (exact), each channel's squared error in
//     double-float;
//   * the quadtree (DCT8 / DCT16 / DCT32, ties keep the split) on those
//     costs, a lane per block.
//
// The reference accumulates each candidate's weighted error in f64, cell by
// cell in row order, and prunes a merge once the running cost reaches the
// split's.  The kernel sums in a fixed tree order instead and carries a bound
// on the distance between the two sums (all terms are non-negative) through
// every comparison, and a region whose comparisons are not all settled by the
// bound is replayed in the reference's own order (sequential f64, row-wise
// pruning) from the candidates' coefficients.  Replays are counted.
#include <cstdint>

#include "jpxlg_common.cuh"
#include "jpxlg_internal.h"
#include "jpxlg_kernels.h"
#include "jpxlg_quant.cuh"

namespace jpxlg {

// Shape s: 0 DCT8 (1 block), 1 DCT16 (2x2), 2 DCT32 (4x4).
__host__ __device__ constexpr int cover_blocks(int s) { return 1 << s; }

constexpr int kCoverSide = 32;            // region side in samples
constexpr int kCoverPitch = kCoverSide + 1;
constexpr int kCoverWarps = 8;
constexpr int kCoverThreads = 32 * kCoverWarps;

// The cost of one candidate, or of a part of it.
struct CoverSums {
  uint32_t bits;
  DF sse[3];
};

struct CoverSmem {
  float src[3][kCoverSide][kCoverPitch];
  float coef[3][3][kCoverSide][kCoverPitch];  // [shape][channel], a candidate at its place
  CoverSums s8[16], s16[4][2], s32[kCoverWarps];
};

__device__ __forceinline__ int cover_dq(int s) {
  return dq_offset(dq_slot(s == 0 ? 0 : (s == 1 ? 4 : 5)));
}

// Forward DCT_2D of the N x N candidates along a strip: row of blocks `row`
// of channel c.  Lane l transforms column l, then row l % N of block l / N
// (dct_1d's order); the strip is this warp's alone.
template <int N>
__device__ __forceinline__ void cover_strip(CoverSmem& sm, int c, int row, int lane) {
  constexpr int S = N == 8 ? 0 : (N == 16 ? 1 : 2);
  float (*out)[kCoverPitch] = sm.coef[S][c];
  const int y0 = row * N, x0 = lane / N * N, j = lane % N;
  float v[N];
#pragma unroll
  for (int r = 0; r < N; ++r) v[r] = sm.src[c][y0 + r][lane];
  dct_1d<N>(v);
#pragma unroll
  for (int r = 0; r < N; ++r) out[y0 + r][lane] = v[r];
  __syncwarp();
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = out[y0 + j][x0 + k];
  dct_1d<N>(v);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < N; ++k) out[y0 + k][x0 + j] = v[k];
}

// The sums of `count` cells a lane of the shape-s candidate at sample
// (x0, y0): cells first + lane, first + lane + 32, ...
__device__ __forceinline__ void cover_cells(const CoverArgs& a, const CoverSmem& sm, int s, int x0,
                                            int y0, int first, int count, int lane,
                                            CoverSums* out) {
  const int lg = 3 + s, n = 1 << s;
  const float* m = a.dq + cover_dq(s);
  uint32_t bits = 0;
  DF sse[3] = {};
#pragma unroll 1
  for (int i = 0; i < count; ++i) {
    const int cell = first + lane + 32 * i, k = cell >> lg, j = cell & ((1 << lg) - 1);
    if (k < n && j < n) continue;
    float ry = 0.0f;
    // Channels in the reference's scoring order: Y (its reconstruction feeds
    // B's targets), X, B.
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      const int c = o == 0 ? 1 : (o == 1 ? 0 : 2);
      const float v = sm.coef[s][c][y0 + k][x0 + j];
      const float target = c == 1 ? v : (c == 0 ? v - 0.0f * ry : v - 1.0f * ry);
      const float step = a.scale[c] * __ldg(&m[c * kDequantTableFloats + cell]);
      float recon;
      const int32_t q = choose(c, target, step, a.err, &recon);
      if (c == 1) ry = recon;
      bits += residual_bits(q);
      const float d = recon - target;
      sse[c] = df_add(sse[c], df_two_prod(d, d));
    }
  }
  bits = __reduce_add_sync(0xffffffffu, bits);
#pragma unroll
  for (int c = 0; c < 3; ++c) sse[c] = df_warp_sum(sse[c]);
  if (lane == 0) {
    out->bits = bits;
#pragma unroll
    for (int c = 0; c < 3; ++c) out->sse[c] = sse[c];
  }
}

// A cost with a bound on its distance from the reference's f64 value.
struct Cost {
  double v, e;
};

// The shape-s candidate's cost from its parts.
__device__ __forceinline__ Cost cover_rd(const CoverArgs& a, int s, const CoverSums* parts, int n) {
  uint32_t bits = 0;
  DF sse[3] = {};
  for (int i = 0; i < n; ++i) {
    bits += parts[i].bits;
#pragma unroll
    for (int c = 0; c < 3; ++c) sse[c] = df_add(sse[c], parts[i].sse[c]);
  }
  double t = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) t += a.w[s][c] * df_value(sse[c]);
  // At most 3 x 1024 non-negative terms: the double-float tree sums lie
  // within cells x 2^-44 of the exact sum, the reference's sequential f64
  // sum within cells x 2^-53, and the products by w and the three-channel
  // sum add a few 2^-53 more; 2^-40 per term covers all of it with margin.
  const double eps = (3.0 * 1024.0 + 64.0) * 9.094947017729282e-13;  // 2^-40
  return {(double)bits + t, eps * t + 1e-300};
}

// A few ulps of an f64 sum of four values.
__device__ __forceinline__ double sum_slack(double v) { return 8.0 * 1.1102230246251565e-16 * fabs(v); }

// A node of the quadtree: whether the single candidate replaces its split.
// *settled turns false when the bounds leave a comparison open.
__device__ __forceinline__ Cost cover_merge(const Cost& split, bool fits, const Cost& rd,
                                            bool* merged, bool* settled) {
  *merged = false;
  if (!fits) return split;
  const double fixed = 34.0 + 0.0;
  if (fabs(fixed - split.v) <= split.e) {
    *settled = false;
    return split;
  }
  if (fixed >= split.v) return split;
  const Cost single{rd.v + fixed, rd.e + sum_slack(rd.v + fixed)};
  // Reference: kept only if not pruned (rd < split - fixed) and
  // single < split; both are this comparison up to rounding.
  if (fabs(single.v - split.v) <= single.e + split.e) *settled = false;
  if (!(single.v < split.v)) return split;
  *merged = true;
  return single;
}

// The four children's costs in order (of the group of lanes `first`,
// first + step, ...), as the reference adds them up.
__device__ __forceinline__ Cost cover_split(const Cost& mine, int first, int step) {
  Cost split{0.0, 0.0};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    split.v += __shfl_sync(0xffffu, mine.v, first + step * i);
    split.e += __shfl_sync(0xffffu, mine.e, first + step * i);
  }
  split.e += sum_slack(split.v);
  return split;
}

// ---- the reference's own order, for regions the bound does not settle ----

// lib.rs:4685 for one channel of a candidate: rows, non-LLF columns, f64
// accumulation cell by cell, the cutoff tested after each row.  B's targets
// subtract Y's reconstruction, recomputed cell by cell.  (x0, y0): the
// candidate's first sample in the region.
__device__ bool exact_channel(const CoverArgs& a, const CoverSmem& sm, int s, int x0, int y0, int c,
                              double cutoff, bool has_cutoff, uint64_t* bits, double* sse) {
  const int N = 8 << s, n = 1 << s;
  const float* m = a.dq + c * kDequantTableFloats + cover_dq(s);
  const float* my = a.dq + kDequantTableFloats + cover_dq(s);
  const double flat_weight = a.lambda[c] * ((double)(N * N) * 1.0);
  for (int row = 0; row < N; ++row) {
    for (int col = row < n ? n : 0; col < N; ++col) {
      float target = sm.coef[s][c][y0 + row][x0 + col];
      if (c != 1) {
        float ry;
        choose(1, sm.coef[s][1][y0 + row][x0 + col], a.scale[1] * my[row * N + col], nullptr, &ry);
        target = c == 0 ? target - 0.0f * ry : target - 1.0f * ry;
      }
      float recon;
      const int32_t q = choose(c, target, a.scale[c] * m[row * N + col], nullptr, &recon);
      *bits += residual_bits(q);
      const double d = (double)(recon - target);
      *sse += flat_weight * (d * d);
    }
    if (has_cutoff && (double)*bits * 1.0 + *sse >= cutoff) return false;
  }
  return true;
}

__device__ bool exact_cost(const CoverArgs& a, const CoverSmem& sm, int s, int x0, int y0,
                           double cutoff, bool has_cutoff, double* cost) {
  uint64_t bits = 0;
  double sse = 0.0;
  if (!exact_channel(a, sm, s, x0, y0, 1, cutoff, has_cutoff, &bits, &sse)) return false;
  if (!exact_channel(a, sm, s, x0, y0, 0, cutoff, has_cutoff, &bits, &sse)) return false;
  if (!exact_channel(a, sm, s, x0, y0, 2, cutoff, has_cutoff, &bits, &sse)) return false;
  *cost = (double)bits * 1.0 + sse;
  return true;
}

// The node of `size` blocks at block (bx, by) of a region with nx x ny blocks
// inside the grid; bit y*4+x of pick[s] marks a chosen shape-s varblock.
__device__ double exact_node(const CoverArgs& a, const CoverSmem& sm, int bx, int by, int size,
                             int nx, int ny, uint32_t* pick) {
  if (bx >= nx || by >= ny) return 0.0;
  if (size == 1) {
    double rd = 0.0;
    exact_cost(a, sm, 0, 8 * bx, 8 * by, 0.0, false, &rd);
    pick[0] |= 1u << (4 * by + bx);
    return rd + 2.0 + 0.0;
  }
  const int half = size / 2;
  uint32_t below[3] = {0, 0, 0};
  double split = 0.0;
  const int qx[4] = {bx, bx + half, bx, bx + half}, qy[4] = {by, by, by + half, by + half};
  for (int i = 0; i < 4; ++i) split += exact_node(a, sm, qx[i], qy[i], half, nx, ny, below);
  if (bx + size <= nx && by + size <= ny) {
    const double fixed = 34.0 + 0.0;
    const int s = size == 2 ? 1 : 2;
    double rd;
    if (!(fixed >= split) &&
        exact_cost(a, sm, s, 8 * bx, 8 * by, split - fixed, true, &rd) && rd + fixed < split) {
      pick[s] |= 1u << (4 * by + bx);
      return rd + fixed;
    }
  }
  for (int s = 0; s < 3; ++s) pick[s] |= below[s];
  return split;
}

// Bound: issue slots and the quantizer's latency (three shapes, three
// channels a cell).  Measured at 1536x1024: 402 us as three scoring kernels
// (the DCT32 one 136, 32 cells a thread and channel) and one thread of serial
// f64 per region (170, twelve CTAs); 104 us now of the call's 182 (112 by
// itself, from a cold cache), nothing but the map in memory.  Four CTAs an SM
// spill some of the DCT32's registers and are still faster than three or two
// (the whole call as it was then: 217, 221, 241 us).
__global__ void __launch_bounds__(kCoverThreads, 4) k_cover(const __grid_constant__ CoverArgs a) {
  extern __shared__ __align__(16) unsigned char cover_smem[];
  CoverSmem& sm = *reinterpret_cast<CoverSmem*>(cover_smem);
  const Geo& geo = a.geo;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int bx0 = 4 * blockIdx.x, by0 = 4 * blockIdx.y;
  const int nx = min(4, geo.bw - bx0), ny = min(4, geo.bh - by0);  // blocks inside the grid
  {
    const size_t plane = (size_t)geo.w * geo.h;
    const int gx = min(8 * bx0 + lane, geo.w - 1);
#pragma unroll
    for (int i = 0; i < 3 * kCoverSide / kCoverWarps; ++i) {
      const int r = warp + kCoverWarps * i, c = r / kCoverSide, y = r % kCoverSide;
      sm.src[c][y][lane] =
          __ldg(a.pre + plane * c + (size_t)min(8 * by0 + y, geo.h - 1) * geo.w + gx);
    }
  }
  __syncthreads();
  // 3 DCT32, 6 DCT16 and 12 DCT8 strips.
#pragma unroll 1
  for (int t = warp; t < 21; t += kCoverWarps) {
    if (t < 3) cover_strip<32>(sm, t, 0, lane);
    else if (t < 9) cover_strip<16>(sm, (t - 3) % 3, (t - 3) / 3, lane);
    else cover_strip<8>(sm, (t - 9) % 3, (t - 9) / 3, lane);
  }
  __syncthreads();
  // A warp's share: two DCT8 candidates, half a DCT16, an eighth of the
  // DCT32 (candidates that do not fit the grid are never read).
#pragma unroll 1
  for (int t = 0; t < 4; ++t) {
    if (t < 2) {
      const int i = 2 * warp + t, x = 2 * (i >> 2 & 1) + (i & 1), y = 2 * (i >> 3) + (i >> 1 & 1);
      if (x < nx && y < ny) cover_cells(a, sm, 0, 8 * x, 8 * y, 0, 2, lane, &sm.s8[i]);
    } else if (t == 2) {
      const int q = warp >> 1, x = 2 * (q & 1), y = 2 * (q >> 1);
      if (x + 2 <= nx && y + 2 <= ny)
        cover_cells(a, sm, 1, 8 * x, 8 * y, 128 * (warp & 1), 4, lane, &sm.s16[q][warp & 1]);
    } else if (nx == 4 && ny == 4) {
      cover_cells(a, sm, 2, 0, 0, 128 * warp, 4, lane, &sm.s32[warp]);
    }
  }
  __syncthreads();
  // The quadtree, lane i for block i in child order (quad i / 4, child i % 4).
  if (threadIdx.x >= 16) return;
  const int i = lane, q = i >> 2;
  const int qx = 2 * (q & 1), qy = 2 * (q >> 1), x = qx + (i & 1), y = qy + (i >> 1 & 1);
  const bool inside = x < nx && y < ny;
  bool settled = true;
  Cost c8{0.0, 0.0};
  if (inside) {
    const Cost rd = cover_rd(a, 0, &sm.s8[i], 1);
    c8 = {rd.v + 2.0 + 0.0, rd.e + sum_slack(rd.v + 2.0)};
  }
  const bool fits16 = qx + 2 <= nx && qy + 2 <= ny, fits32 = nx == 4 && ny == 4;
  bool merged16 = false, merged32 = false;
  Cost c16 = cover_split(c8, 4 * q, 1);
  if (qx < nx && qy < ny)
    c16 = cover_merge(c16, fits16, fits16 ? cover_rd(a, 1, sm.s16[q], 2) : Cost{0.0, 0.0},
                      &merged16, &settled);
  else
    c16 = {0.0, 0.0};
  const Cost c32 = cover_split(c16, 0, 4);
  cover_merge(c32, fits32, fits32 ? cover_rd(a, 2, sm.s32, kCoverWarps) : Cost{0.0, 0.0},
              &merged32, &settled);
  int shape = merged32 ? 2 : (merged16 ? 1 : 0);
  if (__any_sync(0xffffu, !settled)) {
    uint32_t pick[3] = {0, 0, 0};
    if (lane == 0) {
      atomicAdd(a.fallbacks, 1u);
      exact_node(a, sm, 0, 0, 4, nx, ny, pick);
    }
    const uint32_t p1 = __shfl_sync(0xffffu, pick[1], 0), p2 = __shfl_sync(0xffffu, pick[2], 0);
    shape = p2 ? 2 : (p1 >> (4 * qy + qx) & 1u ? 1 : 0);
  }
  if (inside) {
    const bool origin = shape == 0 || (shape == 1 ? (i & 3) == 0 : i == 0);
    const uint8_t sel = shape == 0 ? 0 : (shape == 1 ? 4 : 5);
    a.map[(size_t)(by0 + y) * geo.bw + bx0 + x] = (uint8_t)(sel | (origin ? 0x80 : 0));
  }
}

cudaError_t configure_cover_kernels() {
  return cudaFuncSetAttribute(k_cover, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)sizeof(CoverSmem));
}

int launch_cover(const CoverArgs& a, cudaStream_t s) {
  const dim3 regions((a.geo.bw + 3) / 4, (a.geo.bh + 3) / 4);
  k_cover<<<regions, kCoverThreads, sizeof(CoverSmem), s>>>(a);
  return 1;
}

}  // namespace jpxlg
