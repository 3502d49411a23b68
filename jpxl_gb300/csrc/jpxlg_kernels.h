// jpxlg_kernels.h — argument blocks and launchers of the sm_103a kernels.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "jpxlg_internal.h"

namespace jpxlg {

struct DF;  // double-float partial sums (jpxlg_common.cuh)

// Everything the encoder kernels read and write (device pointers).
struct EncArgs {
  Geo geo;
  QuantScalars qs;
  const float* pre;          // 3 planes w*h: XYB after the optional precondition
  const float* dq;           // [3][kDequantTableFloats] dequant multipliers
  const float* mul_table;    // [kMulTableN] hf multipliers of this call's global_scale
  const uint32_t* hf_mul;    // per 8x8 block (read at varblock origins)
  const uint8_t* block_map;  // per 8x8 block
  float* coeff;              // [3][W8*H8] forward coefficients (f32)
  float* dyhf;               // [W8*H8] reconstructed luma HF
  int32_t* qcoeff;           // [3][W8*H8] quantized coefficients
  float* lfs;                // [3][bw*bh] LF samples
  float* dylf;               // [bw*bh] reconstructed luma LF
  int32_t* lfq;              // [3][bw*bh] quantized LF
  int8_t* cfl_x;             // [tw*th]
  int8_t* cfl_b;             // [tw*th]
  int* lf_factors;           // [2] frame LF factors, unbiased
  const uint32_t* not_gray;  // set by the colour kernel when any pixel is not grey
  uint32_t cfl_enabled;
  float base_mul;            // hf multiplier of the frame's baseline hf_mul
  uint32_t* err;
  uint32_t* cfl_fallbacks;   // count of sequential-order fallbacks taken
};

// Everything the render kernels read and write.
struct RenderArgs {
  Geo geo;
  QuantScalars qs;
  const float* dq;
  const float* mul_table;    // [kMulTableN] hf multipliers of this call's global_scale
  const uint32_t* hf_mul;
  const uint8_t* sharpness;
  const int32_t* qcoeff;     // [3][W8*H8]
  const int32_t* lfq;        // [3][bw*bh]
  const int8_t* cfl_x;
  const int8_t* cfl_b;
  float k_x_lf, k_b_lf;      // frame LF CfL multipliers
  const int* lf_factors_dev; // when non-null, read the LF factors from here
  float* planes;             // [3][w*h] XYB out
  float* sigma;              // [bw*bh]
  const float* lf_float = nullptr;  // [3][bw*bh] final LF (decoded frames); else from lfq
  uint32_t* err = nullptr;   // device error word
};

// LF of a decoded frame: dequantize, LF CfL and (smooth) adaptive smoothing
// into out [3][bw*bh]; also the table of HF multipliers for global_scale.
void launch_lf_prepare(const int32_t* lfq, int bw, int bh, const float m[3], float div, float kx,
                       float kb, bool smooth, float* out, uint32_t global_scale, float* mul_table,
                       int num_sms, cudaStream_t s);
// A staged stream's block (device or pinned host memory, 16-byte aligned): n
// coefficients of q_bytes each (n a multiple of 64) widened to int32 at dst,
// then `rest` bytes (a multiple of 16) as they are behind them.
void launch_unstage(const void* src, int q_bytes, size_t n, size_t rest, void* dst, int num_sms,
                    cudaStream_t s);
// One finished stream of a batch: its lane's device error word to `flag`, in
// pinned host memory, after everything its stream has written before.
void launch_publish(const uint32_t* err, uint32_t* flag, cudaStream_t s);
void upload_dct64(const float* matrix, cudaStream_t s);
void upload_afv(const double* basis, cudaStream_t s);
// Differences over count floats (count + 2^20 at most 2^32) from bit pattern
// `first`: what 0 and 1 the cube roots, else the output levels of the given
// tables.
void launch_sweep_diag(int what, uint32_t first, uint32_t count, const float* thr,
                       const float* levels, const float4* bracket, int nlev,
                       unsigned long long* wrong, int num_sms, cudaStream_t s);
bool launch_special_diag(int kind, const float* coef, int n, float* out, cudaStream_t s);

// Fills table[h] = hf_multiplier_f64(global_scale, h) for h < kMulTableN.
void launch_mul_table(uint32_t global_scale, float* table, cudaStream_t s);

// Per-device kernel attributes (dynamic shared memory above 48 KB); call once
// per device with it current, before any launch or stream capture.
cudaError_t configure_encode_kernels();
cudaError_t configure_render_kernels();

void upload_dct_constants(const float* iv4, const float* iv8, const float* iv16,
                          const float* scale_f, cudaStream_t s);
// mul_table (or null): also the table of HF multipliers for global_scale.
void launch_srgb_to_xyb(const void* rgb, int bits, size_t n, const float* lut, float* x, float* y,
                        float* b, uint32_t* not_gray, uint32_t global_scale, float* mul_table,
                        int num_sms, cudaStream_t s);
// One launch (the ring of tiles along the frame's rows and columns of other
// rules, then the tiles inside it); returns 1.
int launch_precondition(const float* in, float* out, int w, int h, int num_sms, cudaStream_t s);
// The per-shape-class launchers take one stream per class (s[i] for class
// i), so that independent classes can run side by side.  Each returns the
// number of kernels it launched.
int launch_fdct_luma(const EncArgs& a, const uint32_t* const* lists, const int* counts,
                     const cudaStream_t* s);
// LF CfL partials: kLfCtas CTAs, each 7 double-float sums and 8 bit counts.
constexpr int kLfCtas = 128;
constexpr size_t kCflScratchBytes = (size_t)kLfCtas * (7 * 8 + 8 * 4);
// CfL estimation and the chroma quantization: the tiles' kernel on s, the
// LF factors' chain and the chroma LF on lf_s (it reads only the LF planes);
// the caller joins lf_s back.  Returns the number of kernels.
int launch_cfl_chroma(const EncArgs& a, int* lf_seeds, void* lf_scratch, int num_sms, cudaStream_t s,
                      cudaStream_t lf_s);

void launch_render_varblocks(const RenderArgs& a, const uint32_t* const* lists,
                             const int* counts, const cudaStream_t* s);

// Split-precision transforms on the tensor cores (k_tc.cu), square shape
// classes 0..2 (DCT8, DCT16, DCT32); terms = 2 (BF16x3) or 3 (BF16x6).
// Each returns the number of kernels it launched.  The render form needs
// 16-byte aligned coefficient planes.
cudaError_t configure_tc_kernels();
// Sets the tensor-core kernels' persistent CTAs per SM (in quarters of those
// that fit, 1..4; other values leave it) and returns the previous value.
int tc_ctas_per_sm(int value);
void upload_tc_basis(cudaStream_t s);
int launch_fdct_tc(const EncArgs& a, const uint32_t* const* lists, const int* counts, int terms,
                   int num_sms, const cudaStream_t* s);
int launch_render_tc(const RenderArgs& a, const uint32_t* const* lists, const int* counts,
                     const float* const* llf, int terms, int num_sms, const cudaStream_t* s);
// The LLF rectangles (48 floats per varblock: 3 channels x 16) and the EPF
// sigma of square classes 0..2, for launch_render_tc (k_render.cu).
int launch_llf_sigma(const RenderArgs& a, const uint32_t* const* lists, const int* counts,
                     float* const* llf, const cudaStream_t* s);
// Luma LF and HF quantization of the square varblocks from a coefficient
// image the split-precision forward transform wrote (k_fdct8 and k_fdct_sq without their
// own transform).
int launch_luma_from_image(const EncArgs& a, const uint32_t* const* lists, const int* counts,
                           const cudaStream_t* s);
void launch_gaborish(const float* in, float* out, int w, int h, cudaStream_t s);
void launch_epf_step(int step, const float* in, float* out, const float* sigma, int w, int h,
                     int num_sms, cudaStream_t s);
// out_kind: 1 linear f32 planes, 2 sRGB8 interleaved, 3 linear at depth
// pxyb (optional, out_kind 3 only): also the SSIMULACRA2 positive XYB planes
// of the output pixels.
// bracket (out_kind 3, more than 256 levels): per level (the threshold
// below, the threshold above, the level's value); levels: the levels' values.
void launch_colour_out(const float* xyb, int w, int h, int out_kind, const float* thresholds,
                       const float* levels, const float4* bracket, int nlevels, void* out,
                       float* pxyb, int num_sms, cudaStream_t s);
void upload_render_constants(const float* opsin_m, const float* opsin_bias,
                             const float* opsin_bias_cbrt, cudaStream_t s);

// Cover selection (k_cover.cu).  Shape s: 0 DCT8, 1 DCT16, 2 DCT32;
// candidates of shape s sit at every (1 << s)-aligned block position that
// fits the grid.
struct CoverArgs {
  Geo geo;
  const float* pre;        // 3 planes w*h: the transform frame
  const float* dq;         // [3][kDequantTableFloats]
  float scale[3];          // Mul * qm[c] at the baseline HfMul
  double lambda[3];        // lib.rs:2094 per-channel Lagrange multipliers
  double w[3][3];          // [shape][channel] lambda[c] * side^2
  uint8_t* map;            // block map out (bw*bh)
  uint32_t* fallbacks;     // regions replayed in the reference's order
  uint32_t* err;
};
cudaError_t configure_cover_kernels();
int launch_cover(const CoverArgs& a, cudaStream_t s);

// SSIMULACRA2
struct SsimScale {
  int w, h;
  float* xyb;   // [3][w*h]  (reference side)
  float* mu;    // [3][w*h]
  float* s11;   // [3][w*h]
};
constexpr int kMaxScales = 6;
// The blur's constants (taps, resonators) into constant memory.
void upload_blur_consts(cudaStream_t s);
// Widest frame the row pass stages in shared memory (a line plus its output).
constexpr int kBlurMaxWidth = 8192;
cudaError_t configure_blur_kernels();
// Rows of partial sums one scale writes (one per 32 x 32 tile).
int blur_partial_rows(int w, int h);
// Floats of one row-pass plane (rows padded to a 16-byte pitch).
size_t blur_plane_floats(int w, int h);
// Bytes of one scale's segment states in the column pass's scan buffer, which
// also holds kBlurCarryHeader bytes.  The buffer is zeroed when it is
// allocated and carries its launches' epoch from then on.
constexpr size_t kBlurCarryHeader = 64;
size_t blur_carry_bytes(int w, int h, int nch);
// The pyramid of a linear RGB frame as positive XYB planes: level s
// (ceil-halved s times by 2x2 means, edge replicated) into xyb[s], levels
// 1 .. n-1, and level 0 where xyb[0] is not null.
struct PyramidOut {
  float* xyb[kMaxScales];
};
void launch_pyramid(const float* rgb, int w, int h, const PyramidOut& out, int n, cudaStream_t s);
// One scale of the blur: positive XYB x (the candidate's, or the reference's
// own for its moments), the reference's r, and mu and sigma11 (written by
// launch_ref_moments, read by launch_score_scales).
struct BlurScale {
  int w, h;
  const float* x;  // [3][w*h]
  const float* r;  // [3][w*h]
  float* mu;       // [3][w*h]
  float* s11;      // [3][w*h]
  DF* partial;     // blur_partial_rows rows of 18 sums (scoring only)
};
// Reference side of every scale: mu = blur(x), s11 = blur(x * x) per channel;
// hpl (6 row-pass planes per scale) and carry (blur_carry_bytes, summed, plus
// the header) are scratch; a column-scan wait that runs out raises
// kDevBlurTimeout in err.  Two launches: the row pass, the column pass.
void launch_ref_moments(const BlurScale* scales, int n, float* hpl, void* carry, uint32_t* err,
                        cudaStream_t s);
// Candidate side of every scale for channels c0 .. c0+nch-1; hpl (3 * nch
// row-pass planes per scale) and carry are scratch; each scale's partial
// receives one row of 18 double-float sums (8 bytes each) per 32 x 32 tile,
// each channel filling its six.  Returns the number of launches (two).
// The hook is called between the launches when the caller times them: part 0
// before the row pass, 1 after it, 2 before the column pass, 3 after it.
using ScaleHook = void (*)(void* user, int part);
int launch_score_scales(const BlurScale* scales, int n, int c0, int nch, float* hpl, void* carry,
                        uint32_t* err, cudaStream_t s, ScaleHook hook = nullptr,
                        void* user = nullptr);
// The per-scale sums, then the score, in one launch; returns 1.  The sums
// overwrite row 0 of each scale's partial rows; `carry` is the buffer that
// launch_score_scales used.  out receives the score, the raw error and the
// terms; score and raw (each may be null) the first two as well.
int launch_score_finish(DF* partials, const int* ctas_per_scale, int nscales,
                        const int* pixels_per_scale, void* carry, double* out, double* score,
                        double* raw, cudaStream_t s);
// The word of a scan buffer's header that counts finished CTAs.
uint32_t* blur_ticket(void* carry);
// Leaves counts in the header as calls that raced on the buffer may.
cudaError_t blur_disturb(void* carry, cudaStream_t s);

}  // namespace jpxlg
