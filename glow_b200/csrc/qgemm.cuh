// Internal interface of the int8 contraction core (qgemm.cu), shared with the convolution
// front end (conv.cu).
#pragma once
#include "common.cuh"

namespace glowb200 {

// Where a layer's result goes when it is the input of a convolution that wants its padding made real (conv.cu): straight
// into that padded buffer, whose halo the epilogue warps fill beside it.  kind 1: [images, hp, wp, N], pixel (y, x) of an
// image at (y + top, x + left); kind 2: the same split by the parity of the padded coordinates into four planes
// [images, hp / 2, wp / 2, N].  Rows of the product are the images' h * w pixels.
struct PaddedOut {
  int kind;  // 0: no, the result is a matrix
  int images, h, w, hp, wp, top, left, plane;  // plane: pixels of one of the four
  uint32_t word;                               // of the halo
  // the next layer's filter [filter_rows, kw, 64] -> pairs [filter_rows, ceil(kw / 2), 128] (64 channels; else nullptr)
  const int8_t *filter;
  int8_t *pairs;
  int filter_rows, kw;
#ifdef __CUDACC__
  __device__ __forceinline__ int pixel(int image, int y, int x) const {  // padded coordinates
    if (kind == 1) return (image * hp + y) * wp + x;
    return ((y & 1) * 2 + (x & 1)) * plane + (image * (hp >> 1) + (y >> 1)) * (wp >> 1) + (x >> 1);
  }
#endif
};

struct GemmParams {
  int8_t *out;                // [M, N]
  const int32_t *bias;        // [N] or nullptr (MatMul); int8 values when bias_is_i8 (the _i8_i8 kernels)
  const int32_t *b_offsets;   // weight offsets; index j * stride_b_off
  const int32_t *bias_pre, *bias_post, *bias_scale;  // index j * stride_q
  const int32_t *out_pre, *out_post, *out_scale;      // index j * stride_q
  const int32_t *b_row_sums;  // [N] sum_k B[j,k]; b_sum_parts > 1: as many arrays, whose sum it is
  int b_sum_parts;
  const int32_t *a_row_sums;  // [M] sum_k A[i,k], or nullptr when every b offset is 0
  // The Add of a residual block behind the layer (residual != nullptr): out = add(layer's int8 result,
  // residual[M, N]), rows of whole 16-byte pieces, no weight offsets, activation none or Relu.
  const int8_t *residual;
  AddQuant add;
  PaddedOut padded;  // (the TMA path, rows of whole 16-byte pieces)
  int32_t *status;
  const int32_t *bias_offsets;  // per-column bias offsets (channelwise conv), or nullptr: bias_offset
  int M, N, K;                  // K: row pitch of both operands in bytes (a multiple of 16 on the TMA path)
  int a_pitch;                  // row pitch of A when it differs from K (its rows then are zero padded to it); 0 = K
  int k_corr;                   // number of real K entries (<= K; the rest is zero padding); 0 = K
  int32_t a_offset, bias_offset, out_offset;
  // fused activation on the requantised value (glow::FusedActivation: 0 none, 1 relu, 2 clip, 5 leaky relu)
  int32_t act_type, act_args[3];
  // per-tensor layers: one set of scalars for every column instead of the arrays above
  int uniform;
  int bias_is_i8;
  // Shifted-rows convolution (conv_entries > 0; stride 1, no dilation, no groups): the left operand
  // is the padded NHWC input seen as a matrix [padded pixels, C].  Output pixel (n, oh, ow) is row
  // q = (n * Hp + oh) * Wp + ow of the product, and filter tap (kh, kw) reads row q + kh * Wp + kw:
  // k-block kb of a tile starting at row m0 loads rows m0 + conv_row_off[kb / conv_cpb], 128-byte
  // channel block kb % conv_cpb.  Rows whose (oh, ow) fall outside the output are computed and
  // dropped; the result is stored densely as [n, oh, ow, N].
  int conv_entries, conv_cpb;
  // Row-window convolution (conv_windows = windows per plane, != 0; stride 2, few channels -- a stem):
  // the left operand is two planes of 32-byte windows [plane e][n][y][ow], one after the other (the
  // taps (kh = 2a + e, kw = 0..7) of output pixel (n, oh, ow) are window (n, oh + a, ow) of plane e).
  // k-block kb is plane kb: four loads bring windows q + a * conv_wp (a = 0..3) of the tile's 128
  // pixels q as four 128 x 32-byte tiles, one per MMA k-step.  Output pixel (n, oh, ow) is row
  // (n * Y + oh) * OW + ow of the product (conv_hpwp = Y * OW, conv_wp = OW); rows with oh >= conv_oh
  // are computed and dropped.
  int conv_windows;
  // Strided pointwise convolution (strided_lines != 0): the left operand is every second (or third ...) pixel of the
  // input, a 3-D map [lines of output pixels, OW, C] whose box is strided_lines of them; a tile has that many lines' pixels,
  // strided_lines * OW <= 128 of its rows, and the rest are dropped.
  int strided_lines, strided_rows;
  int conv_row_off[32];
  int conv_hpwp, conv_wp, conv_oh, conv_ow;
  int32_t u_b_offset, u_bias_pre, u_bias_post, u_bias_scale, u_out_pre, u_out_post, u_out_scale;
  // Floating-point result (dynamically quantized layers; float_out != 0): out_f16[i,j] =
  // fp16(float(sum_ij) * (row_scales[i] * col_scales[j]) + bias_f32[j]), sum_ij the int32 dot
  // product of (A - 0) and (B - b_offsets[j]); every product and the sum are rounded separately.
  // col_scales / b_offsets may be NULL: u_col_scale / u_b_offset for every column.
  int float_out;
  __half *out_f16;
  const float *row_scales, *col_scales, *bias_f32;
  float u_col_scale;
};

struct ColQuant {
  int32_t b_off, bias_pre, bias_post, bias_scale, out_pre, out_post, out_scale;
};
__device__ __forceinline__ ColQuant col_quant(const GemmParams &p, int j) {
  if (p.uniform) return {p.u_b_offset, p.u_bias_pre, p.u_bias_post, p.u_bias_scale, p.u_out_pre, p.u_out_post, p.u_out_scale};
  return {p.b_offsets[j], p.bias ? p.bias_pre[j] : 0, p.bias ? p.bias_post[j] : 0, p.bias ? p.bias_scale[j] : 0,
          p.out_pre[j], p.out_post[j], p.out_scale[j]};
}

// Whether the result offset of a column may ride on its rounding term, (((v >> pre) * scale + rtn) >> post) + offset ==
// ((v >> pre) * scale + rtn + (offset << post)) >> post, for every v = dot + c that `k` products of two bytes
// can give: nothing may pass 32 bits, where both wrap, each in its own place.
__host__ __device__ inline bool offset_folds(int64_t k, int32_t c, int32_t pre, int32_t post, int32_t scale, int32_t offset) {
  if (pre < 0 || pre > 30 || post < 1 || post > 30 || scale < 0 || k >= 1ll << 24) return false;
  const auto size = [](int32_t x) { return x < 0 ? -(int64_t)x : (int64_t)x; };
  const int64_t most = size(c) + k * (128 * 128);
  return most < 1ll << 31 && ((most >> pre) + 1) * scale + (1ll << (post - 1)) + (size(offset) << post) < 1ll << 31;
}

// bias[j] of either element type (libjit_fc_generic / libjit_rowwise_quantized_fc_generic /
// libjit_*_conv2d_generic are templates over BiasElemTy: int32 for the _i8_i32 entry points, int8 for _i8_i8).
__device__ __forceinline__ int32_t load_bias(const GemmParams &p, int j) {
  return p.bias_is_i8 ? (int32_t) reinterpret_cast<const int8_t *>(p.bias)[j] : p.bias[j];
}

// libjit_activation_i32 (lib/LLVMIRCodeGen/libjit/libjit_defs.h:206-233).
__device__ __forceinline__ int32_t activation_i32(int32_t x, const GemmParams &p) {
  if (p.act_type == 0) return x;
  if (p.act_type == 1) return x > p.out_offset ? x : p.out_offset;
  if (p.act_type == 2) { const int32_t t = x > p.act_args[0] ? x : p.act_args[0]; return t < p.act_args[1] ? t : p.act_args[1]; }
  if (p.act_type == 3 || p.act_type == 4) return x;
  return x >= p.out_offset ? x : scale32(x - p.out_offset, p.act_args[0], p.act_args[1], p.act_args[2], p.out_offset);
}

// out = requant(A[M,K] x B[N,K]^T); b_is_kn: the right-hand side is given as [K, N].  Products with
// few rows take the one-launch kernel of qgemm_small.cu, the others the tcgen05 kernel -- on the
// operands as they are when K is a multiple of 16 and both are 16-byte aligned [rows, K] matrices, else
// on zero-padded (transposed) copies in `ws` -- and the any-shape kernel when asked for (force_any) or
// when `ws` has no room for the copies.  `ws` must hold i8_gemm_core_workspace_bytes(M, N) bytes, with
// i8_gemm_copies_bytes(M, K, N, ...) more for the copies; a [K, N] right-hand side for which it could not hold
// the N * K bytes is an error.  b_row_sums_in may be nullptr (computed here).
int run_gemm(GemmParams p, const int8_t *a, const int8_t *b, const int32_t *b_row_sums_in, bool b_offsets_zero,
             int force_any, void *ws, size_t ws_bytes, cudaStream_t s, bool b_is_kn = false);

// An NHWC convolution: input [N, H, W, C], filter [OC, KH, KW, C / G], output [N, OH, OW, OC].
struct ConvGeom {
  int N, H, W, C, OH, OW, OC, KH, KW, SH, SW, PT, PL, DH, DW, G;
};

// ---- qgemm_small.cu ----
// A convolution of little work as one such product, its left-hand rows read from the input itself (C a
// multiple of 16, one group, 16-byte aligned operands).
bool i8_skinny_conv_wins(const ConvGeom &g);
int run_conv_skinny(GemmParams p, const int8_t *in, const int8_t *filter, const ConvGeom &g, bool b_offsets_zero, cudaStream_t s);
constexpr int kSkinnyRows = 64;
bool i8_skinny_wins(int64_t M, int64_t N, int64_t K, bool b_is_kn);
// Whether run_gemm takes a [M, K] x [N, K] product with the tile kernel, its operands as they are: what can write a PaddedOut.
inline bool i8_tiles_direct(int64_t M, int64_t N, int64_t K, const void *a, const void *b, const void *out) {
  auto whole = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  return K > 0 && K % 16 == 0 && N % 16 == 0 && whole(a) && whole(b) && whole(out) && !i8_skinny_wins(M, N, K, false);
}
int run_gemm_skinny(GemmParams p, const int8_t *a, const int8_t *b, bool b_is_kn, bool b_offsets_zero, cudaStream_t s);

// One operand to prepare: src [rows, K] -> dst [rows, pitch] (pitch a multiple of 16, the rest zero;
// dst may be nullptr: sums only), or with `transpose` src [K, rows] -> dst [rows, pitch].  sums (may be
// nullptr): per row; a transposed operand's come in prep_transposed_parts() arrays to be added up.
struct PrepSide {
  const int8_t *src;
  int8_t *dst;
  int32_t *sums;
  int rows, K, pitch, transpose, k_span;
};
struct PrepParams {
  PrepSide a, b;  // src nullptr: nothing to do on that side
  int a_blocks;
};
constexpr int kMaxSumParts = 16;
int prep_transposed_parts(int64_t rows, int64_t pitch);
void prep_side_rows(PrepSide &o, const int8_t *src, int8_t *dst, int32_t *sums, int rows, int K, int pitch);
void prep_side_transposed(PrepSide &o, const int8_t *src, int8_t *dst, int32_t *sums, int rows, int K, int pitch);
int run_prepare_operands(PrepParams p, cudaStream_t s);

// The shifted-rows convolution on the same kernel: `padded` holds `rows` padded pixels of `C` bytes
// (plus 128 readable bytes behind them), p.conv_* describe the taps, p.M = rows, p.K = bytes of a
// row of b (a multiple of 128).  Weight offsets must all be zero (no input row sums).
// buffer_rows: rows the padded buffer holds when the taps reach beyond `rows` (several planes); 0 = rows.
int run_gemm_shifted_rows(GemmParams p, const int8_t *padded, int64_t rows, int C, const int8_t *b,
                          const int32_t *b_row_sums, cudaStream_t s, int64_t buffer_rows = 0);

// A pointwise convolution of stride s over an input whose height and width are multiples of it, read in place: p.M output
// pixels in `lines` lines of ow; p.K = channels (a multiple of 16).  No weight offsets.
int run_gemm_strided(GemmParams p, const int8_t *in, int64_t lines, int ow, int stride, int width, const int8_t *b, const int32_t *b_row_sums,
                     cudaStream_t s);

// The row-window convolution: `planes` holds two planes of `rows` 32-byte windows each, back to back,
// with 3 * ow + 1 readable windows behind the second; b is [N, 256] (plane, a, 32 bytes).
int run_gemm_row_windows(GemmParams p, const int8_t *planes, int64_t rows, int ow, const int8_t *b, const int32_t *b_row_sums,
                         cudaStream_t s);

inline size_t i8_gemm_core_workspace_bytes(int64_t M, int64_t N) {
  return align_up((size_t)N * 4, 256) + align_up((size_t)M * 4, 256);
}
// Room for a padded copy of either operand and the partial sums of a transposed one.
inline size_t i8_gemm_copies_bytes(int64_t M, int64_t K, int64_t N, bool copy_a, bool copy_b) {
  const size_t pitch = align_up((size_t)K, 16);
  return (copy_a ? align_up((size_t)M * pitch, 256) : 0) +
         (copy_b ? align_up((size_t)N * pitch, 256) + align_up((size_t)N * 4 * kMaxSumParts, 256) : 0);
}

}  // namespace glowb200
