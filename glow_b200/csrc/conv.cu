// Int8 2-D convolution (NHWC, filter [outC, kH, kW, inC/group]) for Glow's
// ChannelwiseQuantizedConvolution and quantized Convolution.
//
// group == 1: the convolution is the int8 contraction of qgemm.cu over an im2col matrix
//   A[n*OH*OW + oh*OW + ow, (kh*KW + kw)*C + c] = X[n, oh*SH - PT + kh*DH, ow*SW - PL + kw*DW, c]
// whose result rows are exactly the NHWC output.  Taps outside the image are skipped by the
// reference (libjit_conv.cpp:209-212), i.e. they contribute (x - inOffset) = 0: im2col writes
// inOffset there.  The filter [outC, kH*kW*C] already is the K-major right-hand side.  A 1x1,
// stride-1, unpadded convolution needs no im2col at all.  When kH*kW*C is not a multiple of 16
// both operands are padded with zeros along K (zeros add nothing to the raw products or to the
// row sums; the offset correction uses the true K).
// group > 1 (and anything else unusual): a direct kernel, one thread per output, the
// reference's loop nest as written.
#include "common.cuh"
#include "qgemm.cuh"

namespace glowb200 {
namespace {

// Blocks of a kernel that walks on: `per_sm` to an SM at most.
unsigned grid_of(int64_t blocks, int per_sm) {
  const int64_t most = (int64_t)kB200Sms * per_sm;
  return (unsigned)(blocks < most ? blocks : most);
}

// one thread per 16-byte chunk of the im2col matrix (C a multiple of 16: a chunk never
// straddles two taps).  64-bit divisions bound it first: every second pixel of 64 x 56 x 56 x 256 13 us, now 10.
struct Im2colRadix {
  Divisor row, pixel, width, height, taps;
  Im2colRadix(const ConvGeom &g, int Kpad) : row(Kpad >> 4), pixel(g.C >> 4), width(g.OW), height(g.OH), taps(g.KW) {}
};
__global__ void __launch_bounds__(256) im2col_i8_vec_kernel(const int8_t *__restrict__ x, int8_t *__restrict__ a,
                                                             const __grid_constant__ ConvGeom g, const __grid_constant__ Im2colRadix radix,
                                                             int Kpad, int pad_word) {
  pdl_wait();
  pdl_launch_dependents();
  const int total = g.N * g.OH * g.OW * (Kpad >> 4), step = gridDim.x * blockDim.x;  // (below 2^31: the launcher's condition)
  for (int64_t at = blockIdx.x * blockDim.x + threadIdx.x; at < total; at += step) {
    const int i = (int)at;
    int n = i, tap = radix.row.rest(n);
    const int ow = radix.width.rest(n), oh = radix.height.rest(n), cc = radix.pixel.rest(tap);
    int4 v = make_int4(0, 0, 0, 0);
    if (tap < g.KH * g.KW) {
      int kh = tap;
      const int kw = radix.taps.rest(kh);
      const int ih = oh * g.SH - g.PT + kh * g.DH, iw = ow * g.SW - g.PL + kw * g.DW;
      if (ih >= 0 && iw >= 0 && ih < g.H && iw < g.W)
        v = __ldg(reinterpret_cast<const int4 *>(x + (((int64_t)n * g.H + ih) * g.W + iw) * g.C) + cc);
      else
        v = make_int4(pad_word, pad_word, pad_word, pad_word);
    }
    reinterpret_cast<int4 *>(a)[i] = v;
  }
}

// any channel count: one thread per byte
__global__ void __launch_bounds__(256) im2col_i8_kernel(const int8_t *__restrict__ x, int8_t *__restrict__ a,
                                                         const __grid_constant__ ConvGeom g, int K, int Kpad, int8_t pad) {
  const int64_t total = (int64_t)g.N * g.OH * g.OW * Kpad;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / Kpad;
    const int k = (int)(i - row * Kpad);
    int8_t v = 0;
    if (k < K) {
      const int tap = k / g.C, c = k - tap * g.C;
      const int kh = tap / g.KW, kw = tap - kh * g.KW;
      const int ow = (int)(row % g.OW);
      const int64_t r2 = row / g.OW;
      const int oh = (int)(r2 % g.OH), n = (int)(r2 / g.OH);
      const int ih = oh * g.SH - g.PT + kh * g.DH, iw = ow * g.SW - g.PL + kw * g.DW;
      v = (ih >= 0 && iw >= 0 && ih < g.H && iw < g.W) ? x[(((int64_t)n * g.H + ih) * g.W + iw) * g.C + c] : pad;
    }
    a[i] = v;
  }
}

// Bytes of a staged input row of im2col_i8_rows_kernel: the image row, its left padding and as much
// on the right as the last output pixel's window reaches.
__host__ __device__ inline int64_t rows_pitch(const ConvGeom &g) {
  const int64_t last = (int64_t)(g.OW - 1) * g.SW + (int64_t)(g.KW - 1) * g.DW + 1;  // pixels from the padded row's start
  const int64_t have = (int64_t)g.PL + g.W;
  return (last > have ? last : have) * g.C;
}

// Any channel count, one block per output image row (n, oh).  The KH input rows the image row
// needs are staged in shared memory with their horizontal padding made real (`pad` left and right
// of the image, whole rows of it above and below), so a tap is a plain offset from the pixel's
// window.  A thread keeps ONE 16-byte piece of the im2col row (piece = thread % pieces per row) for
// all the pixels it visits: the sixteen offsets of its bytes are worked out once, and a piece then
// costs sixteen byte loads, the packing and one vector store.  (Walking (kh, kw, c) with counters
// for every piece, as this kernel first did, took 163 us for a 7 x 7 stride-2 stem over 3 channels
// at batch 64: about 170 instructions per 16 bytes.)
// Shared memory: KH rows of `pitch` bytes (checked by the launcher).
__global__ void __launch_bounds__(256) im2col_i8_rows_kernel(const int8_t *__restrict__ x, int8_t *__restrict__ a,
                                                              const __grid_constant__ ConvGeom g, int K, int Kpad, int8_t pad,
                                                              int pitch) {
  extern __shared__ __align__(16) int8_t rows_smem[];
  const int n = blockIdx.x / g.OH, oh = blockIdx.x - n * g.OH;
  const int row_bytes = g.W * g.C, left = g.PL * g.C;
  for (int kh = 0; kh < g.KH; kh++) {
    const int ih = oh * g.SH - g.PT + kh * g.DH;
    int8_t *dst = rows_smem + kh * pitch;
    if (ih < 0 || ih >= g.H) {
      for (int j = threadIdx.x; j < pitch; j += blockDim.x) dst[j] = pad;
      continue;
    }
    const int8_t *src = x + ((int64_t)n * g.H + ih) * row_bytes;
    for (int j = threadIdx.x; j < pitch - row_bytes; j += blockDim.x) dst[j < left ? j : j + row_bytes] = pad;
    if (((reinterpret_cast<uintptr_t>(src) | (uintptr_t)row_bytes) & 3) == 0) {
      for (int j = threadIdx.x * 4; j < row_bytes; j += blockDim.x * 4) {
        const uint32_t v = __ldg(reinterpret_cast<const uint32_t *>(src + j));
        dst[left + j] = (int8_t)v;
        dst[left + j + 1] = (int8_t)(v >> 8);
        dst[left + j + 2] = (int8_t)(v >> 16);
        dst[left + j + 3] = (int8_t)(v >> 24);
      }
    } else {
      for (int j = threadIdx.x; j < row_bytes; j += blockDim.x) dst[left + j] = src[j];
    }
  }
  const int pieces = Kpad >> 4;
  const int ch = threadIdx.x % pieces, slot = threadIdx.x / pieces, slots = blockDim.x / pieces;
  int off[16];
  uint32_t keep[4] = {0u, 0u, 0u, 0u};  // bytes of the piece that are taps (the rest is the zero padding of K)
#pragma unroll
  for (int b = 0; b < 16; b++) {
    const int k = ch * 16 + b;
    off[b] = 0;
    if (k < K) {
      const int tap = k / g.C, c = k - tap * g.C;
      const int kh = tap / g.KW, kw = tap - kh * g.KW;
      off[b] = kh * pitch + kw * g.DW * g.C + c;
      keep[b >> 2] |= 0xffu << (8 * (b & 3));
    }
  }
  __syncthreads();
  int8_t *out = a + ((int64_t)n * g.OH + oh) * g.OW * Kpad + ch * 16;
  if (slot < slots) {
    for (int ow = slot; ow < g.OW; ow += slots) {
      const uint8_t *win = reinterpret_cast<const uint8_t *>(rows_smem) + ow * g.SW * g.C;
      uint32_t w[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint32_t lo = __byte_perm(win[off[4 * q]], win[off[4 * q + 1]], 0x0040);
        const uint32_t hi = __byte_perm(win[off[4 * q + 2]], win[off[4 * q + 3]], 0x0040);
        w[q] = __byte_perm(lo, hi, 0x5410) & keep[q];
      }
      *reinterpret_cast<int4 *>(out + (int64_t)ow * Kpad) = make_int4((int)w[0], (int)w[1], (int)w[2], (int)w[3]);
    }
  }
}

// Row windows of a stride-2 convolution over few channels (KW * C <= 32, no dilation): plane e
// (e = 0, 1), image n, row y, output column ow holds the KW * C bytes x[n, 2y - PT + e, 2ow - PL .. + KW - 1, :]
// and zeros up to 32 bytes; cells outside the image hold `pad` (the input offset).  Tap (kh = 2a + e, kw)
// of output pixel (n, oh, ow) is byte kw * C + c of window (n, oh + a, ow) of plane e, so the
// convolution is a contraction whose left-hand rows are four windows of one plane, Y = OH + 3 rows
// per image: 2 * 32 bytes per (y, ow) instead of KH * KW * C per output pixel, and no im2col matrix.
// One thread per window, cut from the words of the image row that it lies across; behind them `tail` zero windows (the
// four windows of the last rows reach that far) and the filter re-laid to match: [OC, KH, KW, C] -> [OC, 2 planes, 4 rows a,
// 32 bytes], tap (kh = 2a + e, kw, c) at byte kw * C + c of (e, a), everything else zero.
// What bounds it is the 53 MB that a batch of 64 images of 224 x 224 writes, and instructions beside it: 31 us with a
// window's 21 bytes loaded one by one and 64-bit divisions, 23 by way of shared memory, now 19.
struct WindowRadix {
  Divisor width, height;
  WindowRadix(const ConvGeom &g, int Y) : width(g.OW), height(Y) {}
};
__global__ void __launch_bounds__(256) row_windows_i8_kernel(const int8_t *__restrict__ x, int8_t *__restrict__ planes,
                                                              const __grid_constant__ ConvGeom g, const __grid_constant__ WindowRadix radix,
                                                              int64_t plane_bytes, int8_t pad, int tail, const int8_t *__restrict__ f,
                                                              int8_t *__restrict__ fb) {
  pdl_wait();
  pdl_launch_dependents();
  const int run = g.KW * g.C, row_bytes = g.W * g.C;
  const int per_plane = g.N * radix.height.d * g.OW;
  const int64_t windows = 2 * (int64_t)per_plane, total = windows + tail + (int64_t)g.OC * 8;
  const uint32_t pad4 = 0x01010101u * (uint32_t)(uint8_t)pad;
  const bool whole_words = ((reinterpret_cast<uintptr_t>(x) | (uintptr_t)row_bytes) & 3) == 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t w[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
    int4 *dst;
    if (i < windows) {
      const int e = i >= per_plane ? 1 : 0, at = (int)(i - (e ? per_plane : 0));
      int n = at;
      const int ow = radix.width.rest(n), y = radix.height.rest(n);
      const int ih = 2 * y - g.PT + e, first = (2 * ow - g.PL) * g.C, from = first & ~3;  // bytes of the image row
      if (ih >= 0 && ih < g.H) {
        const int8_t *src = x + ((int64_t)n * g.H + ih) * row_bytes;
        uint32_t word[9];
        if (whole_words) {  // (a word then lies inside the row or outside, none across its ends)
#pragma unroll
          for (int k = 0; k < 9; k++) {
            word[k] = pad4;
            if (4 * k < run + 3 && (unsigned)(from + 4 * k) < (unsigned)row_bytes) word[k] = __ldg(reinterpret_cast<const uint32_t *>(src + from) + k);
          }
        } else {
#pragma unroll
          for (int k = 0; k < 9; k++) {
            word[k] = pad4;
#pragma unroll
            for (int b = 0; b < 4; b++) {
              const int o = from + 4 * k + b;
              if (o - first < run && o >= 0 && o < row_bytes) word[k] = (word[k] & ~(0xffu << (8 * b))) | (uint32_t)(uint8_t)src[o] << (8 * b);
            }
          }
        }
#pragma unroll
        for (int k = 0; k < 8; k++) w[k] = __funnelshift_r(word[k], word[k + 1], 8 * (first & 3));
      } else {
#pragma unroll
        for (int k = 0; k < 8; k++) w[k] = pad4;
      }
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const int valid = run - 4 * k;  // bytes of the word that are taps
        w[k] = valid <= 0 ? 0u : valid >= 4 ? w[k] : w[k] & ((1u << (8 * valid)) - 1u);
      }
      dst = reinterpret_cast<int4 *>(planes + e * plane_bytes + (int64_t)at * 32);
    } else if (i < windows + tail) {
      dst = reinterpret_cast<int4 *>(planes + 2 * plane_bytes + (i - windows) * 32);
    } else {
      const int64_t r = i - windows - tail;  // 32 bytes (e, a) of a filter
      const int oc = (int)(r >> 3), e = (int)(r >> 2) & 1, kh = 2 * ((int)r & 3) + e;
      if (kh < g.KH) {
        const int8_t *src = f + ((int64_t)oc * g.KH + kh) * run;
#pragma unroll
        for (int b = 0; b < 32; b++)
          if (b < run) w[b >> 2] |= (uint32_t)(uint8_t)src[b] << (8 * (b & 3));
      }
      dst = reinterpret_cast<int4 *>(fb + r * 32);
    }
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
                 "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
  }
}

// NHWC input with its padding made real: [N, Hp, Wp, C], the cells outside the image filled with
// `pad_word` (the input offset, which is how the reference's skipped taps read), and 256 zero bytes
// behind it (the window of the last rows reads past them).  16 bytes per thread.
// fb != nullptr (C = 64): the same launch re-lays the filter [OC, KH, KW, 64] -> [OC, KH * ceil(KW / 2), 128],
// taps (kh, 2j) and (kh, 2j + 1) side by side, the partner of a last odd tap zero -- the right-hand side
// that matches left-hand rows made of two neighbouring 64-channel pixels.
__global__ void __launch_bounds__(256) pad_nhwc_i8_kernel(const int8_t *__restrict__ x, int8_t *__restrict__ xp,
                                                           const __grid_constant__ ConvGeom g, int Hp, int Wp, int pad_word,
                                                           const int8_t *__restrict__ f, int8_t *__restrict__ fb) {
  pdl_wait();
  pdl_launch_dependents();
  const int cc = g.C >> 4, pairs = (g.KW + 1) >> 1;
  const int64_t cells = (int64_t)g.N * Hp * Wp * cc, total = cells + 16 + (fb ? (int64_t)g.OC * g.KH * pairs * 8 : 0);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    int4 v = make_int4(0, 0, 0, 0);
    if (i < cells) {
      const int c = (int)(i % cc);
      int64_t r = i / cc;
      const int xw = (int)(r % Wp);
      r /= Wp;
      const int yh = (int)(r % Hp), n = (int)(r / Hp);
      const int ih = yh - g.PT, iw = xw - g.PL;
      v = make_int4(pad_word, pad_word, pad_word, pad_word);
      if (ih >= 0 && iw >= 0 && ih < g.H && iw < g.W)
        v = __ldg(reinterpret_cast<const int4 *>(x + (((int64_t)n * g.H + ih) * g.W + iw) * g.C) + c);
    } else if (i >= cells + 16) {
      const int64_t j = i - cells - 16;
      const int piece = (int)(j & 7);
      int64_t r = j >> 3;
      const int kw = 2 * (int)(r % pairs) + (piece >> 2);
      r /= pairs;  // oc * KH + kh
      if (kw < g.KW) v = __ldg(reinterpret_cast<const int4 *>(f + (r * g.KW + kw) * 64) + (piece & 3));
      reinterpret_cast<int4 *>(fb)[j] = v;
      continue;
    }
    reinterpret_cast<int4 *>(xp)[i] = v;
  }
}

// The same for a stride-2 window, split by the parity of the padded coordinates: plane (ph, pw) holds
// the padded input at (2y + ph, 2x + pw), [4][N, Hq, Wq, C].  Tap (kh, kw) of output pixel (n, oh, ow)
// is then pixel (n, oh + kh / 2, ow + kw / 2) of plane (kh & 1, kw & 1): a row offset again.
__global__ void __launch_bounds__(256) pad_parity_nhwc_i8_kernel(const int8_t *__restrict__ x, int8_t *__restrict__ xp,
                                                                  const __grid_constant__ ConvGeom g, int Hq, int Wq, int pad_word) {
  pdl_wait();
  pdl_launch_dependents();
  const int cc = g.C >> 4;
  const int64_t total = 4ll * g.N * Hq * Wq * cc;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % cc);
    int64_t r = i / cc;
    const int xq = (int)(r % Wq);
    r /= Wq;
    const int yq = (int)(r % Hq);
    r /= Hq;
    const int n = (int)(r % g.N), plane = (int)(r / g.N);
    const int ih = 2 * yq + (plane >> 1) - g.PT, iw = 2 * xq + (plane & 1) - g.PL;
    int4 v = make_int4(pad_word, pad_word, pad_word, pad_word);
    if (ih >= 0 && iw >= 0 && ih < g.H && iw < g.W)
      v = __ldg(reinterpret_cast<const int4 *>(x + (((int64_t)n * g.H + ih) * g.W + iw) * g.C) + c);
    reinterpret_cast<int4 *>(xp)[i] = v;
  }
}

// [rows, K] -> [rows, Kpad], zero padded
__global__ void __launch_bounds__(256) pad_rows_i8_kernel(const int8_t *__restrict__ in, int8_t *__restrict__ out, int rows,
                                                           int K, int Kpad) {
  const int64_t total = (int64_t)rows * Kpad;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / Kpad;
    const int k = (int)(i - r * Kpad);
    out[i] = k < K ? in[r * K + k] : (int8_t)0;
  }
}

// The reference's loop nest (libjit_conv.cpp:151-239 / :49-147), one thread per output element.
__global__ void __launch_bounds__(256) conv2d_i8_direct_kernel(const int8_t *__restrict__ x, const int8_t *__restrict__ f,
                                                                const __grid_constant__ ConvGeom g,
                                                                const __grid_constant__ GemmParams p) {
  const int64_t total = (int64_t)g.N * g.OH * g.OW * g.OC;
  const int icg = g.C / g.G, ocg = g.OC / g.G;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int d = (int)(i % g.OC);
    int64_t r = i / g.OC;
    const int ow = (int)(r % g.OW);
    r /= g.OW;
    const int oh = (int)(r % g.OH), n = (int)(r / g.OH);
    const int grp = d / ocg;
    const ColQuant q = col_quant(p, d);
    uint32_t sum = (uint32_t)scale32(load_bias(p, d) - (p.bias_offsets ? p.bias_offsets[d] : p.bias_offset), q.bias_pre,
                                     q.bias_post, q.bias_scale, 0);
    for (int kh = 0; kh < g.KH; kh++)
      for (int kw = 0; kw < g.KW; kw++) {
        const int ih = oh * g.SH - g.PT + kh * g.DH, iw = ow * g.SW - g.PL + kw * g.DW;
        if (ih < 0 || iw < 0 || ih >= g.H || iw >= g.W) continue;
        const int8_t *xp = x + (((int64_t)n * g.H + ih) * g.W + iw) * g.C + grp * icg;
        const int8_t *fp = f + (((int64_t)d * g.KH + kh) * g.KW + kw) * icg;
        for (int c = 0; c < icg; c++) sum += (uint32_t)(((int32_t)fp[c] - q.b_off) * ((int32_t)xp[c] - p.a_offset));
      }
    p.out[i] = (int8_t)clip_i8(activation_i32(scale32((int32_t)sum, q.out_pre, q.out_post, q.out_scale, p.out_offset), p));
  }
}

int geom_from_dims(ConvGeom &g, const int64_t *out_dims, const int64_t *in_dims, const int64_t *filter_dims,
                   const int64_t *kernels, const int64_t *strides, const int64_t *pads, int64_t group,
                   const int64_t *dilation) {
  GLOWB200_REQUIRE(out_dims && in_dims && filter_dims && kernels && strides && pads && dilation, "NULL shape array");
  for (int i = 0; i < 4; i++)
    GLOWB200_REQUIRE(out_dims[i] >= 0 && in_dims[i] >= 0 && filter_dims[i] >= 0 && out_dims[i] < (1ll << 31) &&
                         in_dims[i] < (1ll << 31) && filter_dims[i] < (1ll << 31), "dimension out of range");
  g.N = (int)in_dims[0]; g.H = (int)in_dims[1]; g.W = (int)in_dims[2]; g.C = (int)in_dims[3];
  g.OH = (int)out_dims[1]; g.OW = (int)out_dims[2]; g.OC = (int)out_dims[3];
  g.KH = (int)kernels[0]; g.KW = (int)kernels[1];
  g.SH = (int)strides[0]; g.SW = (int)strides[1];
  g.PT = (int)pads[0]; g.PL = (int)pads[1];
  g.DH = (int)dilation[0]; g.DW = (int)dilation[1];
  g.G = (int)group;
  GLOWB200_REQUIRE(out_dims[0] == in_dims[0], "batch sizes of input and output differ");
  GLOWB200_REQUIRE(g.G >= 1 && g.C % g.G == 0 && g.OC % g.G == 0, "channels not divisible by the group count");
  GLOWB200_REQUIRE(filter_dims[0] == g.OC && filter_dims[1] == g.KH && filter_dims[2] == g.KW &&
                       filter_dims[3] == g.C / g.G, "filter dims do not match [outC, kH, kW, inC/group]");
  GLOWB200_REQUIRE(g.SH >= 1 && g.SW >= 1 && g.DH >= 1 && g.DW >= 1 && g.KH >= 1 && g.KW >= 1, "bad stride/dilation/kernel");
  return GLOWB200_OK;
}

struct ConvPlan {
  bool direct;       // direct kernel (groups, empty)
  bool need_im2col;  // else the input itself is the left-hand side
  int K, Kpad;
  int64_t M;
  size_t a_bytes, f_bytes, core_bytes;
};

ConvPlan plan_conv(const ConvGeom &g, bool force_direct) {
  ConvPlan pl{};
  pl.M = (int64_t)g.N * g.OH * g.OW;
  pl.K = g.KH * g.KW * g.C;
  pl.Kpad = (pl.K + 15) / 16 * 16;
  pl.direct = force_direct || g.G != 1 || pl.M >= (1ll << 31) || pl.K >= (1 << 24);
  const bool pointwise = g.KH == 1 && g.KW == 1 && g.SH == 1 && g.SW == 1 && g.PT == 0 && g.PL == 0 && g.OH == g.H &&
                         g.OW == g.W && (g.C % 16) == 0;
  pl.need_im2col = !pl.direct && !pointwise;
  pl.a_bytes = pl.need_im2col ? align_up((size_t)pl.M * pl.Kpad, 256) : 0;
  pl.f_bytes = (!pl.direct && pl.Kpad != pl.K) ? align_up((size_t)g.OC * pl.Kpad, 256) : 0;
  pl.core_bytes = pl.direct ? 0 : i8_gemm_core_workspace_bytes(pl.M, g.OC);
  return pl;
}

int pad_word(int32_t offset) {
  const uint32_t b = (uint8_t)offset;
  return (int)(b | (b << 8) | (b << 16) | (b << 24));
}

// Windows over 64 or a multiple of 128 channels, symmetric filters: no im2col matrix.
// Stride 1: the input lies in a padded NHWC buffer [N, h, w, C]; tap (kh, kw) of output row q then is row q + kh * w + kw
// of that buffer, which the contraction's loads address directly (the rows of the product that fall on the
// padding are computed and dropped).  Stride 2 (multiples of 128 channels): the same over four planes by the parity of
// the padded coordinates (see pad_parity_nhwc_i8_kernel).  The scratch sized for the im2col matrix is more than this needs.
// 64 channels: two neighbouring pixels per 128-byte row against a filter re-laid in tap pairs (the
// partner of an odd last tap zero).  One tap per 64-byte k-block in the 64-byte swizzle -- no
// wasted MMAs, a quarter fewer operand bytes, nine k-blocks instead of six for a 3 x 3 window --
// gave the same results and a slower network (1.590 against 1.562 ms per ResNet-50 batch).
struct ShiftedRows {
  int planes, h, w, pairs, entries;  // pairs: of taps in a filter row (64 channels; else 0)
  int64_t rows;                      // pixels of a plane
  size_t input_bytes, pair_bytes;    // of the buffer, and of the filter re-laid behind it
};
bool shifted_rows(const ConvGeom &g, const ConvPlan &pl, int flags, ShiftedRows &r) {
  if (!pl.need_im2col || g.SH != g.SW || g.SH > 2 || g.DH != 1 || g.DW != 1 || !(flags & GLOWB200_FC_WEIGHT_OFFSETS_ZERO)) return false;
  r = ShiftedRows{};
  if (g.SH == 1) {
    if (g.C != 64 && g.C % 128 != 0) return false;
    r.planes = 1;
    r.h = g.OH + g.KH - 1;
    r.w = g.OW + g.KW - 1;
    if (r.h < g.H + g.PT || r.w < g.W + g.PL) return false;
    r.pairs = g.C == 64 ? (g.KW + 1) / 2 : 0;
  } else {
    if (g.C % 128 != 0 || (g.KH == 1 && g.KW == 1)) return false;
    r.planes = 4;
    r.h = g.OH + (g.KH - 1) / 2;
    r.w = g.OW + (g.KW - 1) / 2;
  }
  r.entries = g.KH * (r.pairs ? r.pairs : g.KW);
  r.rows = (int64_t)g.N * r.h * r.w;
  r.input_bytes = align_up((size_t)(r.planes * r.rows) * g.C + 256, 256);
  r.pair_bytes = r.pairs ? align_up((size_t)g.OC * r.entries * 128, 256) : 0;
  return r.entries <= 32 && r.planes * r.rows < (1ll << 31) && r.input_bytes + r.pair_bytes <= pl.a_bytes + pl.f_bytes;
}

// The contraction over such a buffer; b: the filter, in tap pairs where r.pairs.
int run_shifted_rows(GemmParams p, const ConvGeom &g, const ConvPlan &pl, const ShiftedRows &r, const int8_t *xp, const int8_t *b,
                     const int32_t *filter_row_sums, uint8_t *sums_ws, cudaStream_t s) {
  p.K = r.pairs ? r.entries * 128 : g.KH * g.KW * g.C;
  p.k_corr = pl.K;
  p.N = g.OC;
  p.conv_entries = r.entries;
  p.conv_cpb = r.pairs ? 1 : g.C / 128;
  for (int e = 0; e < r.entries; e++) {
    const int kh = e / (r.pairs ? r.pairs : g.KW), kw = r.pairs ? 2 * (e % r.pairs) : e % g.KW;
    p.conv_row_off[e] = r.planes == 1 ? kh * r.w + kw : (int)(((kh & 1) * 2 + (kw & 1)) * r.rows) + (kh >> 1) * r.w + (kw >> 1);
  }
  p.conv_hpwp = r.h * r.w;
  p.conv_wp = r.w;
  p.conv_oh = g.OH;
  p.conv_ow = g.OW;
  if (filter_row_sums == nullptr) {  // zeros added by the pairing do not change the sums
    int32_t *sums = reinterpret_cast<int32_t *>(sums_ws);
    if (int rc = glowb200_i8_row_sums(b, g.OC, p.K, sums, reinterpret_cast<glowb200_stream_t>(s))) return rc;
    filter_row_sums = sums;
  }
  return run_gemm_shifted_rows(p, xp, r.rows, g.C, b, filter_row_sums, s, r.planes * r.rows);
}

int run_conv(GemmParams p, const int8_t *in, const int8_t *filter, const ConvGeom &g, const int32_t *filter_row_sums,
             int flags, void *workspace, size_t workspace_bytes, cudaStream_t s) {
  const int64_t outputs = (int64_t)g.N * g.OH * g.OW * g.OC;
  if (outputs == 0) return GLOWB200_OK;
  const ConvPlan pl = plan_conv(g, (flags & GLOWB200_FC_FORCE_ANY_SHAPE_KERNEL) != 0);
  if (pl.direct) {
    const int64_t blocks = (outputs + 255) / 256;
    conv2d_i8_direct_kernel<<<grid_of(blocks, 32), 256, 0, s>>>(in, filter, g, p);
    GLOWB200_CUDA_OK(cudaGetLastError());
    return GLOWB200_OK;
  }
  const bool aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(filter)) & 15) == 0;
  if (pl.need_im2col && aligned && i8_skinny_conv_wins(g))
    return run_conv_skinny(p, in, filter, g, (flags & GLOWB200_FC_WEIGHT_OFFSETS_ZERO) != 0, s);
  const size_t need = pl.a_bytes + pl.f_bytes + pl.core_bytes;
  if (workspace == nullptr || workspace_bytes < need)
    return set_error(GLOWB200_ERR_WORKSPACE_TOO_SMALL, "workspace of %zu bytes given, %zu needed", workspace_bytes, need);
  GLOWB200_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, "workspace must be 256-byte aligned");
  uint8_t *ws = reinterpret_cast<uint8_t *>(workspace);
  ShiftedRows sr;
  if (aligned && shifted_rows(g, pl, flags, sr)) {
    int8_t *xp = reinterpret_cast<int8_t *>(ws), *pairs = sr.pair_bytes ? reinterpret_cast<int8_t *>(ws + sr.input_bytes) : nullptr;
    const int word = pad_word(p.a_offset);
    if (sr.planes == 1) {
      const int64_t chunks = sr.rows * (g.C >> 4) + 16 + (pairs ? (int64_t)g.OC * sr.entries * 8 : 0), blocks = (chunks + 255) / 256;
      GLOWB200_CUDA_OK(launch_pdl(pad_nhwc_i8_kernel, grid_of(blocks, 64), 256, 0, s, in, xp, g, sr.h, sr.w, word, filter, pairs));
    } else {
      const int64_t chunks = 4 * sr.rows * (g.C >> 4), blocks = (chunks + 255) / 256;
      GLOWB200_CUDA_OK(launch_pdl(pad_parity_nhwc_i8_kernel, grid_of(blocks, 64), 256, 0, s, in, xp, g, sr.h, sr.w, word));
    }
    return run_shifted_rows(p, g, pl, sr, xp, pairs ? pairs : filter, filter_row_sums, ws + pl.a_bytes + pl.f_bytes, s);
  }
  // Stride-2 windows over few channels with symmetric filters (the 7 x 7 stem over 3 channels): row
  // windows instead of an im2col matrix (see row_windows_i8_kernel).
  if (pl.need_im2col && g.SH == 2 && g.SW == 2 && g.DH == 1 && g.DW == 1 && (flags & GLOWB200_FC_WEIGHT_OFFSETS_ZERO) &&
      g.KW * g.C <= 32 && g.KH <= 8 && (reinterpret_cast<uintptr_t>(filter) & 15) == 0) {
    const int Y = g.OH + 3;
    const int64_t rows = (int64_t)g.N * Y * g.OW;
    const int64_t plane_bytes = rows * 32;
    const size_t wp_bytes = align_up((size_t)(2 * plane_bytes + (3 * (int64_t)g.OW + 1) * 32), 256);
    const size_t fb_bytes = align_up((size_t)g.OC * 256, 256);
    if (rows < (1ll << 31) && wp_bytes + fb_bytes <= pl.a_bytes + pl.f_bytes) {
      int8_t *planes = reinterpret_cast<int8_t *>(ws);
      int8_t *fb = reinterpret_cast<int8_t *>(ws + wp_bytes);
      const int tail = (int)((wp_bytes - 2 * plane_bytes) / 32);  // the four windows of the last rows reach past the second plane
      const int64_t items = 2 * rows + tail + (int64_t)g.OC * 8, blocks = (items + 255) / 256;
      GLOWB200_CUDA_OK(launch_pdl(row_windows_i8_kernel, grid_of(blocks, 64), 256, 0, s, in, planes, g, WindowRadix(g, Y),
                                  plane_bytes, (int8_t)p.a_offset, tail, filter, fb));
      const int32_t *bs = filter_row_sums;  // (the zeros of the new layout do not change them)
      if (bs == nullptr) {
        int32_t *sums = reinterpret_cast<int32_t *>(ws + pl.a_bytes + pl.f_bytes);
        if (int rc = glowb200_i8_row_sums(fb, g.OC, 256, sums, reinterpret_cast<glowb200_stream_t>(s))) return rc;
        bs = sums;
      }
      p.K = 256;
      p.k_corr = pl.K;
      p.N = g.OC;
      p.conv_hpwp = Y * g.OW;
      p.conv_wp = g.OW;
      p.conv_oh = g.OH;
      p.conv_ow = g.OW;
      return run_gemm_row_windows(p, planes, rows, g.OW, fb, bs, s);
    }
  }
  // Every s-th pixel of an image whose sides are multiples of s: the contraction's loads take them from the input itself, whole
  // lines of output pixels to a tile.  At least 96 of a tile's 128 rows have to be pixels (28 x 28 of 64 x 56 x 56 x 256 to 512
  // channels, 112 rows to a tile: 10 + 15 us with a copy of the pixels, now 17).
  if (pl.need_im2col && g.KH == 1 && g.KW == 1 && g.SH == g.SW && g.PT == 0 && g.PL == 0 && g.H == g.OH * g.SH && g.W == g.OW * g.SW &&
      (flags & GLOWB200_FC_WEIGHT_OFFSETS_ZERO) && g.C % 16 == 0 && aligned && g.OW <= 128 && 128 / g.OW * g.OW >= 96) {
    const int32_t *sums = filter_row_sums;
    if (sums == nullptr) {
      int32_t *bs = reinterpret_cast<int32_t *>(ws + pl.a_bytes + pl.f_bytes);
      if (int rc = glowb200_i8_row_sums(filter, g.OC, g.C, bs, reinterpret_cast<glowb200_stream_t>(s))) return rc;
      sums = bs;
    }
    p.K = g.C;
    p.N = g.OC;
    return run_gemm_strided(p, in, (int64_t)g.N * g.OH, g.OW, g.SW, g.W, filter, sums, s);
  }
  const int8_t *a = in;
  if (pl.need_im2col) {
    int8_t *abuf = reinterpret_cast<int8_t *>(ws);
    const int8_t pad = (int8_t)p.a_offset;
    if ((g.C % 16) == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0 && pl.M * (pl.Kpad >> 4) < (1ll << 31)) {
      const int64_t chunks = pl.M * (pl.Kpad >> 4);
      const int64_t blocks = (chunks + 255) / 256;
      const uint32_t b = (uint8_t)pad;
      GLOWB200_CUDA_OK(launch_pdl(im2col_i8_vec_kernel, grid_of(blocks, 64), 256, 0, s, in, abuf, g, Im2colRadix(g, pl.Kpad), pl.Kpad,
                                  (int)(b | (b << 8) | (b << 16) | (b << 24))));
    } else if ((int64_t)g.KH * rows_pitch(g) <= 48 * 1024 && (int64_t)g.N * g.OH < (1ll << 31) && (pl.Kpad >> 4) <= 256 &&
               (reinterpret_cast<uintptr_t>(abuf) & 15) == 0) {
      // the KH input rows of an output image row, with their padding, fit the default shared-memory window
      const int pitch = (int)rows_pitch(g);
      im2col_i8_rows_kernel<<<(unsigned)(g.N * g.OH), 256, (size_t)g.KH * pitch, s>>>(in, abuf, g, pl.K, pl.Kpad, pad, pitch);
    } else {
      const int64_t blocks = (pl.M * pl.Kpad + 255) / 256;
      im2col_i8_kernel<<<grid_of(blocks, 64), 256, 0, s>>>(in, abuf, g, pl.K, pl.Kpad, pad);
    }
    GLOWB200_CUDA_OK(cudaGetLastError());
    a = abuf;
  }
  const int8_t *b = filter;
  if (pl.f_bytes) {
    int8_t *fbuf = reinterpret_cast<int8_t *>(ws + pl.a_bytes);
    const int64_t blocks = ((int64_t)g.OC * pl.Kpad + 255) / 256;
    pad_rows_i8_kernel<<<grid_of(blocks, 16), 256, 0, s>>>(filter, fbuf, g.OC, pl.K, pl.Kpad);
    GLOWB200_CUDA_OK(cudaGetLastError());
    b = fbuf;
    filter_row_sums = nullptr;  // recomputed over the padded copy (same values; keeps one code path)
  }
  p.M = (int)pl.M;
  p.N = g.OC;
  p.K = pl.Kpad;
  p.k_corr = pl.K;
  return run_gemm(p, a, b, filter_row_sums, (flags & GLOWB200_FC_WEIGHT_OFFSETS_ZERO) != 0, 0, ws + pl.a_bytes + pl.f_bytes,
                  pl.core_bytes, s);
}

}  // namespace
}  // namespace glowb200

using namespace glowb200;

extern "C" size_t glowb200_conv2d_workspace_bytes(const int64_t *out_dims, const int64_t *in_dims,
                                                  const int64_t *filter_dims, const int64_t *kernels,
                                                  const int64_t *strides, const int64_t *pads, int64_t group,
                                                  const int64_t *dilation) {
  ConvGeom g;
  if (geom_from_dims(g, out_dims, in_dims, filter_dims, kernels, strides, pads, group, dilation) != GLOWB200_OK) return 0;
  const ConvPlan pl = plan_conv(g, false);
  return pl.a_bytes + pl.f_bytes + pl.core_bytes;
}

namespace {
int channelwise_params(GemmParams &p, ConvGeom &g,
    int8_t *out, const int8_t *in, const int8_t *filter, const int32_t *bias, const int64_t *out_dims,
    const int64_t *in_dims, const int64_t *filter_dims, const int64_t *kernels, const int64_t *strides,
    const int64_t *pads, int64_t group, const int64_t *dilation, int32_t out_offset, int32_t in_offset,
    const int32_t *filter_offsets, const int32_t *bias_offsets, const int32_t *bias_pre, const int32_t *bias_post,
    const int32_t *bias_scale, const int32_t *out_pre, const int32_t *out_post, const int32_t *out_scale, int32_t act_type,
    const int32_t *act_args, int flags,
    int32_t *status) {
  if (int rc = geom_from_dims(g, out_dims, in_dims, filter_dims, kernels, strides, pads, group, dilation)) return rc;
  if ((int64_t)g.N * g.OH * g.OW * g.OC == 0) return GLOWB200_OK;  // run_conv has nothing to do either
  GLOWB200_REQUIRE(out && in && filter && bias && filter_offsets && bias_offsets && bias_pre && bias_post && bias_scale &&
                       out_pre && out_post && out_scale, "NULL tensor pointer");
  GLOWB200_REQUIRE(act_type >= 0 && act_type <= 5 && act_type != 3 && act_type != 4,
                   "fused activation %d is not defined for quantized convolution", act_type);
  GLOWB200_REQUIRE(act_type == 0 || act_type == 1 || act_args != nullptr, "activation arguments missing");
  p = GemmParams{};
  p.out = out;
  p.bias = bias;
  p.b_offsets = filter_offsets;
  p.bias_offsets = bias_offsets;
  p.bias_pre = bias_pre; p.bias_post = bias_post; p.bias_scale = bias_scale;
  p.out_pre = out_pre; p.out_post = out_post; p.out_scale = out_scale;
  p.status = status;
  p.a_offset = in_offset; p.out_offset = out_offset;
  p.act_type = act_type;
  p.bias_is_i8 = (flags & GLOWB200_FC_BIAS_INT8) ? 1 : 0;
  if (act_type == 2) { p.act_args[0] = act_args[0]; p.act_args[1] = act_args[1]; }
  if (act_type == 5) { p.act_args[0] = act_args[0]; p.act_args[1] = act_args[1]; p.act_args[2] = act_args[2]; }
  return GLOWB200_OK;
}
}  // namespace

extern "C" int glowb200_channelwise_quantized_conv2d_i8_i32(    int8_t *out, const int8_t *in, const int8_t *filter, const int32_t *bias, const int64_t *out_dims,
    const int64_t *in_dims, const int64_t *filter_dims, const int64_t *kernels, const int64_t *strides,
    const int64_t *pads, int64_t group, const int64_t *dilation, int32_t out_offset, int32_t in_offset,
    const int32_t *filter_offsets, const int32_t *bias_offsets, const int32_t *bias_pre, const int32_t *bias_post,
    const int32_t *bias_scale, const int32_t *out_pre, const int32_t *out_post, const int32_t *out_scale, int32_t act_type,
    const int32_t *act_args, const int32_t *filter_row_sums, int flags, void *workspace, size_t workspace_bytes,
    int32_t *status, glowb200_stream_t stream) {
  GemmParams p;
  ConvGeom g;
  if (int rc = channelwise_params(p, g, out, in, filter, bias, out_dims, in_dims, filter_dims, kernels, strides, pads, group, dilation,
                                  out_offset, in_offset, filter_offsets, bias_offsets, bias_pre, bias_post, bias_scale, out_pre,
                                  out_post, out_scale, act_type, act_args, flags, status)) return rc;
  return run_conv(p, in, filter, g, filter_row_sums, flags, workspace, workspace_bytes, reinterpret_cast<cudaStream_t>(stream));
}

namespace {
int pair_geometry(ConvGeom &a, ConvGeom &b, const int64_t *in_dims, const int64_t *mid_dims, const int64_t *out_dims,
                  const glowb200_conv_layer *first, const glowb200_conv_layer *second) {
  GLOWB200_REQUIRE(first && second, "NULL layer");
  if (int rc = geom_from_dims(a, mid_dims, in_dims, first->filter_dims, first->kernels, first->strides, first->pads, first->group,
                              first->dilation)) return rc;
  return geom_from_dims(b, out_dims, mid_dims, second->filter_dims, second->kernels, second->strides, second->pads, second->group,
                        second->dilation);
}
// What a convolution may ask of the workspace, and the bytes of a pair's tensor in between.
size_t conv_bytes(const ConvGeom &g) {
  const ConvPlan pl = plan_conv(g, false);
  return pl.a_bytes + pl.f_bytes + pl.core_bytes;
}
size_t mid_bytes(const ConvGeom &a) { return align_up((size_t)a.N * a.OH * a.OW * a.OC, 256); }
}  // namespace

extern "C" size_t glowb200_channelwise_quantized_conv2d_pair_workspace_bytes(
    const int64_t *in_dims, const int64_t *mid_dims, const int64_t *out_dims, const glowb200_conv_layer *first,
    const glowb200_conv_layer *second) {
  ConvGeom a, b;
  if (pair_geometry(a, b, in_dims, mid_dims, out_dims, first, second) != GLOWB200_OK) return 0;
  const size_t x = conv_bytes(a), y = conv_bytes(b);
  return mid_bytes(a) + (x > y ? x : y);
}

// A pointwise layer in front of a window over 64 or a multiple of 128 channels writes the padded buffer itself
// (PaddedOut): as launches of their own the copies into it took 139 + 45 us of 1128 of a ResNet-50 batch of 64.
extern "C" int glowb200_channelwise_quantized_conv2d_pair_i8_i32(
    int8_t *out, const int8_t *in, const int64_t *in_dims, const int64_t *mid_dims, const int64_t *out_dims,
    const glowb200_conv_layer *first, const glowb200_conv_layer *second, void *workspace, size_t workspace_bytes,
    int32_t *status, glowb200_stream_t stream) {
  ConvGeom a, b;
  if (int rc = pair_geometry(a, b, in_dims, mid_dims, out_dims, first, second)) return rc;
  if ((int64_t)b.N * b.OH * b.OW * b.OC == 0) return GLOWB200_OK;
  GLOWB200_REQUIRE((int64_t)a.N * a.OH * a.OW * a.OC > 0, "a result of an empty tensor");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const size_t mid = mid_bytes(a);
  if (workspace == nullptr || workspace_bytes < mid)
    return set_error(GLOWB200_ERR_WORKSPACE_TOO_SMALL, "workspace of %zu bytes given, %zu needed", workspace_bytes,
                     glowb200_channelwise_quantized_conv2d_pair_workspace_bytes(in_dims, mid_dims, out_dims, first, second));
  GLOWB200_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, "workspace must be 256-byte aligned");
  uint8_t *ws = reinterpret_cast<uint8_t *>(workspace);
  GemmParams p, q;
  auto params = [&](GemmParams &p, ConvGeom &g, const glowb200_conv_layer *l, int8_t *to, const int8_t *from, const int64_t *from_dims,
                    const int64_t *to_dims) {
    return channelwise_params(p, g, to, from, l->filter, l->bias, to_dims, from_dims, l->filter_dims, l->kernels, l->strides, l->pads,
                              l->group, l->dilation, l->out_offset, l->in_offset, l->filter_offsets, l->bias_offsets, l->bias_pre,
                              l->bias_post, l->bias_scale, l->out_pre, l->out_post, l->out_scale, l->act_type, l->act_args, l->flags, status);
  };
  int8_t *between = reinterpret_cast<int8_t *>(ws);
  if (int rc = params(p, a, first, between, in, in_dims, mid_dims)) return rc;
  if (int rc = params(q, b, second, out, between, mid_dims, out_dims)) return rc;
  const ConvPlan pa = plan_conv(a, (first->flags & GLOWB200_FC_FORCE_ANY_SHAPE_KERNEL) != 0);
  const ConvPlan pb = plan_conv(b, (second->flags & GLOWB200_FC_FORCE_ANY_SHAPE_KERNEL) != 0);
  ShiftedRows r;
  if (!pa.direct && !pa.need_im2col && !pb.direct && (reinterpret_cast<uintptr_t>(second->filter) & 15) == 0 &&
      i8_tiles_direct(pa.M, a.OC, pa.K, in, first->filter, between) && !i8_skinny_conv_wins(b) && shifted_rows(b, pb, second->flags, r)) {
    const int sides = r.planes == 1 ? 1 : 2;  // (a parity plane is half as high and wide as the padded input)
    const size_t need = r.input_bytes + r.pair_bytes + (pa.core_bytes > pb.core_bytes ? pa.core_bytes : pb.core_bytes);
    if (sides * r.h >= b.H + b.PT && sides * r.w >= b.W + b.PL && workspace_bytes >= need) {
      PaddedOut &o = p.padded;
      o.kind = sides;
      o.images = b.N; o.h = b.H; o.w = b.W;
      o.hp = sides * r.h; o.wp = sides * r.w;
      o.top = b.PT; o.left = b.PL;
      o.plane = (int)r.rows;
      o.word = (uint32_t)pad_word(q.a_offset);
      if (r.pairs) {
        o.filter = second->filter;
        o.pairs = reinterpret_cast<int8_t *>(ws + r.input_bytes);
        o.filter_rows = b.OC * b.KH;
        o.kw = b.KW;
      }
      uint8_t *core = ws + r.input_bytes + r.pair_bytes;
      p.M = (int)pa.M;
      p.N = a.OC;
      p.K = p.k_corr = pa.K;
      if (int rc = run_gemm(p, in, first->filter, first->filter_row_sums, (first->flags & GLOWB200_FC_WEIGHT_OFFSETS_ZERO) != 0, 0, core,
                            pa.core_bytes, s)) return rc;
      return run_shifted_rows(q, b, pb, r, between, o.pairs ? o.pairs : second->filter, second->filter_row_sums, core, s);
    }
  }
  if (int rc = run_conv(p, in, first->filter, a, first->filter_row_sums, first->flags, ws + mid, workspace_bytes - mid, s)) return rc;
  return run_conv(q, between, second->filter, b, second->filter_row_sums, second->flags, ws + mid, workspace_bytes - mid, s);
}

// The Add rides in the contraction's drain when the layer is a plain product with whole 16-byte rows and the
// Add's parameters are of the ordinary kind: the layer's own result then never reaches memory (200,704 x 64 x 256
// with its Add: 74 us as two launches, 43 as one).
extern "C" int glowb200_channelwise_quantized_conv2d_add_i8(    int8_t *out, const int8_t *in, const int8_t *filter, const int32_t *bias, const int64_t *out_dims,
    const int64_t *in_dims, const int64_t *filter_dims, const int64_t *kernels, const int64_t *strides,
    const int64_t *pads, int64_t group, const int64_t *dilation, int32_t out_offset, int32_t in_offset,
    const int32_t *filter_offsets, const int32_t *bias_offsets, const int32_t *bias_pre, const int32_t *bias_post,
    const int32_t *bias_scale, const int32_t *out_pre, const int32_t *out_post, const int32_t *out_scale, int32_t act_type,
    const int32_t *act_args, const int32_t *filter_row_sums, int flags, void *workspace, size_t workspace_bytes,
    int32_t *status, const int8_t *residual, int32_t dest_offset, int32_t lhs_offset, int32_t residual_offset,
    int32_t lhs_pre, int32_t lhs_post, int32_t lhs_scale, int32_t residual_pre, int32_t residual_post, int32_t residual_scale,
    int32_t splat, glowb200_stream_t stream) {
  GemmParams p;
  ConvGeom g;
  if (int rc = channelwise_params(p, g, out, in, filter, bias, out_dims, in_dims, filter_dims, kernels, strides, pads, group, dilation,
                                  out_offset, in_offset, filter_offsets, bias_offsets, bias_pre, bias_post, bias_scale, out_pre,
                                  out_post, out_scale, act_type, act_args, flags, status)) return rc;
  const int64_t n = (int64_t)g.N * g.OH * g.OW * g.OC;
  if (n == 0) return GLOWB200_OK;
  GLOWB200_REQUIRE(residual != nullptr, "NULL tensor pointer");
  GLOWB200_REQUIRE(splat >= -128 && splat <= 127, "splat value outside int8");
  auto whole = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  const ConvPlan pl = plan_conv(g, (flags & GLOWB200_FC_FORCE_ANY_SHAPE_KERNEL) != 0);
  if (!pl.direct && !pl.need_im2col && (flags & GLOWB200_FC_WEIGHT_OFFSETS_ZERO) && act_type <= 1 && g.OC % 16 == 0 && whole(out) &&
      whole(in) && whole(filter) && whole(residual) &&
      make_add_quant(p.add, dest_offset, lhs_offset, residual_offset, lhs_pre, lhs_post, lhs_scale, residual_pre, residual_post,
                     residual_scale, splat)) {
    p.residual = residual;
    return run_conv(p, in, filter, g, filter_row_sums, flags, workspace, workspace_bytes, reinterpret_cast<cudaStream_t>(stream));
  }
  if (int rc = run_conv(p, in, filter, g, filter_row_sums, flags, workspace, workspace_bytes, reinterpret_cast<cudaStream_t>(stream)))
    return rc;
  return glowb200_element_add_maxsplat_i8(out, out, residual, n, dest_offset, lhs_offset, residual_offset, lhs_pre, lhs_post, lhs_scale,
                                          residual_pre, residual_post, residual_scale, splat, stream);
}

extern "C" int glowb200_conv2d_i8_i32(
    int8_t *out, const int8_t *in, const int8_t *filter, const int32_t *bias, const int64_t *out_dims,
    const int64_t *in_dims, const int64_t *filter_dims, const int64_t *kernels, const int64_t *strides,
    const int64_t *pads, int64_t group, int32_t out_offset, int32_t in_offset, int32_t filter_offset, int32_t bias_offset,
    int32_t bias_pre, int32_t bias_post, int32_t bias_scale, int32_t out_pre, int32_t out_post, int32_t out_scale,
    const int64_t *dilation, int32_t act_type, const int32_t *act_args, int flags, void *workspace, size_t workspace_bytes,
    int32_t *status, glowb200_stream_t stream) {
  ConvGeom g;
  if (int rc = geom_from_dims(g, out_dims, in_dims, filter_dims, kernels, strides, pads, group, dilation)) return rc;
  if ((int64_t)g.N * g.OH * g.OW * g.OC == 0) return GLOWB200_OK;
  GLOWB200_REQUIRE(out && in && filter && bias, "NULL tensor pointer");
  GLOWB200_REQUIRE(act_type >= 0 && act_type <= 5 && act_type != 3 && act_type != 4,
                   "fused activation %d is not defined for quantized convolution", act_type);
  GLOWB200_REQUIRE(act_type == 0 || act_type == 1 || act_args != nullptr, "activation arguments missing");
  GemmParams p{};
  p.out = out;
  p.bias = bias;
  p.status = status;
  p.a_offset = in_offset; p.out_offset = out_offset; p.bias_offset = bias_offset;
  p.uniform = 1;
  p.u_b_offset = filter_offset;
  p.u_bias_pre = bias_pre; p.u_bias_post = bias_post; p.u_bias_scale = bias_scale;
  p.u_out_pre = out_pre; p.u_out_post = out_post; p.u_out_scale = out_scale;
  p.act_type = act_type;
  p.bias_is_i8 = (flags & GLOWB200_FC_BIAS_INT8) ? 1 : 0;
  if (act_type == 2) { p.act_args[0] = act_args[0]; p.act_args[1] = act_args[1]; }
  if (act_type == 5) { p.act_args[0] = act_args[0]; p.act_args[1] = act_args[1]; p.act_args[2] = act_args[2]; }
  if (filter_offset == 0) flags |= GLOWB200_FC_WEIGHT_OFFSETS_ZERO;
  return run_conv(p, in, filter, g, nullptr, flags, workspace, workspace_bytes, reinterpret_cast<cudaStream_t>(stream));
}
