// Two companions of the int8 contraction core (qgemm.cu):
//   * i8_skinny_kernel -- products with few rows in ONE launch, straight from the operands as they
//     are (any row length, any alignment, right-hand side [N, K] or [K, N], sums included);
//   * i8_prepare_operands_kernel -- copies of the operands in the form the tcgen05 core loads
//     (rows of a multiple of 16 bytes, zero padded; [K, N] right-hand sides transposed) together
//     with the row sums the offsets need, both operands in one launch.
#include "qgemm.cuh"


namespace glowb200 {
namespace {

// Predicated loads (0 when `take` is false), as single instructions: a branch round each load would
// make a thread wait for one before it asks for the next.  volatile: they stay behind pdl_wait().
__device__ __forceinline__ uint32_t load_if(const uint32_t *p, bool take) {
  uint32_t v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.u32 %0, 0;\n\t@p ld.global.u32 %0, [%1];\n\t}"
               : "=r"(v) : "l"(p), "r"((uint32_t)take));
  return v;
}
__device__ __forceinline__ uint4 load_if(const uint4 *p, bool take) {
  uint4 v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
               "@p ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "r"((uint32_t)take));
  return v;
}

// The first `valid` (any number) of four bytes, the others cleared.
__device__ __forceinline__ uint32_t keep_bytes(uint32_t v, int valid) {
  return valid >= 4 ? v : valid <= 0 ? 0u : v & (0xffffffffu >> (32 - 8 * valid));
}

// Four bytes at an address of any alignment, bytes from `valid` on read as zero.  Only aligned
// words that hold at least one wanted byte are touched.
__device__ __forceinline__ uint32_t load4(const int8_t *p, int valid) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  const int sh = (int)(a & 3);
  const uint32_t *w = reinterpret_cast<const uint32_t *>(a - sh);
  const uint32_t lo = load_if(w, valid > 0), hi = load_if(w + 1, sh != 0 && valid > 4 - sh);
  return keep_bytes(__funnelshift_r(lo, hi, 8 * sh), valid);
}

// Sixteen bytes likewise (five words instead of four loads of two).
__device__ __forceinline__ uint4 load16(const int8_t *p, int valid) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  const int sh = (int)(a & 3);
  const uint32_t *w = reinterpret_cast<const uint32_t *>(a - sh);
  uint32_t r[5], o[4];
#pragma unroll
  for (int i = 0; i < 5; i++) r[i] = load_if(w + i, 4 * i - sh < valid && (i < 4 || sh != 0));
#pragma unroll
  for (int i = 0; i < 4; i++) o[i] = keep_bytes(__funnelshift_r(r[i], r[i + 1], 8 * sh), valid - 4 * i);
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// 4 x 4 byte transpose: word i of the result holds byte i of r[0..3].
__device__ __forceinline__ void transpose4x4(const uint32_t (&r)[4], uint32_t (&c)[4]) {
  const uint32_t a = __byte_perm(r[0], r[1], 0x5140), b = __byte_perm(r[2], r[3], 0x5140);  // bytes 0, 1 interleaved
  const uint32_t d = __byte_perm(r[0], r[1], 0x7362), e = __byte_perm(r[2], r[3], 0x7362);  // bytes 2, 3
  c[0] = __byte_perm(a, b, 0x5410);
  c[1] = __byte_perm(a, b, 0x7632);
  c[2] = __byte_perm(d, e, 0x5410);
  c[3] = __byte_perm(d, e, 0x7632);
}

__device__ __forceinline__ int32_t byte_sum(uint32_t w, int32_t acc) { return __dp4a((int32_t)w, 0x01010101, acc); }
__device__ __forceinline__ int32_t byte_sum(const uint4 &v, int32_t acc) {
  return byte_sum(v.w, byte_sum(v.z, byte_sum(v.y, byte_sum(v.x, acc))));
}

// ---------------------------------------------------------------------------------------
// Operand preparation
// ---------------------------------------------------------------------------------------
// Bound by memory: 2048 x 479 and 1024 x 479 are copied (and summed) in about 2.5 us, where the
// thread-per-output kernel that used to take row lengths off the 16-byte grid needed 784 us for the
// product; a 4096 x 4096 right-hand side is transposed in about 10 us (30 us as 32 x 32-byte tiles).
constexpr int kPrepThreads = 256;
constexpr int kPrepTile = 64;  // columns of a transposed tile, and its depth per step

// blocks [0, p.a_blocks): the left operand, a warp per row; the others: the right operand, a warp
// per row or, transposed, blocks of 64 columns by a slice of the depth.
__global__ void __launch_bounds__(kPrepThreads) i8_prepare_operands_kernel(const __grid_constant__ PrepParams p) {
  __shared__ uint32_t tile[kPrepTile * (kPrepTile / 4 + 1)];
  __shared__ int32_t col_sums[kPrepTile];
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool left = (int)blockIdx.x < p.a_blocks;
  const PrepSide &o = left ? p.a : p.b;
  const int block = left ? (int)blockIdx.x : (int)blockIdx.x - p.a_blocks;
  if (!o.transpose) {
    const int row = block * (kPrepThreads / 32) + warp;
    if (row >= o.rows) return;
    const int8_t *src = o.src + (size_t)row * o.K;
    uint32_t *dst = o.dst ? reinterpret_cast<uint32_t *>(o.dst + (size_t)row * o.pitch) : nullptr;
    int32_t sum = 0;
    if (o.K == o.pitch && (reinterpret_cast<uintptr_t>(o.src) & 15) == 0) {
#pragma unroll 4
      for (int w = lane; w < (o.K >> 4); w += 32) {
        const uint4 v = reinterpret_cast<const uint4 *>(src)[w];
        if (dst) reinterpret_cast<uint4 *>(dst)[w] = v;
        sum = byte_sum(v, sum);
      }
    } else {
      // (sixteen bytes, five words that lie across them, at a time: one word per lane and step took a row of 3000 bytes through
      // six fetches one after the other: 400 x 3000 x 900 17.4 -> 14.5 us in all, 756 x 3141 x 107 18.1 -> 15.0)
#pragma unroll 4
      for (int w = lane; w < (o.pitch >> 4); w += 32) {
        const uint4 v = load16(src + 16 * w, o.K - 16 * w);
        if (dst) reinterpret_cast<uint4 *>(dst)[w] = v;
        sum = byte_sum(v, sum);
      }
    }
    if (o.sums) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
      if (lane == 0) o.sums[row] = sum;
    }
    return;
  }
  // [K, rows] -> [rows, pitch]: a thread takes 4 x 4 bytes (four words down, transposed in
  // registers), the tile passes through shared memory and leaves as 16-byte pieces of its rows.
  const int strips = (o.rows + kPrepTile - 1) / kPrepTile;
  const int n0 = (block % strips) * kPrepTile, part = block / strips;
  const int k_begin = part * o.k_span, k_end = min(o.pitch, k_begin + o.k_span);
  const int nq = threadIdx.x & 15, kq = threadIdx.x >> 4;
  if (threadIdx.x < kPrepTile) col_sums[threadIdx.x] = 0;
  __syncthreads();
  int32_t sums[4] = {0, 0, 0, 0};
  uint32_t r[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int k = k0 + 4 * kq + i, n = n0 + 4 * nq;
      r[i] = load4(o.src + (size_t)k * o.rows + n, k < o.K ? o.rows - n : 0);
    }
  };
  fetch(k_begin);
  for (int k0 = k_begin; k0 < k_end; k0 += kPrepTile) {
    uint32_t c[4];
    transpose4x4(r, c);
    if (k0 + kPrepTile < k_end) fetch(k0 + kPrepTile);  // on its way while this tile passes through shared memory
    __syncthreads();  // the tile before this one has left
#pragma unroll
    for (int i = 0; i < 4; i++) {
      tile[(4 * nq + i) * (kPrepTile / 4 + 1) + kq] = c[i];
      sums[i] = byte_sum(c[i], sums[i]);
    }
    __syncthreads();
    const int n = threadIdx.x >> 2, piece = threadIdx.x & 3, k = k0 + 16 * piece;
    if (n0 + n < o.rows && k < k_end) {
      const uint32_t *t = &tile[n * (kPrepTile / 4 + 1) + 4 * piece];
      *reinterpret_cast<uint4 *>(o.dst + (size_t)(n0 + n) * o.pitch + k) = make_uint4(t[0], t[1], t[2], t[3]);
    }
  }
  if (o.sums) {
#pragma unroll
    for (int i = 0; i < 4; i++) atomicAdd(&col_sums[4 * nq + i], sums[i]);
    __syncthreads();
    if (threadIdx.x < kPrepTile && n0 + (int)threadIdx.x < o.rows)
      o.sums[(size_t)part * o.rows + n0 + threadIdx.x] = col_sums[threadIdx.x];
  }
}

// ---------------------------------------------------------------------------------------
// Products with few rows
// ---------------------------------------------------------------------------------------
// What bounds such a product is latency, not the tensor pipe: 8 x 1024 x 1024 reads 1 MB of weights
// and nothing else.  A tcgen05 tile of 128 rows would be mostly padding, and its prologue (tensor
// memory, descriptors, a pipeline to fill), the row sums and any copy of the operands cost launches
// of their own.  Here every warp of a block takes its share of the depth, loads fragments of both
// operands straight from global memory -- 16 contiguous bytes per lane: the order of the depth inside
// a 64-byte step does not matter as long as both operands use the same one -- multiplies them with
// the warp-level int8 MMA, and the block adds its warps' partial products in shared memory (integers:
// exact in any order).  8 x 1024 x 1024: 2.4 us where the tile kernel needs 5.0 and, with weight offsets,
// its row-sum pass 2.6 more; 8 x 4096 x 4096 (16 MB of weights) 12.4 -> 4.8 us.

__device__ __forceinline__ void mma_i8(int32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <bool VEC>
__device__ __forceinline__ uint4 row16(const int8_t *p, int valid) {
  if constexpr (VEC) return load_if(reinterpret_cast<const uint4 *>(p), valid > 0);
  else return load16(p, valid);
}

// MT row tiles of 16, NT column tiles of 8 per block (KN: always 4).  KN: the right-hand side is
// [K, N], its 4 x 4-byte blocks transposed in registers.  VEC: rows of the operands that are read 16
// bytes at a time start on 16-byte boundaries and hold a multiple of 16 bytes.
// CONV: the left-hand row of output pixel (n, oh, ow) is its window of the NHWC input, read where it lies:
// a lane's 16 bytes never straddle two taps (C a multiple of 16), and a tap outside the image reads as
// the input offset, which is how the reference's skipped taps count (libjit_conv.cpp:209-212).
template <int MT, int NT, bool KN, bool VEC, bool CONV>
__global__ void __launch_bounds__(512) i8_skinny_kernel(const int8_t *a, const int8_t *b, const __grid_constant__ GemmParams p,
                                                         int need_a_sums, const __grid_constant__ ConvGeom cg) {
  constexpr int kCols = NT * 8;
  // row pitch of the shared sums: the lanes of one atomic (rows g, columns 2t or 8t) meet in no bank, or in pairs
  constexpr int kPitch = KN ? kCols + 1 : (kCols == 8 ? 8 : kCols + 8);
  // steps whose loads are in flight together
  constexpr int UNROLL = KN ? 2 : 1;
  __shared__ int32_t acc_s[MT * 16 * kPitch];
  __shared__ int32_t a_sum_s[MT * 16], b_sum_s[NT * 8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = (int)(blockDim.x >> 5);
  const int g = lane >> 2, t = lane & 3;
  const int m0 = blockIdx.y * (MT * 16), n0 = blockIdx.x * kCols;
  const int K = p.k_corr, lda = p.a_pitch ? p.a_pitch : p.K;
  for (int i = tid; i < MT * 16 * kPitch; i += blockDim.x) acc_s[i] = 0;
  if (tid < MT * 16) a_sum_s[tid] = 0;
  if (tid < kCols) b_sum_s[tid] = 0;
  __syncthreads();
  pdl_wait();
  pdl_launch_dependents();

  // CONV: first pixel and corner of the windows of this lane's rows g and g + 8 of every row tile
  int pixel[CONV ? MT : 1][2], corner_h[CONV ? MT : 1][2], corner_w[CONV ? MT : 1][2];
  const uint32_t pad_word = (uint32_t)(uint8_t)p.a_offset * 0x01010101u;
  if constexpr (CONV) {
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int row = m0 + 16 * mt + 8 * i + g, r = row < p.M ? row : 0;
        const int ow = r % cg.OW, q = r / cg.OW, oh = q % cg.OH, n = q / cg.OH;
        corner_h[mt][i] = row < p.M ? oh * cg.SH - cg.PT : -(1 << 20);  // (rows that are not there: never inside the image)
        corner_w[mt][i] = ow * cg.SW - cg.PL;
        pixel[mt][i] = (n * cg.H + oh * cg.SH - cg.PT) * cg.W + corner_w[mt][i];
      }
  }

  int32_t acc[MT][NT][4] = {};
  int32_t a_sums[MT][2] = {}, b_sums[NT] = {};
  constexpr int kStep = KN ? 32 : 64;
#pragma unroll UNROLL
  for (int k0 = warp * kStep; k0 < K; k0 += warps * kStep) {
    if constexpr (KN) {
      // lane (g, t): rows k0 + 16h + 4t .. + 3 of columns n0 + 4g .. + 3, so column 4g + i is column g
      // of column tile i; depth 16h + 4t + j is what half h of the fragments holds
      uint32_t bw[2][4];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        uint32_t r[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int k = k0 + 16 * h + 4 * t + j, n = n0 + 4 * g;
          r[j] = load4(b + (size_t)k * p.N + n, k < K ? p.N - n : 0);
        }
        transpose4x4(r, bw[h]);
#pragma unroll
        for (int i = 0; i < 4; i++) b_sums[i] = byte_sum(bw[h][i], b_sums[i]);
      }
#pragma unroll
      for (int mt = 0; mt < MT; mt++) {
        uint32_t aw[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {  // i = 2h + (row half)
          const int row = m0 + 16 * mt + g + 8 * (i & 1), k = k0 + 16 * (i >> 1) + 4 * t;
          aw[i] = load4(a + (size_t)row * lda + k, row < p.M ? K - k : 0);
          a_sums[mt][i & 1] = byte_sum(aw[i], a_sums[mt][i & 1]);
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++) mma_i8(acc[mt][nt], aw[0], aw[1], aw[2], aw[3], bw[0][nt], bw[1][nt]);
      }
    } else {
      const int k = k0 + 16 * t;
      uint4 bv[NT];
#pragma unroll
      for (int nt = 0; nt < NT; nt++) {
        const int n = n0 + 8 * nt + g;
        bv[nt] = row16<VEC>(b + (size_t)n * p.K + k, n < p.N ? K - k : 0);
      }
      int tap_h = 0, tap_w = 0, channel = 0;
      if constexpr (CONV) {
        const int tap = k / cg.C, kh = tap / cg.KW;
        channel = k - tap * cg.C;
        tap_h = kh * cg.DH;
        tap_w = (tap - kh * cg.KW) * cg.DW;
      }
#pragma unroll
      for (int mt = 0; mt < MT; mt++) {
        uint4 lo, hi;
        if constexpr (CONV) {
          uint4 v[2];
          bool in[2];
#pragma unroll
          for (int i = 0; i < 2; i++) {
            in[i] = (unsigned)(corner_h[mt][i] + tap_h) < (unsigned)cg.H && (unsigned)(corner_w[mt][i] + tap_w) < (unsigned)cg.W;
            v[i] = load_if(reinterpret_cast<const uint4 *>(a + (int64_t)(pixel[mt][i] + tap_h * cg.W + tap_w) * cg.C + channel), in[i] && k < K);
          }
          const uint32_t fill = k < K ? pad_word : 0u;
#pragma unroll
          for (int i = 0; i < 2; i++)
            if (!in[i]) v[i] = make_uint4(fill, fill, fill, fill);
          lo = v[0];
          hi = v[1];
        } else {
          const int row = m0 + 16 * mt + g;
          lo = row16<VEC>(a + (size_t)row * lda + k, row < p.M ? K - k : 0);
          hi = row16<VEC>(a + (size_t)(row + 8) * lda + k, row + 8 < p.M ? K - k : 0);
        }
        if (need_a_sums) {
          a_sums[mt][0] = byte_sum(lo, a_sums[mt][0]);
          a_sums[mt][1] = byte_sum(hi, a_sums[mt][1]);
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
          mma_i8(acc[mt][nt], lo.x, hi.x, lo.y, hi.y, bv[nt].x, bv[nt].y);
          mma_i8(acc[mt][nt], lo.z, hi.z, lo.w, hi.w, bv[nt].z, bv[nt].w);
        }
      }
#pragma unroll
      for (int nt = 0; nt < NT; nt++) b_sums[nt] = byte_sum(bv[nt], b_sums[nt]);
    }
  }
  if (warp * kStep < K) {
    // accumulator i of a tile: row g + 8 * (i >> 1), column 2t + (i & 1)
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int nt = 0; nt < NT; nt++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int c = 2 * t + (i & 1);
          atomicAdd(&acc_s[(16 * mt + g + 8 * (i >> 1)) * kPitch + (KN ? 4 * c + nt : 8 * nt + c)], acc[mt][nt][i]);
        }
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      int32_t v = b_sums[nt];
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      if (t == 0) atomicAdd(&b_sum_s[KN ? 4 * g + nt : 8 * nt + g], v);
    }
    if (need_a_sums) {
#pragma unroll
      for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
          int32_t v = a_sums[mt][i];
          v += __shfl_xor_sync(0xffffffffu, v, 1);
          v += __shfl_xor_sync(0xffffffffu, v, 2);
          if (t == 0) atomicAdd(&a_sum_s[16 * mt + 8 * i + g], v);
        }
    }
  }
  __syncthreads();
  // a thread keeps its column (the block's thread count is a multiple of the columns)
  const int c = tid % kCols, j = n0 + c;
  if (j >= p.N) return;
  if (p.float_out) {
    const int32_t b_off = p.b_offsets ? p.b_offsets[j] : p.u_b_offset;
    const float cs = p.col_scales ? p.col_scales[j] : p.u_col_scale, bias = p.bias_f32[j];
    for (int i = tid / kCols; i < MT * 16 && m0 + i < p.M; i += blockDim.x / kCols) {
      const int32_t v = (int32_t)((uint32_t)acc_s[i * kPitch + c] - (uint32_t)b_off * (uint32_t)a_sum_s[i]);
      p.out_f16[(size_t)(m0 + i) * p.N + j] =
          __float2half_rn(__fadd_rn(__fmul_rn((float)v, __fmul_rn(p.row_scales[m0 + i], cs)), bias));
    }
    return;
  }
  const ColQuant q = col_quant(p, j);
  uint32_t base = (uint32_t)K * (uint32_t)p.a_offset * (uint32_t)q.b_off - (uint32_t)p.a_offset * (uint32_t)b_sum_s[c];
  if (p.bias)
    base += (uint32_t)scale32(load_bias(p, j) - (p.bias_offsets ? p.bias_offsets[j] : p.bias_offset), q.bias_pre, q.bias_post,
                              q.bias_scale, 0);
  for (int i = tid / kCols; i < MT * 16 && m0 + i < p.M; i += blockDim.x / kCols) {
    const uint32_t v = (uint32_t)acc_s[i * kPitch + c] + base - (uint32_t)q.b_off * (uint32_t)a_sum_s[i];
    int32_t x = clip_i8(activation_i32(scale32((int32_t)v, q.out_pre, q.out_post, q.out_scale, p.out_offset), p));
    if (p.residual)
      x = (int32_t)add_quant_word((uint32_t)x & 0xffu, (uint8_t)p.residual[(size_t)(m0 + i) * p.N + j], p.add);
    p.out[(size_t)(m0 + i) * p.N + j] = (int8_t)x;
  }
}

template <int MT, int NT, bool KN>
cudaError_t launch_skinny(const GemmParams &p, const int8_t *a, const int8_t *b, bool vec, int need_a_sums, cudaStream_t s,
                          const ConvGeom *conv = nullptr) {
  const dim3 grid((unsigned)((p.N + 8 * NT - 1) / (8 * NT)), (unsigned)((p.M + 16 * MT - 1) / (16 * MT)));
  // Warps share the depth in equal parts: up to 16 of them, 8 once the blocks alone fill the SMs.  (CTAs of a
  // cluster sharing it as well, adding up through distributed shared memory, cost more than they brought:
  // 8 x 1024 x 1024 2.5 -> 3.4 us.)
  const int steps = (p.k_corr + (KN ? 31 : 63)) / (KN ? 32 : 64), most = (int64_t)grid.x * grid.y >= 220 ? 8 : 16;
  const int rounds = (steps + most - 1) / most, warps = (steps + rounds - 1) / rounds;
  const unsigned threads = 32 * (warps < 4 ? 4 : warps);
  if constexpr (!KN) {
    if (conv) return launch_pdl(i8_skinny_kernel<MT, NT, KN, true, true>, grid, threads, 0, s, a, b, p, need_a_sums, *conv);
    if (vec) return launch_pdl(i8_skinny_kernel<MT, NT, KN, true, false>, grid, threads, 0, s, a, b, p, need_a_sums, ConvGeom{});
  }
  return launch_pdl(i8_skinny_kernel<MT, NT, KN, false, false>, grid, threads, 0, s, a, b, p, need_a_sums, ConvGeom{});
}

// Rows and columns of a block's tile, in MMA tiles of 16 and 8.  Small weights: 16 x 32 (the four column
// tiles share a row's loads), fewer columns while the tiles leave SMs idle, more rows once they are four
// to an SM -- 3 x 3 layers of one image, device time: 64 channels at 56 x 56 9.5 (as 64 x 8) -> 3.9 us, 256 at
// 14 x 14 5.5 -> 4.6, 512 at 7 x 7 9.1 -> 5.0.  Weights of 4 MB and more: all rows in a block as far as they fit,
// so that the weights are read once.
struct SkinnyTile { int mt, nt; };
SkinnyTile skinny_tile(int64_t M, int64_t N, int64_t K, bool kn) {
  auto blocks = [&](int mt, int nt) { return ((M + 16 * mt - 1) / (16 * mt)) * ((N + 8 * nt - 1) / (8 * nt)); };
  constexpr int64_t sms = kB200Sms;
  SkinnyTile t{M <= 16 ? 1 : M <= 32 ? 2 : 4, 4};
  if (N * K >= (1 << 22)) {
    if (!kn) t.nt = N >= 8 * 4 * (t.mt == 4 ? 110 : sms * 2) ? 4 : N >= 8 * 2 * sms ? 2 : 1;
    return t;
  }
  if (kn) {
    while (t.mt > 1 && blocks(t.mt, 4) < 100) t.mt /= 2;
    return t;
  }
  t.mt = 1;
  while (t.nt > 1 && blocks(1, t.nt) < 100) t.nt /= 2;
  if (K > 64 && blocks(1, 4) >= sms * 4) t.mt = blocks(2, 4) >= sms * 6 ? 4 : 2;
  return t;
}

cudaError_t launch_skinny_tile(SkinnyTile t, const GemmParams &p, const int8_t *a, const int8_t *b, bool vec, int need, cudaStream_t s,
                               const ConvGeom *conv) {
#define GLOWB200_SKINNY(MT)                                                                            \
  (t.nt == 1 ? launch_skinny<MT, 1, false>(p, a, b, vec, need, s, conv)                                \
             : t.nt == 2 ? launch_skinny<MT, 2, false>(p, a, b, vec, need, s, conv) : launch_skinny<MT, 4, false>(p, a, b, vec, need, s, conv))
  return t.mt == 1 ? GLOWB200_SKINNY(1) : t.mt == 2 ? GLOWB200_SKINNY(2) : GLOWB200_SKINNY(4);
#undef GLOWB200_SKINNY
}

}  // namespace

// Measured against the tcgen05 kernel (device time per product, us): 8 x 1024 x 1024 2.4 against 5.0,
// 64 x 4096 x 4096 10.1 against 12.1, 128 x 1024 x 1024 4.5 against 5.1, 512 x 512 x 1024 7.8 against
// 4.1; many results per product cost too (their stores are narrow).  A [K, N] right-hand side, whose
// fragments are four loads and a byte transpose each: 32 x 4096 x 4096 15 against 23 with its copy,
// 64 x 1024 x 1024 9.5 against 7.1, 512 x 256 x 256 4.8 against 5.2.
bool i8_skinny_wins(int64_t M, int64_t N, int64_t K, bool b_is_kn) {
  if (M <= (b_is_kn ? 32 : kSkinnyRows)) return true;
  return M * N <= (1 << 18) && M * N * K <= (b_is_kn ? 1ll << 25 : 1ll << 27);
}

int run_gemm_skinny(GemmParams p, const int8_t *a, const int8_t *b, bool b_is_kn, bool b_offsets_zero, cudaStream_t s) {
  if (p.k_corr == 0) p.k_corr = p.K;
  const int need = b_offsets_zero ? 0 : 1;
  const bool vec = (p.K % 16) == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
  const SkinnyTile t = skinny_tile(p.M, p.N, p.k_corr, b_is_kn);
  cudaError_t e;
  if (b_is_kn) {
    e = t.mt == 1 ? launch_skinny<1, 4, true>(p, a, b, false, need, s) : t.mt == 2 ? launch_skinny<2, 4, true>(p, a, b, false, need, s)
                                                                                 : launch_skinny<4, 4, true>(p, a, b, false, need, s);
  } else {
    e = launch_skinny_tile(t, p, a, b, vec, need, s, nullptr);
  }
  if (e != cudaSuccess) return set_error(GLOWB200_ERR_CUDA, "few-row contraction launch failed: %s", cudaGetErrorString(e));
  return GLOWB200_OK;
}

bool i8_skinny_conv_wins(const ConvGeom &g) {
  // (against a padded copy or im2col matrix and the tile kernel, two launches of 2 and 7 us for the 3 x 3
  // layers of a ResNet-50 on one image)
  const int64_t M = (int64_t)g.N * g.OH * g.OW, K = (int64_t)g.KH * g.KW * g.C;
  return g.G == 1 && g.C % 16 == 0 && M * g.OC <= (1 << 19) && M * g.OC * K <= (1ll << 28);
}

int run_conv_skinny(GemmParams p, const int8_t *in, const int8_t *filter, const ConvGeom &g, bool b_offsets_zero, cudaStream_t s) {
  p.M = g.N * g.OH * g.OW;
  p.N = g.OC;
  p.K = p.k_corr = g.KH * g.KW * g.C;
  const int need = b_offsets_zero ? 0 : 1;
  const cudaError_t e = launch_skinny_tile(skinny_tile(p.M, p.N, p.K, false), p, in, filter, true, need, s, &g);
  if (e != cudaSuccess) return set_error(GLOWB200_ERR_CUDA, "small convolution launch failed: %s", cudaGetErrorString(e));
  return GLOWB200_OK;
}

void prep_side_rows(PrepSide &o, const int8_t *src, int8_t *dst, int32_t *sums, int rows, int K, int pitch) {
  o = PrepSide{src, dst, sums, rows, K, pitch, 0, 0};
}

int prep_transposed_parts(int64_t rows, int64_t pitch) {
  const int64_t strips = (rows + kPrepTile - 1) / kPrepTile, steps = (pitch + kPrepTile - 1) / kPrepTile;
  int64_t parts = (8 * kB200Sms + strips - 1) / strips;
  if (parts > kMaxSumParts) parts = kMaxSumParts;
  if (parts > steps) parts = steps;
  const int64_t span = (steps + parts - 1) / parts;  // steps per part; no part may be empty
  return (int)((steps + span - 1) / span);
}

void prep_side_transposed(PrepSide &o, const int8_t *src, int8_t *dst, int32_t *sums, int rows, int K, int pitch) {
  const int parts = prep_transposed_parts(rows, pitch);
  const int steps = (pitch + kPrepTile - 1) / kPrepTile;
  o = PrepSide{src, dst, sums, rows, K, pitch, 1, (steps + parts - 1) / parts * kPrepTile};
}

int run_prepare_operands(PrepParams p, cudaStream_t s) {
  auto blocks = [](const PrepSide &o) -> int64_t {
    if (o.src == nullptr || o.rows == 0) return 0;
    if (!o.transpose) return (o.rows + kPrepThreads / 32 - 1) / (kPrepThreads / 32);
    return (int64_t)((o.rows + kPrepTile - 1) / kPrepTile) * prep_transposed_parts(o.rows, o.pitch);
  };
  const int64_t na = blocks(p.a), nb = blocks(p.b);
  if (na + nb == 0) return GLOWB200_OK;
  GLOWB200_REQUIRE(na + nb < (1ll << 31), "operands too large to prepare");
  p.a_blocks = (int)na;
  GLOWB200_CUDA_OK(launch_pdl(i8_prepare_operands_kernel, dim3((unsigned)(na + nb)), kPrepThreads, 0, s, p));
  return GLOWB200_OK;
}

}  // namespace glowb200
