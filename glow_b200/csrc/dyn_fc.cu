// Dynamically quantized fully connected layers: DynamicRowwiseQuantizedFullyConnected and
// DynamicQuantizedFullyConnected.
//
// Reference: fwdDynRowwiseQuantizedFullyConnectedInstPreimpl / ...InstImpl and
// fwdDynamicQuantizedFullyConnectedInst (lib/Backends/Interpreter/InterpreterNodes.cpp:4677-4790;
// the CPU backend has no kernel for these nodes).  Every row of the fp16 input gets its own
// symmetric int8 parameters from its minimum and maximum (chooseQuantizationParams,
// lib/Quantization/Base/Base.cpp:433-565), is quantized with them (quantization::quantize,
// include/glow/Quantization/Base/Base.h:322-329), multiplied with the int8 weights into int32
// sums, and the result is fp16(float(sum) * (row scale * weight scale[j]) + bias[j]).
//
// Two launches: a warp or a block per input row finds the range, derives the parameters in the
// reference's double arithmetic and writes the int8 row (zero padded to whole 16-byte pieces), its
// scale and (for weights with offsets) its sum; then the contraction runs with its floating-point
// drain.  Weights off that grid, or given as [K, N], are copied first, in a launch of their own.
#include "qgemm.cuh"
#include "quant_math.cuh"

namespace glowb200 {
namespace {

// quantization::quantize<int8_t> (include/glow/Quantization/Base/Base.h:322-329) with an offset already a float.
__device__ __forceinline__ int32_t quantize_i8(float x, float scale, float offset) {
  const float r = __fadd_rn(__fdiv_rn(x, scale), offset);
  long long v = (long long)rintf(r);
  return (int32_t)(v < -128 ? -128 : (v > 127 ? 127 : v));
}

// fp16 bits -> float through the mixed-precision add (adding -0 keeps every value): conversion
// instructions issue at an eighth of the rate.
__device__ __forceinline__ float widen_f16(uint32_t h) {
  float d;
  asm("add.rn.f32.f16 %0, %1, %2;" : "=f"(d) : "h"((uint16_t)(h & 0xFFFFu)), "f"(-0.0f));
  return d;
}

// Eight fp16 numbers from `p` on, positions from `valid` on replaced by `fill`.  VEC: rows are 16-byte
// aligned multiples of 8; else only 4-byte words that hold a wanted number are touched.
template <bool VEC>
__device__ __forceinline__ void load8(const __half *p, int valid, uint32_t fill, uint32_t (&w)[4]) {
  if constexpr (VEC) {
    const uint4 v = valid > 0 ? *reinterpret_cast<const uint4 *>(p) : make_uint4(fill, fill, fill, fill);
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
  } else {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const int odd = (int)(a >> 1) & 1;
    const uint32_t *x = reinterpret_cast<const uint32_t *>(a - 2 * odd);
    uint32_t r[5];
#pragma unroll
    for (int i = 0; i < 5; i++) r[i] = (2 * i - odd < valid && (i < 4 || odd)) ? x[i] : 0u;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      w[i] = __funnelshift_r(r[i], r[i + 1], 16 * odd);
      const int left = valid - 2 * i;
      if (left == 1) w[i] = __byte_perm(w[i], fill, 0x5410);
      else if (left <= 0) w[i] = fill;
    }
  }
}

// in [M, K] fp16 -> q [M, pitch] int8 (zero behind column K), row_scales [M], row_sums [M] (may be
// nullptr).  WPR warps per row: one when the rows fill the SMs, else eight (a row of 4096 is then one
// or two steps of its block instead of sixteen of a warp).  The range is found on the fp16 pairs
// themselves; the second pass reads the row again (from L1 / L2) so that few registers are held and
// many warps stay resident.  Eight elements are quantized by reciprocal at a time; a tie candidate
// among them sends the eight through the exact division.
// CH > 0: rows of at most CH steps, whose numbers stay in registers between the two passes.
template <int WPR, bool VEC, int CH>
__global__ void __launch_bounds__(256) dyn_quantize_rows_kernel(const __half *in, int M, int K, int pitch,
                                                                int8_t *__restrict__ q, float *__restrict__ row_scales,
                                                                int32_t *__restrict__ row_sums, int32_t *status) {
  __shared__ float s_mn[8], s_mx[8];
  __shared__ int32_t s_sum[8];
  pdl_wait();
  pdl_launch_dependents();  // a contraction that follows may set up now (it waits for this kernel before its loads)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = WPR == 1 ? blockIdx.x * 8 + warp : blockIdx.x;
  if (row >= M) return;
  const int first = (WPR == 1 ? lane : (int)threadIdx.x) * 8;
  constexpr int kStep = WPR * 256;
  const __half *x = in + (size_t)row * K;
  // minMaxArg over the row (NaNs never win a comparison; min / max of fp16 numbers is exact)
  const __half2 x00 = __half2half2(x[0]);
  const uint32_t fill = *reinterpret_cast<const uint32_t *>(&x00);
  __half2 mn2 = x00, mx2 = x00;
  uint32_t kept[CH ? CH : 1][4];
  auto range = [&](const uint32_t (&w)[4]) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const __half2 h = *reinterpret_cast<const __half2 *>(&w[i]);
      mn2 = __hmin2(mn2, h);
      mx2 = __hmax2(mx2, h);
    }
  };
  if constexpr (CH > 0) {
#pragma unroll
    for (int c = 0; c < CH; c++) load8<VEC>(x + first + c * kStep, K - first - c * kStep, fill, kept[c]);
#pragma unroll
    for (int c = 0; c < CH; c++) range(kept[c]);
  } else {
#pragma unroll 4
    for (int k = first; k < K; k += kStep) {
      uint32_t w[4];
      load8<VEC>(x + k, K - k, fill, w);
      range(w);
    }
  }
  float mn = fminf(__low2float(mn2), __high2float(mn2)), mx = fmaxf(__low2float(mx2), __high2float(mx2));
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, d));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
  }
  if constexpr (WPR > 1) {
    if (lane == 0) { s_mn[warp] = mn; s_mx[warp] = mx; }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < WPR; i++) {
      mn = fminf(mn, s_mn[i]);
      mx = fmaxf(mx, s_mx[i]);
    }
  }
  // Handle::minMaxArg starts from element 0 and keeps what no later element beats: a NaN there
  // stays (every comparison with it is false), a NaN anywhere else never gets in.  The min / max
  // instructions above drop NaNs wherever they are, so the first element is looked at again.
  {
    const float x0 = __half2float(x[0]);
    if (x0 != x0) mn = mx = x0;
  }
  double scale_d;
  int32_t offset;
  choose_quantization_params_basic(mn, mx, /*Symmetric*/ 1, -128, 127, scale_d, offset);
  const float scale = (float)scale_d, foffset = (float)offset;
  const float rcp = __frcp_rn(scale);
  // A symmetric range always nudges the zero point to 0; the contraction relies on it.
  if (offset != 0 && first == 0 && status != nullptr) atomicOr(status, GLOWB200_STATUS_UNSUPPORTED_TABLE);
  int32_t sum = 0;
  int8_t *o = q + (size_t)row * pitch;
  auto quantize = [&](int k, const uint32_t (&w)[4]) {
    float f[8];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      f[2 * i] = widen_f16(w[i]);
      f[2 * i + 1] = widen_f16(w[i] >> 16);
    }
    int32_t r[8];
    bool exact = offset != 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      // x times the row's reciprocal, rounded to the nearest integer by the 1.5 * 2^23 trick, which
      // leaves the integer in the mantissa; within 1e-4 of a tie (the product is within 3e-5 of
      // the true quotient at |quotient| <= 128), or when not small, the exact division decides
      const float p = __fmul_rn(f[i], rcp);
      const float m = __fadd_rn(p, 12582912.0f);
      const float d = fabsf(__fsub_rn(p, __fsub_rn(m, 12582912.0f)));
      exact |= !(d < 0.4999f) || !(fabsf(p) < 1000.0f);
      const int32_t t = __float_as_int(m) - 0x4B400000;
      r[i] = t < -128 ? -128 : (t > 127 ? 127 : t);
    }
    if (exact) {  // (unrolled: a loop would put f and r into local memory)
#pragma unroll
      for (int i = 0; i < 8; i++) r[i] = quantize_i8(f[i], scale, foffset);
    }
    if (k + 8 > K) {  // the padding
#pragma unroll
      for (int i = 0; i < 8; i++)
        if (k + i >= K) r[i] = 0;
    }
    uint32_t packed[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      sum += r[4 * h] + r[4 * h + 1] + r[4 * h + 2] + r[4 * h + 3];
      packed[h] = (uint32_t)(r[4 * h] & 0xff) | ((uint32_t)(r[4 * h + 1] & 0xff) << 8) | ((uint32_t)(r[4 * h + 2] & 0xff) << 16) |
                  ((uint32_t)(r[4 * h + 3] & 0xff) << 24);
    }
    *reinterpret_cast<uint2 *>(o + k) = make_uint2(packed[0], packed[1]);
  };
  if constexpr (CH > 0) {
#pragma unroll
    for (int c = 0; c < CH; c++)
      if (first + c * kStep < pitch) quantize(first + c * kStep, kept[c]);
  } else {
#pragma unroll 2
    for (int k = first; k < pitch; k += kStep) {
      uint32_t w[4];
      load8<VEC>(x + k, K - k, fill, w);
      quantize(k, w);
    }
  }
  if (row_sums != nullptr) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if constexpr (WPR > 1) {
      if (lane == 0) s_sum[warp] = sum;
      __syncthreads();
      sum = 0;
#pragma unroll
      for (int i = 0; i < WPR; i++) sum += s_sum[i];
    }
    if (first == 0) row_sums[row] = sum;
  }
  if (first == 0) row_scales[row] = scale;
}

template <int WPR, int CH>
cudaError_t launch_quantize_rows(bool vec, const __half *x, int M, int K, int pitch, int8_t *q, float *scales, int32_t *sums,
                                 int32_t *status, cudaStream_t s) {
  const dim3 grid((unsigned)(WPR == 1 ? (M + 7) / 8 : M));
  return vec ? launch_pdl(dyn_quantize_rows_kernel<WPR, true, CH>, grid, 256, 0, s, x, M, K, pitch, q, scales, sums, status)
             : launch_pdl(dyn_quantize_rows_kernel<WPR, false, CH>, grid, 256, 0, s, x, M, K, pitch, q, scales, sums, status);
}

cudaError_t quantize_rows(bool vec, const __half *x, int M, int K, int pitch, int8_t *q, float *scales, int32_t *sums,
                          int32_t *status, cudaStream_t s) {
  if (K <= 256 * 2) return launch_quantize_rows<1, 2>(vec, x, M, K, pitch, q, scales, sums, status, s);
  if (M >= 8 * 2 * kB200Sms) return launch_quantize_rows<1, 0>(vec, x, M, K, pitch, q, scales, sums, status, s);
  if (K <= 8 * 256 * 2) return launch_quantize_rows<8, 2>(vec, x, M, K, pitch, q, scales, sums, status, s);
  return launch_quantize_rows<8, 0>(vec, x, M, K, pitch, q, scales, sums, status, s);
}

int run(void *out, const void *in, const int8_t *weights, const float *bias, const float *scales, const int32_t *offsets,
        float u_scale, int32_t u_offset, int64_t M, int64_t K, int64_t N, const int8_t *weights_transposed, int flags,
        void *workspace, size_t workspace_bytes, int32_t *status, cudaStream_t s) {
  GLOWB200_REQUIRE(M >= 0 && N >= 0 && K > 0 && M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 24),
                   "matrix dimensions out of range");
  if (M == 0 || N == 0) return GLOWB200_OK;
  GLOWB200_REQUIRE(out && in && (weights || weights_transposed) && bias, "NULL tensor pointer");
  const size_t need = glowb200_dynamic_fc_workspace_bytes(M, K, N);
  if (workspace == nullptr || workspace_bytes < need)
    return set_error(GLOWB200_ERR_WORKSPACE_TOO_SMALL, "workspace of %zu bytes given, %zu needed", workspace_bytes, need);
  GLOWB200_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, "workspace must be 256-byte aligned");
  uint8_t *w = reinterpret_cast<uint8_t *>(workspace);
  const int pitch = (int)align_up((size_t)K, 16);
  int8_t *q = reinterpret_cast<int8_t *>(w);
  w += align_up((size_t)M * pitch, 256);
  float *row_scales = reinterpret_cast<float *>(w);
  w += align_up((size_t)M * 4, 256);
  int32_t *row_sums = reinterpret_cast<int32_t *>(w);
  w += align_up((size_t)M * 4, 256);
  const bool offsets_zero = (flags & GLOWB200_FC_WEIGHT_OFFSETS_ZERO) != 0 || (offsets == nullptr && u_offset == 0);
  const bool vec = (K % 8) == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0;
  int32_t *sums = offsets_zero ? nullptr : row_sums;
  const __half *x = reinterpret_cast<const __half *>(in);
  GLOWB200_CUDA_OK(quantize_rows(vec, x, (int)M, (int)K, pitch, q, row_scales, sums, status, s));
  GemmParams p{};
  p.float_out = 1;
  p.out_f16 = reinterpret_cast<__half *>(out);
  p.row_scales = row_scales;
  p.col_scales = scales;
  p.u_col_scale = u_scale;
  p.bias_f32 = bias;
  p.b_offsets = offsets;
  p.u_b_offset = u_offset;
  p.a_row_sums = offsets_zero ? nullptr : row_sums;
  p.status = status;
  p.M = (int)M; p.N = (int)N; p.K = (int)K;
  p.k_corr = (int)K;
  p.a_pitch = pitch;
  const size_t used = (size_t)(w - reinterpret_cast<uint8_t *>(workspace));
  const bool kn = weights_transposed == nullptr || ((flags & GLOWB200_FC_FORCE_ANY_SHAPE_KERNEL) != 0 && weights != nullptr);
  return run_gemm(p, q, kn ? weights : weights_transposed, nullptr, offsets_zero, (flags & GLOWB200_FC_FORCE_ANY_SHAPE_KERNEL) != 0, w,
                  workspace_bytes - used, s, kn);
}

}  // namespace
}  // namespace glowb200

using namespace glowb200;

extern "C" size_t glowb200_dynamic_fc_workspace_bytes(int64_t M, int64_t K, int64_t N) {
  if (M < 0 || N < 0 || K < 0) return 0;
  // quantized input, row scales, row sums, the contraction's own and its copy of the weights
  return align_up((size_t)M * align_up((size_t)K, 16), 256) + 2 * align_up((size_t)M * 4, 256) +
         i8_gemm_core_workspace_bytes(M, N) + i8_gemm_copies_bytes(M, K, N, false, true);
}

extern "C" int glowb200_dynamic_rowwise_quantized_fc(void *out, const void *in, const int8_t *weights, const float *bias,
                                                      const float *scales, const int32_t *offsets, int64_t M, int64_t K,
                                                      int64_t N, const int8_t *weights_transposed, int flags,
                                                      void *workspace, size_t workspace_bytes, int32_t *status,
                                                      glowb200_stream_t stream) {
  GLOWB200_REQUIRE(N == 0 || M == 0 || (scales != nullptr && offsets != nullptr), "scales / offsets is NULL");
  return run(out, in, weights, bias, scales, offsets, 0.0f, 0, M, K, N, weights_transposed, flags, workspace,
             workspace_bytes, status, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int glowb200_dynamic_quantized_fc(void *out, const void *in, const int8_t *weights, const float *bias,
                                              float weights_scale, int32_t weights_offset, int64_t M, int64_t K, int64_t N,
                                              const int8_t *weights_transposed, int flags, void *workspace,
                                              size_t workspace_bytes, int32_t *status, glowb200_stream_t stream) {
  return run(out, in, weights, bias, nullptr, nullptr, weights_scale, weights_offset, M, K, N, weights_transposed, flags,
             workspace, workspace_bytes, status, reinterpret_cast<cudaStream_t>(stream));
}
