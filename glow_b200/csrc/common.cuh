// Shared host/device helpers of the glow_b200 kernels.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>

#include "glow_b200.h"

namespace glowb200 {

// Thread-local message behind glowb200_last_error().
char *last_error_buffer();
int set_error(int code, const char *fmt, ...);

#define GLOWB200_CUDA_OK(expr)                                                                  \
  do {                                                                                          \
    cudaError_t e__ = (expr);                                                                   \
    if (e__ != cudaSuccess)                                                                     \
      return ::glowb200::set_error(GLOWB200_ERR_CUDA, "%s failed: %s", #expr,                   \
                                   cudaGetErrorString(e__));                                    \
  } while (0)

#define GLOWB200_REQUIRE(cond, ...)                                                             \
  do {                                                                                          \
    if (!(cond)) return ::glowb200::set_error(GLOWB200_ERR_INVALID_ARGUMENT, __VA_ARGS__);      \
  } while (0)

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Number of SMs of the current device (cached per device; asking for the device takes some 0.1 us).
int sm_count();
// ... and of a B200, for rules that need not know the device: a few-row product is 3 us in all.
constexpr int kB200Sms = 148;

// Bag boundaries of one lengths array (defined beside the gather-pool kernels):
// seg_begin[i] = min(sum(max(lengths[0..i), 0)), num_indices) for i in [0, segments]; the array
// must hold glowb200_slws_workspace_bytes(segments, 1) bytes.  Raises the status bits of
// negative lengths and of lengths that overrun num_indices.
int launch_segments_from_lengths(const int32_t *lengths, int64_t segments, int64_t num_indices,
                                 void *workspace, size_t workspace_bytes, int32_t *status,
                                 cudaStream_t stream);

// ---- integer requantisation (device side) ----------------------------------------------
// libjit_scale<int32,int32> (lib/LLVMIRCodeGen/libjit/libjit_defs.h:158-173): arithmetic
// shifts, 32-bit wrapping multiply/add, rounding term only when post > 0, offset added last.
__host__ __device__ __forceinline__ int32_t scale32(int32_t input, int32_t pre, int32_t post,
                                                    int32_t scale, int32_t offset) {
  const uint32_t rtn = (post > 0) ? (1u << (post - 1)) : 0u;
  const int32_t a = input >> pre;
  const int32_t c = (int32_t)((uint32_t)a * (uint32_t)scale + rtn);
  return (int32_t)((uint32_t)(c >> post) + (uint32_t)offset);
}

// The quantized Add of two int8 values (scale32 of either side, the result's offset, clip, optionally max with
// a constant) for parameters of the ordinary kind: no shift before the multiplication, a scale of 16 bits, and
// nothing in 32-bit overflow.  A side then is one dot-product instruction -- byte * scale + constant, the byte
// picked from its word -- and a shift, and the result's offset rides on the left constant: 3.5 ALU and 2
// multiplier instructions per element where the formula as written took 10.8 and 4.9.
struct AddQuant {
  int32_t l_scale, l_const, l_post, r_scale, r_const, r_post, floor;
};
inline bool make_add_quant(AddQuant &q, int32_t dest_off, int32_t l_off, int32_t r_off, int32_t l_pre, int32_t l_post,
                           int32_t l_scale, int32_t r_pre, int32_t r_post, int32_t r_scale, int32_t splat) {
  auto off_ok = [](int32_t o) { return o >= -512 && o <= 512; };
  auto side_ok = [](int32_t pre, int32_t post, int32_t scale) {
    return pre == 0 && post >= 0 && post <= 20 && scale >= 0 && scale < (1 << 15);
  };
  if (!off_ok(dest_off) || !off_ok(l_off) || !off_ok(r_off) || !side_ok(l_pre, l_post, l_scale) || !side_ok(r_pre, r_post, r_scale))
    return false;
  // |byte * scale + constant| < 2^22 + 2^19 + 2^24 + 2^29
  q = {l_scale, ((1 << l_post) >> 1) - l_off * l_scale + dest_off * (1 << l_post), l_post,
       r_scale, ((1 << r_post) >> 1) - r_off * r_scale, r_post, splat};
  return true;
}
#ifdef __CUDACC__
// four elements: the bytes of two words (FLOOR false: saturation alone reaches q.floor)
template <bool FLOOR = true>
__device__ __forceinline__ uint32_t add_quant_word(uint32_t l, uint32_t r, const AddQuant &q) {
  auto one = [&](int32_t a, int32_t b) {
    if constexpr (FLOOR) return __viaddmax_s32(a >> q.l_post, b >> q.r_post, q.floor);
    else return (a >> q.l_post) + (b >> q.r_post);
  };
  const int lh = q.l_scale << 16, rh = q.r_scale << 16;
  const int32_t e0 = one(__dp2a_lo(q.l_scale, (int)l, q.l_const), __dp2a_lo(q.r_scale, (int)r, q.r_const));
  const int32_t e1 = one(__dp2a_lo(lh, (int)l, q.l_const), __dp2a_lo(rh, (int)r, q.r_const));
  const int32_t e2 = one(__dp2a_hi(q.l_scale, (int)l, q.l_const), __dp2a_hi(q.r_scale, (int)r, q.r_const));
  const int32_t e3 = one(__dp2a_hi(lh, (int)l, q.l_const), __dp2a_hi(rh, (int)r, q.r_const));
  uint32_t w;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(e3), "r"(e2), "r"(0));
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(e1), "r"(e0), "r"(w));
  return w;
}
#endif

#ifdef __CUDACC__
// x / d for 0 <= x < 2^31 with reciprocal = floor((2^32 - 1) / d): the estimate is the quotient or one less.
__device__ __forceinline__ int fast_div(int x, int d, uint32_t reciprocal) {
  const int q = (int)__umulhi((uint32_t)x, reciprocal);
  return q + (x - q * d >= d ? 1 : 0);
}
// nearbyintf(x / scale + offset) as an integer, by the reciprocal of the scale.  Where neither the sum nor the offset is beyond
// +- 2000, the quotient is below 4000: three roundings of a relative 2^-24 (of the reciprocal, the product and the division; 7.2e-4) and
// those of both sums (1.2e-4) stay below 1e-3.  Next to a tie, and beyond, `sure` becomes false and the division has to decide (what
// rounds beyond int8 is clipped then).  limit: reciprocal_limit(offset), beyond which no sum is sure.
__host__ __device__ inline float reciprocal_limit(int32_t offset) { return offset >= -2000 && offset <= 2000 ? 2000.0f : 0.0f; }
__device__ __forceinline__ int32_t quantize_by_reciprocal(float x, float inverse, float offset, float limit, bool &sure) {
  constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: its sum with u has rint(u) in the low bits
  const float u = __fadd_rn(__fmul_rn(x, inverse), offset), m = __fadd_rn(u, kMagic);
  sure = sure && fabsf(u) < limit && fabsf(__fadd_rn(u, -__fadd_rn(m, -kMagic))) < 0.499f;
  return __float_as_int(m) - __float_as_int(kMagic);
}
// Walks x down a mixed radix: returns x % d and leaves x / d.
struct Divisor {
  int d;
  uint32_t reciprocal;
  __host__ __device__ explicit Divisor(int d) : d(d), reciprocal(d > 0 ? 0xffffffffu / (uint32_t)d : 0u) {}
  __device__ __forceinline__ int rest(int &x) const {
    const int q = fast_div(x, d, reciprocal), r = x - q * d;
    x = q;
    return r;
  }
};
#endif

// libjit_clip_i8 (libjit_defs.h:146-148).
__host__ __device__ __forceinline__ int32_t clip_i8(int32_t v) {
  return v < -128 ? -128 : (v > 127 ? 127 : v);
}

// Programmatic dependent launch: a kernel launched with the programmatic-serialization attribute may
// start (set up its barriers, tensor memory, shared memory) while the kernel before it in the stream
// is still running, once every block of that kernel has passed pdl_launch_dependents(); it must not
// touch global memory before pdl_wait(), which returns when the earlier kernel has completed and its
// writes are visible.  Both are no-ops in a kernel launched the ordinary way.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Programmatic launches are on unless the environment says GLOWB200_PDL=0 (read once).  A waiting
// kernel holds its shared memory and thread slots, which costs a kernel that runs beside it on
// another stream: a caller that overlaps streams can switch them off.
bool pdl_enabled();
// Launches `kernel` so that it may start beside the tail of the kernel before it (see pdl_wait()).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, unsigned block, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace glowb200
