// What the gather-pool sources (slws.cu, slws_run.cu, slws_spread.cu) share: the description of a launch
// and the small device helpers.
#pragma once
#include <climits>

#include "common.cuh"

namespace glowb200 {

struct SlwsLaunch {
  const glowb200_slws_job *jobs;  // device array, or nullptr when `single` is the only job
  glowb200_slws_job single;
  int64_t *seg_begin;  // workspace: per job an int64 [segments + 1] array, then a word: the longest length if they are skewed, else 0
  int64_t seg_stride;  // int64 elements between the arrays of consecutive jobs
  int64_t max_segments;  // bags a table's array has room for (a descriptor naming more is cut short)
  int32_t *status;
  int32_t in_line, out_line;
  int32_t lpr_log2;
  // 1: the tables are row-range shards (row_begin / global_rows of the descriptors are honoured)
  int32_t sharded;
  // slws_run.cu, slws_spread.cu: element types that need no kernel of their own, and whether the warps add up the
  // lengths before their bags themselves (no boundary array exists then)
  int32_t kind, idx64, out16, inline_lengths;
  int32_t skewed_run;   // slws_run.cu: bags of a warp of a table with skewed lengths (the word behind its boundaries is not 0)
  // Two launches that share the tables: slws_run.cu leaves those alone whose word is skip_from or more (0: pools all), and
  // slws_spread.cu, launched behind it, pools those whose word is only_from or more (0: all).
  int32_t skip_from, only_from;
};

// Bags of a table as the kernels walk them: never more than its boundary array has room for.
__device__ __forceinline__ int64_t bags_of(const SlwsLaunch &p, const glowb200_slws_job *jp) {
  return jp->segments < p.max_segments ? jp->segments : p.max_segments;
}

__device__ __forceinline__ void raise_status(int32_t *status, int32_t bits) {
  if (status != nullptr && bits != 0) atomicOr(status, bits);
}

// Loads taken when `row` is not negative; otherwise the result is whatever the register held (such rows
// get the weight 0).  Single volatile instructions: neither a branch round one nor a conversion of its
// value may stand between the loads of a step.
__device__ __forceinline__ uint32_t ldg_if(const void *p, int row) {
  uint32_t v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %2, 0;\n\t@p ld.global.nc.u32 %0, [%1];\n\t}" : "=r"(v) : "l"(p), "r"(row));
  return v;
}
// an index of either width
__device__ __forceinline__ uint2 ldg_index(const void *p, int row, bool wide) {
  uint2 v;
  asm volatile("{\n\t.reg .pred p, q, a, b;\n\tsetp.ge.s32 p, %3, 0;\n\tsetp.ne.u32 q, %4, 0;\n\tand.pred a, p, q;\n\tnot.pred q, q;\n\t"
      "and.pred b, p, q;\n\t@a ld.global.nc.v2.u32 {%0, %1}, [%2];\n\t@b ld.global.nc.u32 %0, [%2];\n\t}"
      : "=r"(v.x), "=r"(v.y) : "l"(p), "r"(row), "r"((uint32_t)wide));
  return v;
}

constexpr unsigned kAllLanes = 0xffffffffu;

// A run of up to 32 consecutive bags of a table, as a warp holds it: lane l has where bag l begins, relative to
// `begin`, and how many rows it has.
constexpr int kMaxRun = 32;
struct SlwsRun {
  int64_t first_bag, begin;  // begin: where in the index array the run begins
  int32_t bags, from, len;
};
// False when the table has no such bags (the whole warp agrees).
__device__ __forceinline__ bool take_run(const SlwsLaunch &p, const glowb200_slws_job *jp, int64_t segments, int64_t first_bag, int most,
                                         int lane, SlwsRun &run, int32_t &flags) {
  if (first_bag >= segments) return false;
  run.first_bag = first_bag;
  run.bags = (int)(first_bag + most < segments ? most : segments - first_bag);
  const int64_t N = jp->num_indices;
  int64_t begin = 0, len = 0;
  if (p.inline_lengths) {
    const int32_t *lengths = jp->lengths;
    const int fb = (int)first_bag;
    int64_t before = 0;  // rows of the bags before the run
    auto add = [&](int32_t v) { before += v > 0 ? v : 0; };
    int i = 0;
    if ((reinterpret_cast<uintptr_t>(lengths) & 15) == 0) {
#pragma unroll 4
      for (int k = lane; k < fb / 4; k += 32) {
        const int4 v = reinterpret_cast<const int4 *>(lengths)[k];
        add(v.x); add(v.y); add(v.z); add(v.w);
      }
      i = fb & ~3;
    }
#pragma unroll 4
    for (i += lane; i < fb; i += 32) add(lengths[i]);
    int32_t own = lane < run.bags ? lengths[fb + lane] : 0;
    if (own < 0) { own = 0; flags |= GLOWB200_STATUS_NEGATIVE_LENGTH; }
    int64_t end = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      before += __shfl_xor_sync(kAllLanes, before, d);
      const int64_t v = __shfl_up_sync(kAllLanes, end, d);
      if (lane >= d) end += v;
    }
    end += before;
    begin = end - own;
    if (end > N) { end = N; flags |= GLOWB200_STATUS_LENGTHS_OVERRUN; }
    if (begin > N) begin = N;
    len = end - begin;
    if (first_bag == 0 && jp->segments > p.max_segments) flags |= GLOWB200_STATUS_BAD_OFFSETS;
  } else if (lane < run.bags) {
    const int64_t *sb = p.seg_begin + (int64_t)blockIdx.y * p.seg_stride + first_bag + lane;
    begin = sb[0];
    len = sb[1] - begin;
    if (len < 0) { len = 0; flags |= GLOWB200_STATUS_BAD_OFFSETS; }
  }
  // Positions are 32-bit, relative to where the run begins.  (Index arrays of 2^31 entries and more are the
  // any-shape kernel's where the host can see them; here a run that long is cut short and reported.)
  run.begin = __shfl_sync(kAllLanes, begin, 0);
  int64_t rel = begin - run.begin;
  if (lane < run.bags && (rel + len > INT32_MAX || rel < INT32_MIN)) { rel = 0; len = 0; flags |= GLOWB200_STATUS_LENGTHS_OVERRUN; }
  run.from = (int32_t)rel;
  run.len = (int32_t)len;
  return true;
}

// The word behind a table's boundaries: the longest of its lengths if that is a step's rows beyond 2.5 times their
// mean, else 0.
__device__ __forceinline__ int64_t skew_word(int32_t longest, int64_t sum, int64_t bags) {
  return 2 * bags * ((int64_t)longest - 16) > 5 * sum ? longest : 0;
}

// The row an index (as ldg_index gives it) names, or -1: out of range, or another shard's.
__device__ __forceinline__ int32_t row_number(const SlwsLaunch &p, const glowb200_slws_job *jp, int32_t rows, uint2 index, bool idx64,
                                              int32_t &flags) {
  if (p.sharded) {
    const int64_t raw = idx64 ? (int64_t)((uint64_t)index.y << 32 | index.x) : (int64_t)(int32_t)index.x, v = raw - jp->row_begin;
    if (v >= 0 && v < rows) return (int32_t)v;
    if (raw < 0 || raw >= jp->global_rows) flags |= GLOWB200_STATUS_INDEX_OUT_OF_RANGE;  // else: another shard's row
    return -1;
  }
  if (index.x < (uint32_t)rows && (!idx64 || index.y == 0)) return (int32_t)index.x;
  flags |= GLOWB200_STATUS_INDEX_OUT_OF_RANGE;
  return -1;
}

__device__ __forceinline__ uint2 ldg2_if(const void *p, int row) {
  uint2 v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %3, 0;\n\t@p ld.global.nc.v2.u32 {%0, %1}, [%2];\n\t}"
      : "=r"(v.x), "=r"(v.y) : "l"(p), "r"(row));
  return v;
}
// four bytes at any address, `valid` of them (none if not positive) inside the row
__device__ __forceinline__ uint32_t ldg_any(const uint8_t *p, int valid, int row) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  const int sh = (int)(a & 3);
  const uint8_t *w = p - sh;
  const uint32_t lo = ldg_if(w, valid > 0 ? row : -1), hi = ldg_if(w + 4, sh != 0 && valid > 4 - sh ? row : -1);
  return __funnelshift_r(lo, hi, 8 * sh);
}

// acc[i] += a * q_i for the 2 * PAIRS columns of a word (a in both halves of a2).
//  * uint8 rows: the byte dropped into the mantissa of 2^23, minus 2^23, is q exactly; sm_100's packed
//    two-lane add and fma (the roundings of the scalar forms, element by element).
//  * 4-bit rows: column 2m is the low nibble of byte m, column 2m+1 the high one
//    (include/glow/Quantization/Base/Base.h:399-406).  The nibbles are spread into bytes 0x8q (three
//    logic ops per word), a byte permute drops each into bits 16..23 of 0x3F80'0000, which
//    reads as m = 1 + q/128, and acc[i] += (128*a) * m.  The surplus sum_j 128*a_j is the same for
//    every column and is taken out once per row through the shared offset sum.  m is exact; the
//    products are about 8-128 times larger than the wanted a*q, which costs at most 7 of the 24
//    mantissa bits -- inside the fp32 tolerance.
template <int BITS, int PAIRS>
__device__ __forceinline__ void pool_word(uint32_t w, uint64_t a2, uint64_t *acc) {
  if constexpr (BITS == 8) {
    uint64_t magic2;
    asm("mov.b64 %0, {%1, %1};" : "=l"(magic2) : "f"(-8388608.0f));
#pragma unroll
    for (int i = 0; i < PAIRS; i++) {
      uint64_t q2;
      asm("mov.b64 %0, {%1, %2};" : "=l"(q2) : "r"(__byte_perm(w, 0x4B000000u, 0x7440 + 2 * i)), "r"(__byte_perm(w, 0x4B000000u, 0x7441 + 2 * i)));
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(q2) : "l"(q2), "l"(magic2));
      asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(acc[i]) : "l"(a2), "l"(q2), "l"(acc[i]));
    }
  } else {
    const uint32_t lo = (w & 0x0F0F0F0Fu) | 0x80808080u, hi = ((w >> 4) & 0x0F0F0F0Fu) | 0x80808080u;
#pragma unroll
    for (int i = 0; i < PAIRS; i++) {
      uint64_t m2;
      asm("mov.b64 %0, {%1, %2};" : "=l"(m2) : "r"(__byte_perm(lo, 0x3F000000u, 0x7044 + (i << 8))), "r"(__byte_perm(hi, 0x3F000000u, 0x7044 + (i << 8))));
      asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(acc[i]) : "l"(a2), "l"(m2), "l"(acc[i]));
    }
  }
}

// Rows: BITS of a column, SO16 (scale and offset are halves), ALIGN (bytes every row starts on: 8, 4, 1 -- where
// scale and offset are floats, 8 makes them one load: 91 bags of 4-bit rows as above 28.2 -> 17.2 us)
template <int BITS, bool SO16, int ALIGN>
struct Rows {
  static constexpr int kBytes = BITS;  // bytes of 8 columns

  __device__ static __forceinline__ uint2 chunk(const uint8_t *at, int valid, int row) {
    if constexpr (BITS == 4) {
      if constexpr (ALIGN >= 4) return make_uint2(ldg_if(at, row), 0u);
      else return make_uint2(ldg_any(at, valid, row), 0u);
    } else {
      if constexpr (ALIGN == 8) return ldg2_if(at, row);
      else if constexpr (ALIGN == 4) return make_uint2(ldg_if(at, row), ldg_if(at + 4, row));
      else return make_uint2(ldg_any(at, valid, row), ldg_any(at + 4, valid - 4, row));
    }
  }
  // raw scale / offset words from the end of the row
  __device__ static __forceinline__ uint2 tail(const uint8_t *end, int row) {
    if constexpr (SO16) {
      if constexpr (ALIGN >= 4) return make_uint2(ldg_if(end - 4, row), 0u);
      else return make_uint2(ldg_any(end - 4, 4, row), 0u);
    } else {
      if constexpr (ALIGN == 8) return ldg2_if(end - 8, row);
      else if constexpr (ALIGN == 4) return make_uint2(ldg_if(end - 8, row), ldg_if(end - 4, row));
      else return make_uint2(ldg_any(end - 8, 8, row), ldg_any(end - 4, 4, row));
    }
  }
  __device__ static __forceinline__ void scale_offset(uint2 t, float &scale, float &offset) {
    if constexpr (SO16) {
      const __half2 h = *reinterpret_cast<const __half2 *>(&t.x);
      scale = __low2float(h);
      offset = __high2float(h);
    } else {
      scale = __uint_as_float(t.x);
      offset = __uint_as_float(t.y);
    }
  }
  // what pool_word wants instead of w * scale is that times kUnit
  static constexpr float kUnit = BITS == 4 ? 128.0f : 1.0f;
  // acc += a * q for the 8 columns of a chunk
  __device__ static __forceinline__ void pool(uint2 c, float a, uint64_t (&acc)[4]) {
    uint64_t a2;
    asm("mov.b64 %0, {%1, %1};" : "=l"(a2) : "f"(a));
    pool_word<BITS, 16 / BITS>(c.x, a2, acc);
    if constexpr (BITS == 8) pool_word<BITS, 2>(c.y, a2, acc + 2);
  }
};

// The sums of a lane's V columns, `valid` of them (a multiple of 8, or of V) inside the row.
template <int V>
__device__ __forceinline__ void store_columns(void *base, int64_t at, const uint64_t *acc, float bias, bool out16, int valid) {
  constexpr int kGroup = V < 8 ? V : 8;
  uint64_t bias2;
  asm("mov.b64 %0, {%1, %1};" : "=l"(bias2) : "f"(bias));
#pragma unroll
  for (int c = 0; c < V; c += kGroup) {
    if (c >= valid) break;
    float o[kGroup];
#pragma unroll
    for (int i = 0; i < kGroup / 2; i++) {
      uint64_t sum;
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(sum) : "l"(acc[c / 2 + i]), "l"(bias2));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(o[2 * i]), "=f"(o[2 * i + 1]) : "l"(sum));
    }
    if (out16) {
      __half *d = reinterpret_cast<__half *>(base) + at + c;
      __half2 h[kGroup / 2];
#pragma unroll
      for (int i = 0; i < kGroup / 2; i++) h[i] = __floats2half2_rn(o[2 * i], o[2 * i + 1]);
      if ((reinterpret_cast<uintptr_t>(d) & (2 * kGroup - 1)) == 0) {
        if constexpr (kGroup == 8) *reinterpret_cast<uint4 *>(d) = *reinterpret_cast<const uint4 *>(h);
        else if constexpr (kGroup == 4) *reinterpret_cast<uint2 *>(d) = *reinterpret_cast<const uint2 *>(h);
        else *reinterpret_cast<__half2 *>(d) = h[0];
      } else {
#pragma unroll
        for (int i = 0; i < kGroup; i++) d[i] = i & 1 ? __high2half(h[i / 2]) : __low2half(h[i / 2]);
      }
    } else {
      float *d = reinterpret_cast<float *>(base) + at + c;
      if ((reinterpret_cast<uintptr_t>(d) & (kGroup == 2 ? 7 : 15)) == 0) {
        if constexpr (kGroup == 2) {
          *reinterpret_cast<float2 *>(d) = make_float2(o[0], o[1]);
        } else {
#pragma unroll
          for (int i = 0; i < kGroup; i += 4) *reinterpret_cast<float4 *>(d + i) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
        }
      } else {
#pragma unroll
        for (int i = 0; i < kGroup; i++) d[i] = o[i];
      }
    }
  }
}

// Lanes of a group and chunks of 8 columns per lane for a row of `chunks` of them: two chunks per lane once
// a row has 8 or more halve the per-row bookkeeping per byte; four when 32 lanes cannot cover the row
// otherwise, and for 4-bit rows of 128 or more columns, where a chunk is only 4 payload bytes and a lane's
// load would otherwise be 8 bytes (measured on the 4-bit sweep: +12 % at 128 columns, +15 % at 256; at 64
// and 32 columns four chunks per lane leave too few lanes per row and lose 20-25 %).
inline int chunks_per_lane(int chunks, bool four_bit) {
  return chunks > 64 || (four_bit && chunks >= 16) ? 4 : (chunks >= 8 ? 2 : 1);
}

// Bags of a table up to which the warps of slws_run.cu add up the lengths before their bags themselves.
constexpr int64_t kInlineLengthsMax = 2048;

// Rows of a warp's run that slws_run.cu counts: while one group walks a bag, four rows to a step, up to seven others
// ask for one at every step, and how often they asked is a 32-bit number.  (A minimum on that count instead cost the
// 256 even tables 12 % and the recommendation model's pooling 30 %: the registers.)
constexpr int64_t kMostRows = INT32_MAX / 7 * 4ll;

// Gather-pool with fp32 accumulation for rows of a multiple of 8 columns, any alignment (align: what
// every row of every table starts on -- 8, 4 or 1 bytes), or any that slws_stream_takes: chooses between the three
// kernels (slws_spread.cu) by the bags and, where the caller knows them, the rows of the launch (kRowsUnknown: it does not).
constexpr int64_t kRowsUnknown = -1;
cudaError_t launch_slws(SlwsLaunch L, int align, int64_t max_segments, int64_t num_jobs, int64_t rows, cudaStream_t s);
// slws_stream.cu: whether it can pool a launch's rows at all, and the launch.
bool slws_stream_takes(const SlwsLaunch &L, int align);
cudaError_t launch_slws_stream(const SlwsLaunch &L, int align, int64_t max_segments, int64_t num_jobs, cudaStream_t s);
cudaError_t launch_slws_run(SlwsLaunch L, int align, int64_t max_segments, int64_t num_jobs, cudaStream_t s);

}  // namespace glowb200
