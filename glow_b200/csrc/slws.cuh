// What the gather-pool sources (slws.cu, slws_run.cu) share: the description of a launch
// and the small device helpers.
#pragma once
#include "common.cuh"

namespace glowb200 {

struct SlwsLaunch {
  const glowb200_slws_job *jobs;  // device array, or nullptr when `single` is the only job
  glowb200_slws_job single;
  int64_t *seg_begin;  // workspace: per job an int64 [segments + 1] array, then a word: are its lengths skewed?
  int64_t seg_stride;  // int64 elements between the arrays of consecutive jobs
  int64_t max_segments;  // bags a table's array has room for (a descriptor naming more is cut short)
  int32_t *status;
  int32_t in_line, out_line;
  int32_t lpr_log2;
  // 1: the tables are row-range shards (row_begin / global_rows of the descriptors are honoured)
  int32_t sharded;
  // slws_run.cu: element types that need no kernel of their own, and whether the warps add up the
  // lengths before their bags themselves (no boundary array exists then)
  int32_t kind, idx64, out16, inline_lengths;
  int32_t skewed_run;  // bags of a warp of a table with skewed lengths (the word behind its boundaries is not 0)
};

// Bags of a table as the kernels walk them: never more than its boundary array has room for.
__device__ __forceinline__ int64_t bags_of(const SlwsLaunch &p, const glowb200_slws_job *jp) {
  return jp->segments < p.max_segments ? jp->segments : p.max_segments;
}

__device__ __forceinline__ void raise_status(int32_t *status, int32_t bits) {
  if (status != nullptr && bits != 0) atomicOr(status, bits);
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

// Gather-pool with fp32 accumulation for rows of a multiple of 8 columns, any alignment (align: what
// every row of every table starts on -- 8, 4 or 1 bytes).
cudaError_t launch_slws_run(SlwsLaunch L, int align, int64_t max_segments, int64_t num_jobs, cudaStream_t s);

}  // namespace glowb200
