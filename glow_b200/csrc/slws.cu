// Embedding gather-pool kernels for fused-rowwise quantized tables on sm_100a:
// FusedRowwiseQuantizedSparseLengthsWeightedSum (uint8 and 4-bit rows, fp32 or fp16
// scale/offset, fp32 or fp16 result) and EmbeddingBagByteRowwiseOffsets.
//
// Launches:
//   * a "segments" kernel turns lengths (or offsets) into validated bag boundaries in the caller's
//     workspace, one int64 array per table (tables of up to 2048 bags pooled with fp32 accumulation need none:
//     their warps add up the lengths before their bags themselves);
//   * fp32 accumulation over rows of a multiple of 8 columns is slws_run.cu's, in launches where the longest
//     bag decides slws_spread.cu's and in those that fill the GPU with rows that suit it slws_stream.cu's;
//   * fp16 accumulation, which the reference rounds at every step, is done exactly that way, step by
//     step, by slws_gather_kernel below: a group of `lpr` lanes (a power of two, 1..32) per bag, each
//     lane with P chunks of 8 columns, indices read coalesced and handed round by shuffles, kUnroll rows
//     requested before the first is consumed;
//   * any other row width takes slws_gather_any_kernel: the reference's operations in its order.
#include "slws.cuh"

#include <climits>
#include <mutex>

namespace glowb200 {
namespace {

constexpr int kGatherThreads = 64;  // small blocks: a block's SM slots stay taken until its slowest warp is done
constexpr int kSegThreads = 1024;

__device__ __forceinline__ uint32_t ldg_stream_u32(const void *p) {
  uint32_t v;
  asm("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// ------------------------------------------------------------------------------------------
// Bag boundaries.  One block per table.
//   lengths form : seg_begin[i] = min(sum(max(lengths[0..i), 0)), num_indices)
//   offsets form : seg_begin[i] = clamp(offsets[i], 0, num_indices); the closing entry is
//                  offsets[segments] when an end offset is present, else num_indices
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ int64_t block_exclusive_scan(int64_t v, int64_t *warp_tot, int64_t &block_total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    int64_t t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += t;
  }
  if (lane == 31) warp_tot[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int64_t w = (lane < (int)(blockDim.x >> 5)) ? warp_tot[lane] : 0;
    int64_t winc = w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      int64_t t = __shfl_up_sync(0xffffffffu, winc, d);
      if (lane >= d) winc += t;
    }
    warp_tot[lane] = winc - w;  // exclusive prefix of warp totals
    if (lane == 31) warp_tot[32] = winc;
  }
  __syncthreads();
  const int64_t res = warp_tot[warp] + inc - v;
  block_total = warp_tot[32];
  __syncthreads();
  return res;
}

__global__ void __launch_bounds__(kSegThreads) slws_segments_from_lengths_kernel(const __grid_constant__ SlwsLaunch p) {
  pdl_wait();               // the gather before this one may still read the boundaries this kernel rewrites
  pdl_launch_dependents();  // this launch's gather may take its place on the SMs (it waits before reading them)
  __shared__ int64_t warp_tot[33];
  __shared__ int longest;
  if (threadIdx.x == 0) longest = 0;
  int32_t my_longest = 0;
  const glowb200_slws_job job = p.jobs ? p.jobs[blockIdx.x] : p.single;
  int64_t *out = p.seg_begin + (int64_t)blockIdx.x * p.seg_stride;
  int32_t flags = 0;
  int64_t S = job.segments;
  if (S > p.max_segments) { S = p.max_segments; flags |= GLOWB200_STATUS_BAD_OFFSETS; }
  const int64_t N = job.num_indices;
  constexpr int kItems = 4;
  int64_t carry = 0;
  for (int64_t tile = 0; tile < S; tile += (int64_t)kSegThreads * kItems) {
    const int64_t first = tile + (int64_t)threadIdx.x * kItems;
    int64_t v[kItems], sum = 0;
#pragma unroll
    for (int i = 0; i < kItems; i++) {
      int64_t l = (first + i < S) ? (int64_t)job.lengths[first + i] : 0;
      if (l < 0) { l = 0; flags |= GLOWB200_STATUS_NEGATIVE_LENGTH; }
      v[i] = l;
      sum += l;
      my_longest = max(my_longest, (int32_t)l);
    }
    int64_t tile_total;
    int64_t run = carry + block_exclusive_scan(sum, warp_tot, tile_total);
#pragma unroll
    for (int i = 0; i < kItems; i++) {
      if (first + i < S) out[first + i] = run < N ? run : N;
      run += v[i];
    }
    carry += tile_total;
  }
  my_longest = __reduce_max_sync(0xffffffffu, my_longest);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) atomicMax(&longest, my_longest);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (carry > N) flags |= GLOWB200_STATUS_LENGTHS_OVERRUN;
    out[S] = carry < N ? carry : N;
    out[S + 1] = skew_word(longest, carry, S);
  }
  raise_status(p.status, flags);
}

template <typename IdxT>
__global__ void __launch_bounds__(256) slws_segments_from_offsets_kernel(const __grid_constant__ SlwsLaunch p,
                                                                           const IdxT *offsets, int has_end) {
  const int64_t S = p.single.segments, N = p.single.num_indices;
  int32_t flags = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= S; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t v = (i < S || has_end) ? (int64_t)offsets[i] : N;
    if (v < 0) { v = 0; flags |= GLOWB200_STATUS_BAD_OFFSETS; }
    if (v > N) { v = N; flags |= GLOWB200_STATUS_BAD_OFFSETS; }
    p.seg_begin[i] = v;
  }
  raise_status(p.status, flags);
  if (blockIdx.x != 0) return;
  // Whether the lengths are skewed, from up to kSampled bags spread over the table: the word decides only which
  // kernel pools the table, and in runs of how many bags.
  constexpr int64_t kSampled = 2048;
  __shared__ int longest;
  if (threadIdx.x == 0) longest = 0;
  __syncthreads();
  auto at = [&](int64_t i) {
    const int64_t v = (i < S || has_end) ? (int64_t)offsets[i] : N;
    return v < 0 ? 0 : v > N ? N : v;
  };
  const int64_t sampled = S < kSampled ? S : kSampled;
  int64_t mine = 0;
  for (int64_t k = threadIdx.x; k < sampled; k += blockDim.x) {
    const int64_t i = k * S / sampled, len = at(i + 1) - at(i);
    mine = mine > len ? mine : len;
  }
  const int most = __reduce_max_sync(0xffffffffu, (int)(mine < INT32_MAX ? mine : INT32_MAX));
  if ((threadIdx.x & 31) == 0) atomicMax(&longest, most);
  __syncthreads();
  if (threadIdx.x == 0) p.seg_begin[S + 1] = skew_word(longest, at(S) > at(0) ? at(S) - at(0) : 0, S);
}

// ------------------------------------------------------------------------------------------
// Gather-pool with fp16 accumulation (tables with fp16 scale / offset, fp16 weights and result).
// AccumT = float16 (InterpreterNodes.cpp:5799,5832; Float16.h:38-56): the addend d*w is rounded to fp32
// then to fp16, the fp16 sum is widened, added and rounded, row after row.
// grid = (ceil(max_segments / bags_per_block), num_jobs).
// ------------------------------------------------------------------------------------------
struct Chunk { uint32_t lo, hi; };  // 8 columns of a row

template <int BITS>
__device__ __forceinline__ Chunk load_chunk(const uint8_t *row, int chunk) {  // rows are 4-byte aligned
  if constexpr (BITS == 4) return {ldg_stream_u32(row + chunk * 4), 0u};
  else return {ldg_stream_u32(row + chunk * 8), ldg_stream_u32(row + chunk * 8 + 4)};
}

// Column i (0..7) of a chunk as an exact float: the byte / nibble is dropped into the
// mantissa of 2^23 and 2^23 is subtracted.  4-bit rows keep column 2m in the low nibble of
// byte m and column 2m+1 in the high nibble (include/glow/Quantization/Base/Base.h:399-406).
template <int BITS>
__device__ __forceinline__ float column(const Chunk &c, int i) {
  uint32_t m;
  if constexpr (BITS == 8) m = __byte_perm(i < 4 ? c.lo : c.hi, 0x4B000000u, 0x7440 + (i & 3));  // {byte i, 0, 0, 0x4B}
  else m = ((c.lo >> (4 * i)) & 0xFu) | 0x4B000000u;
  return __uint_as_float(m) - 8388608.0f;
}

template <int BITS, typename IdxT, int P>
__global__ void __launch_bounds__(kGatherThreads, P == 4 ? 8 : 12) slws_gather_kernel(const __grid_constant__ SlwsLaunch p) {
  constexpr int kUnroll = 4;
  const int job_id = blockIdx.y;
  const glowb200_slws_job *jp = p.jobs ? (p.jobs + job_id) : &p.single;
  const int64_t segments = bags_of(p, jp);
  const int lpr = 1 << p.lpr_log2;
  const int gl = threadIdx.x & (lpr - 1);
  const int64_t bag = (int64_t)blockIdx.x * (kGatherThreads >> p.lpr_log2) + (threadIdx.x >> p.lpr_log2);
  if (bag >= segments) return;  // whole groups leave together

  const uint8_t *data = reinterpret_cast<const uint8_t *>(jp->data);
  const IdxT *indices = reinterpret_cast<const IdxT *>(jp->indices);
  const __half *weights = reinterpret_cast<const __half *>(jp->weights);
  const int64_t rows = jp->rows;
  const int64_t *sb = p.seg_begin + (int64_t)job_id * p.seg_stride;
  const int64_t in_line = p.in_line;
  const int chunks = p.out_line >> 3;

  const unsigned lane = threadIdx.x & 31u;
  const unsigned gmask = (lpr == 32) ? 0xffffffffu : (((1u << lpr) - 1u) << (lane & ~(unsigned)(lpr - 1)));

  int64_t begin = sb[bag], end = sb[bag + 1];
  int32_t flags = 0;
  if (end < begin) { end = begin; flags |= GLOWB200_STATUS_BAD_OFFSETS; }

  bool has[P];
  float acc[P][8];
#pragma unroll
  for (int c = 0; c < P; c++) {
    has[c] = (c * lpr + gl) < chunks;
#pragma unroll
    for (int i = 0; i < 8; i++) acc[c][i] = 0.0f;
  }

  // Row numbers travel as int32 inside the group (-1 = skip): tables have fewer than 2^31 rows
  // (checked on the host).  The next `lpr` indices are requested before the current ones are
  // consumed, and looked at (range check, narrowing) only after the rows of the chunk before are on
  // their way, or the warp would sit out the index latency first and the row latency after it.
  auto request = [&](int64_t pos, IdxT &v, float &w) {
    v = 0;
    w = 0.0f;
    if (pos < end) {
      v = indices[pos];
      w = __half2float(weights[pos]);
    }
  };
  auto resolve = [&](int64_t pos, IdxT raw) -> int32_t {
    if (pos >= end) return -1;
    const int64_t v = (int64_t)raw;
    if (v >= 0 && v < rows) return (int32_t)v;
    flags |= GLOWB200_STATUS_INDEX_OUT_OF_RANGE;
    return -1;
  };
  int32_t r_mine;
  IdxT v_next;
  float w_mine, w_next;
  request(begin + gl, v_next, w_mine);
  r_mine = resolve(begin + gl, v_next);
  for (int64_t base = begin; base < end; base += lpr) {
    request(base + lpr + gl, v_next, w_next);
    const int n = (int)((end - base) < (int64_t)lpr ? (end - base) : (int64_t)lpr);
    for (int t = 0; t < n; t += kUnroll) {
      int32_t r[kUnroll];
      float w[kUnroll];
      Chunk pay[kUnroll][P];
      uint32_t tl[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; u++) {
        r[u] = __shfl_sync(gmask, r_mine, t + u, lpr);
        w[u] = __shfl_sync(gmask, w_mine, t + u, lpr);
        if (t + u >= n) r[u] = -1;
      }
#pragma unroll
      for (int u = 0; u < kUnroll; u++) {
        if (r[u] >= 0) {
          const uint8_t *row = data + (int64_t)r[u] * in_line;
#pragma unroll
          for (int c = 0; c < P; c++)
            if (has[c]) pay[u][c] = load_chunk<BITS>(row, c * lpr + gl);
          tl[u] = ldg_stream_u32(row + in_line - 4);
        }
      }
#pragma unroll
      for (int u = 0; u < kUnroll; u++) {
        if (r[u] >= 0) {
          const __half2 h = *reinterpret_cast<const __half2 *>(&tl[u]);
          const float scale = __low2float(h), offset = __high2float(h);
          // q*scale is exact in fp32 for an fp16 scale, so the FMA equals multiply-then-add
#pragma unroll
          for (int c = 0; c < P; c++)
            if (has[c]) {
#pragma unroll
              for (int i = 0; i < 8; i++) {
                const float d = __fmaf_rn(column<BITS>(pay[u][c], i), scale, offset);
                const float addend = __half2float(__float2half_rn(__fmul_rn(d, w[u])));
                acc[c][i] = __half2float(__float2half_rn(__fadd_rn(acc[c][i], addend)));
              }
            }
        }
      }
    }
    r_mine = resolve(base + lpr + gl, v_next);
    w_mine = w_next;
  }

  // Every bag writes its row, empty bags write zeros (the reference zero-fills dest first).
  const int64_t dest_stride = jp->dest_stride;
  void *dest_base = jp->dest;
  int64_t dest_row = bag;
  if (jp->bags_per_dest > 0) {  // scatter over several (possibly remote) destination buffers
    const int64_t which = bag / jp->bags_per_dest;
    dest_base = jp->dests[which];
    dest_row = bag - which * jp->bags_per_dest;
  }
#pragma unroll
  for (int c = 0; c < P; c++) {
    if (!has[c]) continue;
    __half *d = reinterpret_cast<__half *>(dest_base) + dest_row * dest_stride + (int64_t)(c * lpr + gl) * 8;
    __half2 h[4];
#pragma unroll
    for (int i = 0; i < 4; i++) h[i] = __floats2half2_rn(acc[c][2 * i], acc[c][2 * i + 1]);
    if ((reinterpret_cast<uintptr_t>(d) & 15u) == 0) {
      *reinterpret_cast<uint4 *>(d) = *reinterpret_cast<const uint4 *>(h);
    } else {  // a result may start at any element
#pragma unroll
      for (int i = 0; i < 8; i++) d[i] = i & 1 ? __high2half(h[i / 2]) : __low2half(h[i / 2]);
    }
  }
  raise_status(p.status, flags);
}

// ------------------------------------------------------------------------------------------
// Any-shape gather-pool: rows of any width and alignment (a column count that is not a
// multiple of 8 -- uint8 rows of a multiple of 4 go to slws_stream.cu, which has these operations as well --, a
// table that is not 8-byte aligned).  One warp per bag, byte loads, column
// tiles of 128; the row-by-row arithmetic of the reference in its order, without FMA
// contraction.  Correct for everything, fast for nothing -- real tables take the kernel above.
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) slws_gather_any_kernel(const __grid_constant__ SlwsLaunch p, int bits,
                                                               int so16, int out16, int acc16, int idx64) {
  const int job_id = blockIdx.y;
  const glowb200_slws_job *jp = p.jobs ? (p.jobs + job_id) : &p.single;
  const int64_t bag = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (bag >= bags_of(p, jp)) return;
  const int lane = threadIdx.x & 31;
  const uint8_t *data = reinterpret_cast<const uint8_t *>(jp->data);
  const int64_t *sb = p.seg_begin + (int64_t)job_id * p.seg_stride;
  int64_t begin = sb[bag], end = sb[bag + 1];
  int32_t flags = 0;
  if (end < begin) { end = begin; flags |= GLOWB200_STATUS_BAD_OFFSETS; }
  const int64_t in_line = p.in_line;
  const int D = p.out_line;
  for (int tile = 0; tile < D; tile += 128) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int64_t j = begin; j < end; j++) {
      int64_t r = idx64 ? reinterpret_cast<const int64_t *>(jp->indices)[j]
                        : (int64_t) reinterpret_cast<const int32_t *>(jp->indices)[j];
      const int64_t g = r;
      if (p.sharded) r -= jp->row_begin;
      if (r < 0 || r >= jp->rows) {
        if (!p.sharded || g < 0 || g >= jp->global_rows) flags |= GLOWB200_STATUS_INDEX_OUT_OF_RANGE;
        continue;
      }
      const float w = out16 ? __half2float(reinterpret_cast<const __half *>(jp->weights)[j])
                            : reinterpret_cast<const float *>(jp->weights)[j];
      const uint8_t *row = data + r * in_line;
      float scale, offset;
      if (so16) {
        const uint8_t *t = row + in_line - 4;
        scale = __half2float(__ushort_as_half((unsigned short)(t[0] | (t[1] << 8))));
        offset = __half2float(__ushort_as_half((unsigned short)(t[2] | (t[3] << 8))));
      } else {
        const uint8_t *t = row + in_line - 8;
        scale = __uint_as_float(t[0] | (t[1] << 8) | (t[2] << 16) | ((uint32_t)t[3] << 24));
        offset = __uint_as_float(t[4] | (t[5] << 8) | (t[6] << 16) | ((uint32_t)t[7] << 24));
      }
#pragma unroll
      for (int s = 0; s < 4; s++) {
        const int k = tile + s * 32 + lane;
        if (k < D) {
          uint32_t q;
          if (bits == 8) q = row[k];
          else { q = row[k >> 1]; q = (k & 1) ? (q >> 4) : (q & 0xFu); }
          const float d = __fadd_rn(__fmul_rn((float)q, scale), offset);
          const float prod = __fmul_rn(d, w);
          if (acc16) acc[s] = __half2float(__float2half_rn(__fadd_rn(acc[s], __half2float(__float2half_rn(prod)))));
          else acc[s] = __fadd_rn(acc[s], prod);
        }
      }
    }
#pragma unroll
    for (int s = 0; s < 4; s++) {
      const int k = tile + s * 32 + lane;
      if (k < D) {
        void *dest_base = jp->dest;
        int64_t dest_row = bag;
        if (jp->bags_per_dest > 0) {
          const int64_t which = bag / jp->bags_per_dest;
          dest_base = jp->dests[which];
          dest_row = bag - which * jp->bags_per_dest;
        }
        if (out16) reinterpret_cast<__half *>(dest_base)[dest_row * jp->dest_stride + k] = __float2half_rn(acc[s]);
        else reinterpret_cast<float *>(dest_base)[dest_row * jp->dest_stride + k] = acc[s];
      }
    }
  }
  raise_status(p.status, flags);
}

// ------------------------------------------------------------------------------------------
// Host dispatch
// ------------------------------------------------------------------------------------------
struct GatherConfig {
  int kind, idx64, out16, acc16;
};
enum class Form { kAnyShape, kRuns, kFp16Steps };  // the any-shape kernel, slws_run.cu / slws_spread.cu / slws_stream.cu, slws_gather_kernel

template <int BITS, typename IdxT>
cudaError_t launch_fp16_steps(SlwsLaunch L, int64_t max_segments, int64_t num_jobs, cudaStream_t s) {
  const int chunks = L.out_line / 8, P = chunks_per_lane(chunks, BITS == 4);
  L.lpr_log2 = 0;
  while ((P << L.lpr_log2) < chunks) L.lpr_log2++;
  const int bags_per_block = kGatherThreads >> L.lpr_log2;
  const dim3 grid((unsigned)((max_segments + bags_per_block - 1) / bags_per_block), (unsigned)num_jobs);
  if (P == 1) slws_gather_kernel<BITS, IdxT, 1><<<grid, kGatherThreads, 0, s>>>(L);
  else if (P == 2) slws_gather_kernel<BITS, IdxT, 2><<<grid, kGatherThreads, 0, s>>>(L);
  else slws_gather_kernel<BITS, IdxT, 4><<<grid, kGatherThreads, 0, s>>>(L);
  return cudaGetLastError();
}

int payload_bytes(int kind, int64_t out_line) { return (int)(kind >= 2 ? out_line / 2 : out_line); }
int tail_bytes(int kind) { return (kind & 1) ? 4 : 8; }

// Validates the shape arguments shared by every entry point and picks the kernel.  align: what the
// tables start on (a power of two); it becomes what every row starts on.
int plan(const GatherConfig &g, int64_t in_line, int64_t out_line, bool operands_fit, int &align, Form &form) {
  const int kind = g.kind;
  GLOWB200_REQUIRE(kind >= 0 && kind <= 3, "unknown fused table kind %d", kind);
  GLOWB200_REQUIRE(out_line >= 0 && in_line > 0 && in_line < (1 << 30), "bad line sizes");
  GLOWB200_REQUIRE(kind < 2 || (out_line % 2) == 0, "4-bit rows need an even column count");
  // Rows may be wider than payload + scale/offset: the columns come first, the scale/offset
  // pair is the LAST bytes of the row (where the reference kernel looks for it,
  // libjit.cpp:1263-1264), and whatever lies between is padding -- a table stored with its rows
  // padded to a memory-friendly stride is pooled as it is.
  GLOWB200_REQUIRE(in_line >= payload_bytes(kind, out_line) + tail_bytes(kind),
                   "in_line_size %lld is too small for %lld columns of kind %d", (long long)in_line,
                   (long long)out_line, kind);
  align = (int)((align | in_line) & -(align | in_line));
  align = align >= 8 ? 8 : align >= 4 ? 4 : 1;
  form = Form::kAnyShape;
  // (the any-shape kernel takes 4.5 times as long for 100 columns as any other for 104; both give the reference's bits)
  if (out_line % 8 == 4 && out_line > 36 && operands_fit && !g.acc16 && kind < 2) {
    SlwsLaunch L{};
    L.kind = kind;
    L.in_line = (int32_t)in_line;
    L.out_line = (int32_t)out_line;
    L.single.data = reinterpret_cast<const void *>((uintptr_t)align);  // (as far as where rows start goes)
    if (slws_stream_takes(L, align)) form = Form::kRuns;
    return GLOWB200_OK;
  }
  // (above 1024 columns, and for other widths, the any-shape kernel's operation order stays)
  if (out_line == 0 || out_line % 8 != 0 || out_line > 1024 || !operands_fit) return GLOWB200_OK;
  if (!g.acc16) form = Form::kRuns;
  else if (align >= 4) form = Form::kFp16Steps;
  return GLOWB200_OK;
}

int run_gather(const SlwsLaunch &L, const GatherConfig &g, Form form, int align, int64_t max_segments, int64_t num_jobs, int64_t rows,
               cudaStream_t s) {
  if (max_segments == 0 || num_jobs == 0) return GLOWB200_OK;
  cudaError_t e;
  if (form == Form::kRuns) {
    e = launch_slws(L, align, max_segments, num_jobs, rows, s);
  } else if (form == Form::kFp16Steps) {
    if (g.kind >= 2)
      e = g.idx64 ? launch_fp16_steps<4, int64_t>(L, max_segments, num_jobs, s) : launch_fp16_steps<4, int32_t>(L, max_segments, num_jobs, s);
    else
      e = g.idx64 ? launch_fp16_steps<8, int64_t>(L, max_segments, num_jobs, s) : launch_fp16_steps<8, int32_t>(L, max_segments, num_jobs, s);
  } else {
    dim3 grid((unsigned)((max_segments + 7) / 8), (unsigned)num_jobs);
    slws_gather_any_kernel<<<grid, 256, 0, s>>>(L, g.kind >= 2 ? 4 : 8, g.kind & 1, g.out16, g.acc16, g.idx64);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return set_error(GLOWB200_ERR_CUDA, "gather-pool launch failed: %s", cudaGetErrorString(e));
  return GLOWB200_OK;
}

void set_types(SlwsLaunch &L, const GatherConfig &g) {
  L.kind = g.kind;
  L.idx64 = g.idx64;
  L.out16 = g.out16;
}

// The boundaries of every table of a launch from its lengths -- unless the gather's warps work them out.
cudaError_t segments_from_lengths(SlwsLaunch &L, Form form, int64_t max_segments, int64_t num_jobs, cudaStream_t s) {
  if (form == Form::kRuns && max_segments <= kInlineLengthsMax) {
    L.inline_lengths = 1;
    return cudaSuccess;
  }
  return launch_pdl(slws_segments_from_lengths_kernel, dim3((unsigned)num_jobs), kSegThreads, 0, s, L);
}

size_t seg_stride_elems(int64_t max_segments) { return align_up((size_t)(max_segments + 2) * 8, 256) / 8; }

bool aligned_to(const void *p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

}  // namespace
}  // namespace glowb200

int glowb200::launch_segments_from_lengths(const int32_t *lengths, int64_t segments, int64_t num_indices,
                                           void *workspace, size_t workspace_bytes, int32_t *status,
                                           cudaStream_t stream) {
  GLOWB200_REQUIRE(segments >= 0 && segments < (1ll << 31) && num_indices >= 0, "segments / num_indices out of range");
  if (segments == 0) return GLOWB200_OK;
  GLOWB200_REQUIRE(lengths != nullptr, "lengths is NULL");
  const size_t need = seg_stride_elems(segments) * 8;
  if (workspace == nullptr || workspace_bytes < need)
    return set_error(GLOWB200_ERR_WORKSPACE_TOO_SMALL, "workspace of %zu bytes given, %zu needed", workspace_bytes, need);
  GLOWB200_REQUIRE(aligned_to(workspace, 8), "workspace must be 8-byte aligned");
  SlwsLaunch L{};
  L.single.lengths = lengths;
  L.single.segments = segments;
  L.single.num_indices = num_indices;
  L.seg_begin = reinterpret_cast<int64_t *>(workspace);
  L.seg_stride = (int64_t)seg_stride_elems(segments);
  L.max_segments = segments;
  L.status = status;
  slws_segments_from_lengths_kernel<<<1, kSegThreads, 0, stream>>>(L);
  GLOWB200_CUDA_OK(cudaGetLastError());
  return GLOWB200_OK;
}

using namespace glowb200;

extern "C" size_t glowb200_slws_workspace_bytes(int64_t max_segments, int64_t num_jobs) {
  if (max_segments < 0 || num_jobs <= 0) return 0;
  return seg_stride_elems(max_segments) * 8 * (size_t)num_jobs;
}

namespace {
int run_batched(const glowb200_slws_job *jobs, int64_t num_jobs, int64_t max_segments, int kind, int indices_are_int64,
                int64_t in_line_size, int64_t out_line_size, int out_is_fp16, int use_fp16_accumulation,
                int64_t num_indices, void *workspace, size_t workspace_bytes, int32_t *status, glowb200_stream_t stream, bool sharded) {
  GLOWB200_REQUIRE(num_jobs >= 0 && num_jobs <= 65535, "num_jobs must be in [0, 65535]");
  GLOWB200_REQUIRE(max_segments >= 0 && max_segments < (1ll << 31), "max_segments out of range");
  if (num_jobs == 0 || max_segments == 0) return GLOWB200_OK;
  GLOWB200_REQUIRE(jobs != nullptr, "jobs is NULL");
  GatherConfig g{kind, indices_are_int64 ? 1 : 0, out_is_fp16 ? 1 : 0,
                 (use_fp16_accumulation && out_is_fp16 && (kind & 1)) ? 1 : 0};
  int align = 16;
  Form form;
  // Table / result pointers of a batched launch live in device memory: the descriptors are
  // required to hold 16-byte aligned tables, which every cudaMalloc'ed slab offset that keeps
  // Glow's 64-byte TensorAlignment satisfies.
  if (int rc = plan(g, in_line_size, out_line_size, true, align, form)) return rc;
  const size_t need = glowb200_slws_workspace_bytes(max_segments, num_jobs);
  if (workspace == nullptr || workspace_bytes < need)
    return set_error(GLOWB200_ERR_WORKSPACE_TOO_SMALL, "workspace of %zu bytes given, %zu needed", workspace_bytes, need);
  GLOWB200_REQUIRE(aligned_to(workspace, 8), "workspace must be 8-byte aligned");
  SlwsLaunch L{};
  L.jobs = jobs;
  L.seg_begin = reinterpret_cast<int64_t *>(workspace);
  L.seg_stride = (int64_t)seg_stride_elems(max_segments);
  L.max_segments = max_segments;
  L.status = status;
  L.in_line = (int32_t)in_line_size;
  L.out_line = (int32_t)out_line_size;
  L.sharded = sharded ? 1 : 0;
  set_types(L, g);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  GLOWB200_CUDA_OK(segments_from_lengths(L, form, max_segments, num_jobs, s));
  return run_gather(L, g, form, align, max_segments, num_jobs, num_indices, s);
}
}  // namespace

extern "C" int glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum_batched(
    const glowb200_slws_job *jobs, int64_t num_jobs, int64_t max_segments, int kind, int indices_are_int64,
    int64_t in_line_size, int64_t out_line_size, int out_is_fp16, int use_fp16_accumulation, void *workspace,
    size_t workspace_bytes, int32_t *status, glowb200_stream_t stream) {
  return run_batched(jobs, num_jobs, max_segments, kind, indices_are_int64, in_line_size, out_line_size, out_is_fp16,
                     use_fp16_accumulation, kRowsUnknown, workspace, workspace_bytes, status, stream, false);
}

extern "C" int glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum_batched_sized(
    const glowb200_slws_job *jobs, int64_t num_jobs, int64_t max_segments, int kind, int indices_are_int64,
    int64_t in_line_size, int64_t out_line_size, int out_is_fp16, int use_fp16_accumulation, int64_t num_indices,
    void *workspace, size_t workspace_bytes, int32_t *status, glowb200_stream_t stream) {
  return run_batched(jobs, num_jobs, max_segments, kind, indices_are_int64, in_line_size, out_line_size, out_is_fp16,
                     use_fp16_accumulation, num_indices, workspace, workspace_bytes, status, stream, false);
}

extern "C" int glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum_row_sharded(
    const glowb200_slws_job *jobs, int64_t num_jobs, int64_t max_segments, int kind, int indices_are_int64,
    int64_t in_line_size, int64_t out_line_size, void *workspace, size_t workspace_bytes, int32_t *status,
    glowb200_stream_t stream) {
  return run_batched(jobs, num_jobs, max_segments, kind, indices_are_int64, in_line_size, out_line_size, 0, 0,
                     kRowsUnknown, workspace, workspace_bytes, status, stream, true);
}

namespace {
int fill_single(SlwsLaunch &L, GatherConfig &g, Form &form, int &align, void *dest, const void *data, int kind, int64_t rows,
                const void *weights, const void *indices, int idx64, const int32_t *lengths, int64_t segments,
                int64_t num_indices, int64_t in_line, int64_t out_line, int out16, int acc16, void *workspace,
                size_t workspace_bytes, int32_t *status) {
  GLOWB200_REQUIRE(segments >= 0 && segments < (1ll << 31), "segments out of range");
  GLOWB200_REQUIRE(rows >= 0 && rows < (1ll << 31) && num_indices >= 0, "rows must be in [0, 2^31), num_indices >= 0");
  GLOWB200_REQUIRE(segments == 0 || (dest && (num_indices == 0 || (data && weights && indices))),
                   "NULL tensor pointer");
  // (slws_run.cu counts rows in 32 bits)
  const bool fit = aligned_to(dest, out16 ? 2 : 4) && aligned_to(weights, out16 ? 2 : 4) && aligned_to(indices, idx64 ? 8 : 4) &&
                   num_indices <= kMostRows;
  g = GatherConfig{kind, idx64 ? 1 : 0, out16 ? 1 : 0, (acc16 && out16 && (kind & 1)) ? 1 : 0};
  align = (int)(reinterpret_cast<uintptr_t>(data) & 15) | 16;
  if (int rc = plan(g, in_line, out_line, fit, align, form)) return rc;
  const size_t need = glowb200_slws_workspace_bytes(segments, 1);
  if (segments > 0 && (workspace == nullptr || workspace_bytes < need))
    return set_error(GLOWB200_ERR_WORKSPACE_TOO_SMALL, "workspace of %zu bytes given, %zu needed", workspace_bytes, need);
  GLOWB200_REQUIRE(aligned_to(workspace, 8), "workspace must be 8-byte aligned");
  L = SlwsLaunch{};
  L.jobs = nullptr;
  L.single.data = data;
  L.single.weights = weights;
  L.single.indices = indices;
  L.single.lengths = lengths;
  L.single.dest = dest;
  L.single.rows = rows;
  L.single.num_indices = num_indices;
  L.single.dest_stride = out_line;
  L.single.segments = segments;
  L.seg_begin = reinterpret_cast<int64_t *>(workspace);
  L.seg_stride = (int64_t)seg_stride_elems(segments);
  L.max_segments = segments;
  L.status = status;
  L.in_line = (int32_t)in_line;
  L.out_line = (int32_t)out_line;
  set_types(L, g);
  return GLOWB200_OK;
}
}  // namespace

extern "C" int glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum(
    void *dest, const void *data, int kind, int64_t rows, const void *weights, const void *indices,
    int indices_are_int64, const int32_t *lengths, int64_t segments, int64_t num_indices, int64_t in_line_size,
    int64_t out_line_size, int out_is_fp16, int use_fp16_accumulation, void *workspace, size_t workspace_bytes,
    int32_t *status, glowb200_stream_t stream) {
  SlwsLaunch L;
  GatherConfig g;
  Form form;
  int align;
  if (int rc = fill_single(L, g, form, align, dest, data, kind, rows, weights, indices, indices_are_int64, lengths, segments,
                           num_indices, in_line_size, out_line_size, out_is_fp16, use_fp16_accumulation, workspace,
                           workspace_bytes, status))
    return rc;
  if (segments == 0) return GLOWB200_OK;
  GLOWB200_REQUIRE(lengths != nullptr, "lengths is NULL");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  GLOWB200_CUDA_OK(segments_from_lengths(L, form, segments, 1, s));
  return run_gather(L, g, form, align, segments, 1, num_indices, s);
}

extern "C" int glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum_low_latency(
    void *dest, const void *data, int kind, int64_t rows, const void *weights, const void *indices,
    int indices_are_int64, const int32_t *lengths, int64_t segments, int64_t num_indices, int64_t in_line_size,
    int64_t out_line_size, int out_is_fp16, void *workspace, size_t workspace_bytes, int32_t *status,
    glowb200_stream_t stream) {
  return glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum(dest, data, kind, rows, weights, indices, indices_are_int64,
                                                                      lengths, segments, num_indices, in_line_size, out_line_size,
                                                                      out_is_fp16, 0, workspace, workspace_bytes, status, stream);
}

extern "C" int glowb200_embedding_bag_byte_rowwise_offsets(
    void *dest, const void *data, int kind, int64_t rows, const void *weights, const void *indices,
    const void *offsets, int indices_are_int64, int64_t num_offsets, int64_t num_indices, int64_t in_line_size,
    int64_t out_line_size, int has_end_offset, int out_is_fp16, int use_fp16_accumulation, void *workspace,
    size_t workspace_bytes, int32_t *status, glowb200_stream_t stream) {
  GLOWB200_REQUIRE(num_offsets >= 0, "negative num_offsets");
  const int64_t segments = has_end_offset ? num_offsets - 1 : num_offsets;
  if (segments <= 0) return GLOWB200_OK;
  GLOWB200_REQUIRE(offsets != nullptr, "offsets is NULL");
  SlwsLaunch L;
  GatherConfig g;
  Form form;
  int align;
  if (int rc = fill_single(L, g, form, align, dest, data, kind, rows, weights, indices, indices_are_int64, nullptr, segments,
                           num_indices, in_line_size, out_line_size, out_is_fp16, use_fp16_accumulation, workspace,
                           workspace_bytes, status))
    return rc;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const unsigned blocks = (unsigned)((segments + 1 + 255) / 256 < 1024 ? (segments + 1 + 255) / 256 : 1024);
  if (indices_are_int64)
    slws_segments_from_offsets_kernel<int64_t><<<blocks, 256, 0, s>>>(L, reinterpret_cast<const int64_t *>(offsets), has_end_offset ? 1 : 0);
  else
    slws_segments_from_offsets_kernel<int32_t><<<blocks, 256, 0, s>>>(L, reinterpret_cast<const int32_t *>(offsets), has_end_offset ? 1 : 0);
  GLOWB200_CUDA_OK(cudaGetLastError());
  return run_gather(L, g, form, align, segments, 1, num_indices, s);
}

// ------------------------------------------------------------------------------------------
// Pooling with no caller-provided workspace and no allocation of any kind.
//
// Who needs this: code that serves requests after all device memory has been handed out.  A
// Glow DeviceManager sizes its slabs when a network is loaded and accounts every byte against
// the device's budget; on its request thread a cudaMalloc could fail against that budget and,
// succeed or fail, stalls every stream of the device while the driver takes its allocator
// lock.  A plug-in that is only ever handed buffers by its host has no allocator at all.  Such
// callers cannot size a workspace per request either, so the bag boundaries go into a fixed
// array that is part of the library image.
//
// The array costs kStaticScratchMaxSegments * 8 bytes (+ padding) of device memory on every
// GPU that loads the library, for the life of the process.
// ------------------------------------------------------------------------------------------
namespace glowb200 {
namespace {
constexpr int64_t kStaticScratchMaxSegments = 65536;
constexpr size_t kStaticScratchBytes = ((kStaticScratchMaxSegments + 2) * 8 + 255) / 256 * 256;
constexpr int kStaticScratchMaxDevices = 64;
}  // namespace
}  // namespace glowb200

// Device storage.  In host code this name is only a handle for the runtime's symbol lookup --
// it is NOT a device address and must never be passed to a kernel as one.
static __device__ __align__(256) unsigned char g_slws_static_scratch[glowb200::kStaticScratchBytes];

namespace glowb200 {
namespace {
// Device address of g_slws_static_scratch on the CURRENT device, looked up once per device.
int static_scratch_address(void **out) {
  static void *cached[kStaticScratchMaxDevices] = {nullptr};
  static bool known[kStaticScratchMaxDevices] = {false};
  static std::mutex lock;
  int dev = -1;
  GLOWB200_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kStaticScratchMaxDevices)
    return set_error(GLOWB200_ERR_UNSUPPORTED, "device ordinal %d is beyond the %d this entry point tracks", dev,
                     kStaticScratchMaxDevices);
  std::lock_guard<std::mutex> guard(lock);
  if (!known[dev]) {
    void *ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_slws_static_scratch);
    if (e != cudaSuccess || ptr == nullptr)
      return set_error(GLOWB200_ERR_CUDA, "cudaGetSymbolAddress(static scratch) on device %d failed: %s", dev,
                       cudaGetErrorString(e));
    cached[dev] = ptr;
    known[dev] = true;
  }
  *out = cached[dev];
  return GLOWB200_OK;
}
}  // namespace
}  // namespace glowb200

extern "C" int64_t glowb200_slws_static_scratch_max_segments(void) { return glowb200::kStaticScratchMaxSegments; }

extern "C" int glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum_static_scratch(
    void *dest, const void *data, int kind, int64_t rows, const void *weights, const void *indices,
    int indices_are_int64, const int32_t *lengths, int64_t segments, int64_t num_indices, int64_t in_line_size,
    int64_t out_line_size, int out_is_fp16, int use_fp16_accumulation, int32_t *status, glowb200_stream_t stream) {
  if (segments > kStaticScratchMaxSegments)
    return set_error(GLOWB200_ERR_UNSUPPORTED,
                     "%lld bags exceed the %lld the built-in scratch array holds; use the entry point that takes a "
                     "workspace", (long long)segments, (long long)kStaticScratchMaxSegments);
  if (segments <= 0) {
    GLOWB200_REQUIRE(segments == 0, "segments out of range");
    return GLOWB200_OK;
  }
  void *scratch = nullptr;
  if (int rc = static_scratch_address(&scratch)) return rc;
  SlwsLaunch L;
  GatherConfig g;
  Form form;
  int align;
  if (int rc = fill_single(L, g, form, align, dest, data, kind, rows, weights, indices, indices_are_int64, lengths, segments,
                           num_indices, in_line_size, out_line_size, out_is_fp16, use_fp16_accumulation, scratch,
                           kStaticScratchBytes, status))
    return rc;
  GLOWB200_REQUIRE(lengths != nullptr, "lengths is NULL");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // The segments kernel rewrites everything this call reads (segments + 1 boundaries); nothing in the
  // array has to start at zero, and whatever an earlier call left beyond them is never read.
  GLOWB200_CUDA_OK(segments_from_lengths(L, form, segments, 1, s));
  return run_gather(L, g, form, align, segments, 1, num_indices, s);
}
