// Gather-pool with fp32 accumulation for launches in which the longest bag decides: a bag is spread over many
// lanes with few columns each, two steps of its rows in flight.
//
// slws_run.cu gives a bag to a group of 4 .. 32 lanes of 8 columns each, which suits bags that all SMs are full of.
// In a small launch, or one of a few skewed tables, the groups of a warp have long run out of bags when its longest
// is still a chain of steps, each of them a fetch and the instructions of 8 columns per lane and row.  Here LANES lanes
// (a warp, or half of one) with V = 2, 4 or 8 columns each take a bag: a row is two to four times fewer
// instructions on that chain, a step 16 or 32 rows, and the rows of the next step are requested before those of this
// one are added up.  Every column is the same chain of operations in the same order as in slws_run.cu,
//     acc[k] = fma(w * scale, q[k], acc[k])   and   offsets = fma(w, offset, offsets)
// row by row, so a bag has the same bits in either kernel.
//
// What bounds it is that chain.  Row numbers, and later {w * scale twice, w, offset}, pass from the lane that has them
// to the group through shared memory, four rows (one row) per load: a shuffle per row in front of each row's load
// cost 115 - 190 cycles a row, the whole chain now takes about 60.  What decides beside it is that no load in flight
// is spilled (blocks_per_sm).  18 tables, 91 skewed bags of up to 200 rows of 64 columns: 16.5 -> 12.0 us, of 4-bit
// rows 16.8 -> 14.3; even bags of 40 rows 7.2 -> 6.2; 64 x 100 skewed bags of 128 columns 41 -> 33, even ones
// 24.6 -> 18.0; 1024 even bags of 64 columns, one table 6.8 -> 5.6.
#include <algorithm>

#include "slws.cuh"

namespace glowb200 {
namespace {

constexpr int kThreads = 64;
constexpr int kWarps = kThreads / 32;

// The V columns of a lane, one word of them, as they lie in a row.
template <int BYTES>
__device__ __forceinline__ uint32_t ldg_columns(const uint8_t *p) {
  uint32_t v;
  if constexpr (BYTES == 1) {
    asm volatile("ld.global.nc.u8 %0, [%1];" : "=r"(v) : "l"(p));
  } else if constexpr (BYTES == 2) {
    uint16_t h;
    asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(h) : "l"(p));
    v = h;
  } else {
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
  }
  return v;
}

// Blocks on an SM: as many as leave every load in flight a register.
constexpr int blocks_per_sm(int bits, int v, int lanes, int r) {
  return lanes == 32 ? (r == 32 || bits == 8 ? 6 : 8) : v == 8 ? (bits == 4 ? 7 : 6) : 8;
}

// V columns per lane, LANES lanes per bag, R rows per step.
template <int BITS, bool SO16, int ALIGN, int V, int LANES, int R>
__global__ void __launch_bounds__(kThreads, blocks_per_sm(BITS, V, LANES, R)) slws_spread_kernel(const __grid_constant__ SlwsLaunch p, int bags_per_warp) {
  // (beside the launch of the even tables, which has waited already; whoever waits for this one waits for both)
  if (!p.only_from) pdl_wait();
  pdl_launch_dependents();
  using Row = Rows<BITS, SO16, ALIGN>;
  constexpr int kBytes = V * BITS / 8, kWords = (kBytes + 3) / 4, kPairs = V / 2;
  constexpr int kPairsOfWord = kPairs < 16 / BITS ? kPairs : 16 / BITS;
  static_assert(R <= LANES, "lane l of a group knows row l of a step");
  constexpr int kGroups = 32 / LANES;
  __shared__ float4 shared_terms[kWarps][kGroups * R];
  __shared__ int4 shared_rows[kWarps][kGroups * R / 4];
  const glowb200_slws_job *jp = p.jobs ? p.jobs + blockIdx.y : &p.single;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gl = lane & (LANES - 1), group = lane / LANES;
  SlwsRun run;
  int32_t flags = 0;
  const int64_t segments = bags_of(p, jp);
  auto leave = [&]() { if (p.only_from && blockIdx.x == 0 && blockIdx.y == 0) pdl_wait(); };
  if (p.only_from && p.seg_begin[(int64_t)blockIdx.y * p.seg_stride + segments + 1] < p.only_from) return leave();
  if (!take_run(p, jp, segments, ((int64_t)blockIdx.x * kWarps + warp) * bags_per_warp, bags_per_warp, lane, run, flags)) return leave();  // whole warps leave together
  const int32_t rows = (int32_t)jp->rows;
  const int in_line = p.in_line;
  float4 *terms = shared_terms[warp] + group * R;  // of the rows being added up: {w * scale, the same, w, offset}
  int4 *row_numbers = shared_rows[warp] + group * (R / 4);
  const bool idx64 = p.idx64 != 0, out16 = p.out16 != 0;
  const int idx_bytes = idx64 ? 8 : 4, w_bytes = out16 ? 2 : 4;
  const char *indices = reinterpret_cast<const char *>(jp->indices) + (run.begin + gl) * idx_bytes;
  const char *weights = reinterpret_cast<const char *>(jp->weights) + (run.begin + gl) * w_bytes;
  const int column = gl * V;
  const bool active = column < p.out_line;
  const uint8_t *data = reinterpret_cast<const uint8_t *>(jp->data), *columns_at = data + (active ? gl * kBytes : 0);

  uint64_t acc[kPairs];
  float bias = 0.0f;  // sum of w * offset (and, 4-bit, minus the surplus)
#pragma unroll
  for (int i = 0; i < kPairs; i++) acc[i] = 0;

  struct Step {
    int n, bag;  // rows (n = 0: an empty bag), and the bag they belong to (-1: the group has none)
    bool last;   // they end it
  };
  struct Request {  // of lane l: row l of the step
    uint2 index;
    uint32_t word;  // the weight, or (fp16) the word that holds it
    bool high;
  };
  struct Block {  // the rows of a step on their way
    uint32_t columns[R][kWords];
    uint2 tail;  // of lane l: row l
    float w;
    int32_t r;
  };
  int counter = 0;  // bags of the run handed out
  int bag = -1, left = 0, pos = 0;
  auto request = [&](Step &s, Request &q) {
    if (counter < run.bags) {
      const unsigned asking = __ballot_sync(kAllLanes, left == 0 && gl == 0);
      const int mine = counter + __popc(asking & ((1u << (lane - gl)) - 1u));
      counter += __popc(asking);
      const int32_t f = __shfl_sync(kAllLanes, run.from, mine & 31), l = __shfl_sync(kAllLanes, run.len, mine & 31);
      if (left == 0) {
        const bool got = mine < run.bags;
        bag = got ? mine : -1;
        left = got ? l : 0;
        pos = f;
      }
    } else if (left == 0) {
      bag = -1;
    }
    s.n = left < R ? left : R;
    s.bag = bag;
    left -= s.n;
    s.last = bag >= 0 && left == 0;
    const uintptr_t at = reinterpret_cast<uintptr_t>(weights) + (int64_t)pos * w_bytes;
    const int take = s.n - 1 - gl;
    q.high = (at & 2) != 0;
    q.index = ldg_index(indices + (int64_t)pos * idx_bytes, take, idx64);
    q.word = ldg_if(reinterpret_cast<const void *>(at & ~(uintptr_t)3), take);
    pos += s.n;
  };
  auto most = [&](int n) { return kGroups == 1 ? n : (int)__reduce_max_sync(kAllLanes, (unsigned)n); };
  auto fetch = [&](const Step &s, const Request &q, Block &b) {
    __syncwarp();
    b.r = gl < s.n ? row_number(p, jp, rows, q.index, idx64, flags) : -1;
    b.w = out16 ? __half2float(__ushort_as_half((unsigned short)(q.high ? q.word >> 16 : q.word))) : __uint_as_float(q.word);
    // One word of columns: a row that is not there is read as row 0, without a predicate, and adds nothing (13 tables,
    // 2164 skewed 4-bit bags 94 -> 80 us; where a lane has two words of them 131 -> 144).
    if (gl < R) reinterpret_cast<int32_t *>(row_numbers)[gl] = kWords == 1 && b.r < 0 ? 0 : b.r;
    __syncwarp();
    b.tail = Row::tail(data + (int64_t)b.r * in_line + in_line, b.r);
    if (kWords == 1 && rows == 0) return;  // (the whole warp)
    const int n = most(s.n);
    constexpr int kAtOnce = 8;
#pragma unroll
    for (int u0 = 0; u0 < R; u0 += kAtOnce) {
      if (u0 > 0 && u0 >= n) break;
      int4 r4[kAtOnce / 4];
#pragma unroll
      for (int k = 0; k < kAtOnce / 4; k++) r4[k] = row_numbers[u0 / 4 + k];
#pragma unroll
      for (int k = 0; k < kAtOnce; k++) {
        const int32_t r = k % 4 == 0 ? r4[k / 4].x : k % 4 == 1 ? r4[k / 4].y : k % 4 == 2 ? r4[k / 4].z : r4[k / 4].w;
        if constexpr (kWords == 1) {
          b.columns[u0 + k][0] = ldg_columns<kBytes>(columns_at + (int64_t)r * in_line);
        } else {
          const uint8_t *at = data + (int64_t)r * in_line + gl * kBytes;
          const uint2 q = ALIGN == 8 ? ldg2_if(at, active ? r : -1) : make_uint2(ldg_if(at, active ? r : -1), ldg_if(at + 4, active ? r : -1));
          b.columns[u0 + k][0] = q.x;
          b.columns[u0 + k][kWords - 1] = q.y;
        }
      }
    }
  };
  auto add_up = [&](const Step &s, const Block &b) {
    __syncwarp();
    float scale, offset;
    Row::scale_offset(b.tail, scale, offset);
    const float a = b.w * scale * Row::kUnit;
    // (a row that is not there adds nothing: -0 leaves every sum as it is)
    if (gl < R) terms[gl] = b.r >= 0 ? make_float4(a, a, b.w, offset) : make_float4(0.0f, 0.0f, 0.0f, -0.0f);
    __syncwarp();
    const int n = most(s.n);
#pragma unroll
    for (int u = 0; u < R; u++) {
      if ((u & 3) == 0 && u >= n) break;
      const float4 c = terms[u];
      uint64_t a2;
      asm("mov.b64 %0, {%1, %2};" : "=l"(a2) : "f"(c.x), "f"(kWords == 1 ? c.y : c.x));
#pragma unroll
      for (int k = 0; k < kWords; k++) pool_word<BITS, kPairsOfWord>(b.columns[u][k], a2, acc + k * kPairsOfWord);
      bias = fmaf(c.z, c.w, bias);
      if (BITS == 4) bias -= c.x;
    }
    if (s.last) {
      const int64_t bag_number = run.first_bag + s.bag;
      void *to = jp->dest;
      int64_t dest_row = bag_number;
      if (jp->bags_per_dest > 0) {  // scatter over several (possibly remote) destination buffers
        const int64_t bags_per_dest = jp->bags_per_dest, which = bag_number < bags_per_dest ? 0 : (int64_t)((uint32_t)bag_number / (uint32_t)bags_per_dest);
        to = jp->dests[which];
        dest_row = bag_number - which * bags_per_dest;
      }
      store_columns<V>(to, dest_row * jp->dest_stride + column, acc, bias, out16, active ? V : 0);
      bias = 0.0f;
#pragma unroll
      for (int i = 0; i < kPairs; i++) acc[i] = 0;
    }
  };
  Step s0, s1, s2;
  Request q0, q1;
  Block even, odd;
  request(s0, q0);
  request(s1, q1);
  fetch(s0, q0, even);
  while (true) {
    // (two steps: each has its own registers)
    request(s2, q0);
    fetch(s1, q1, odd);
    add_up(s0, even);
    if (!__any_sync(kAllLanes, s1.bag >= 0)) break;
    s0 = s2;
    request(s2, q1);
    fetch(s0, q0, even);
    add_up(s1, odd);
    if (!__any_sync(kAllLanes, s0.bag >= 0)) break;
    s1 = s2;
  }
  raise_status(p.status, flags);
  leave();
}

struct SpreadShape { int columns, lanes, rows, run; };  // V, LANES, R and the bags of a warp

template <int BITS, bool SO16, int ALIGN>
cudaError_t launch_shape(const SlwsLaunch &L, const SpreadShape &c, dim3 grid, cudaStream_t s) {
#define GLOWB200_SPREAD(V, LANES, R) \
  if (c.columns == V && c.lanes == LANES && c.rows == R) return launch_pdl(slws_spread_kernel<BITS, SO16, ALIGN, V, LANES, R>, grid, kThreads, 0, s, L, c.run)
  GLOWB200_SPREAD(2, 32, 32);
  GLOWB200_SPREAD(4, 16, 16);
  GLOWB200_SPREAD(4, 32, 32);
  GLOWB200_SPREAD(8, 16, 16);
  if constexpr (BITS == 4) GLOWB200_SPREAD(8, 32, 32);
  GLOWB200_SPREAD(8, 32, 16);
#undef GLOWB200_SPREAD
  return cudaErrorInvalidValue;
}

cudaError_t launch_slws_spread(const SlwsLaunch &L, SpreadShape c, int align, int64_t max_segments, int64_t num_jobs, cudaStream_t s) {
  const int64_t warps = (max_segments + c.run - 1) / c.run;
  const dim3 grid((unsigned)((warps + kWarps - 1) / kWarps), (unsigned)num_jobs);
  switch (L.kind) {
    case GLOWB200_UINT8_FUSED: return align == 8 ? launch_shape<8, false, 8>(L, c, grid, s) : launch_shape<8, false, 4>(L, c, grid, s);
    case GLOWB200_UINT8_FUSED_FP16: return launch_shape<8, true, 4>(L, c, grid, s);
    case GLOWB200_UINT4_FUSED: return align == 8 ? launch_shape<4, false, 8>(L, c, grid, s) : launch_shape<4, false, 4>(L, c, grid, s);
    default: return launch_shape<4, true, 4>(L, c, grid, s);
  }
}

}  // namespace

// Which kernel pools a launch.  Rows of up to 256 columns at 4-byte boundaries; wider ones fill a warp in
// slws_run.cu as well.  Widths off the eights have slws_stream.cu alone.
//   * slws_stream.cu takes the rows that suit it (see there for both sides of every line) from 24 bags per SM on of up to 64
//     columns; of wider ones from 64 on, or, where the boundaries are known and with them the skewed tables, from 84 on (47 x 250
//     41 against 33 us, 8 x 1000 of 20 rows 14.2 against 15.7; one table of 12,000 skewed bags 38 against 43).  Not bags of fewer than
//     five rows on average, nor of twelve in launches of up to 150 bags per SM (64 x 250 of 10 rows 14.2 against 16.0).
//     Where the host does not know the rows (the unsized entry points, row shards) bags of a few may be among them: 16 x 2000 even bags of one, three and
//     ten rows of 64 columns 15 -> 21, 18 -> 23 and 31.5 -> 32.5 us, of 40 47 -> 46; but skewed ones of one to three on average 66 -> 40 and
//     73 -> 44, of 20 98 -> 76.  The rows of a row shard that are elsewhere take a place in a step all the same, which the widths that leave no lanes of
//     slws_run.cu's groups idle show (half, a quarter, an eighth of the rows here, 2 M to a table, 16 x 2000 bags of 40: 128 4-bit
//     columns even 72 - 66 -> 76 - 71, skewed 194 - 187 -> 125 - 116; uint8 80 - 69 -> 79 - 71, 181 - 168 -> 134 - 122; of 96 columns 78 - 69 -> 73 - 66, 180 - 168 ->
//     124 - 114).
//     What follows is the rules for the others.
//   * small launches take this one: up to the 12 bags per SM that are resident at once of rows of 32 columns, which leave
//     half of the lanes idle here (2 x 211 skewed bags 16.9 -> 11.4 us); up to 24 of 64 columns (26 x 128 13.7 -> 11.7); up to 84 of
//     wider rows, which occupy a warp per bag in either kernel (30 tables, 400 skewed 4-bit bags of 96 columns: 67 -> 50,
//     even ones 31.3 -> 31.3; 14 x 567, 192 columns 73 -> 50; 5 x 1465 even uint8 bags of 256 columns 45 -> 41). Above that even
//     bags are slws_run.cu's (86 x 244 of 128 columns 32.7 against 38.6), and so are those just above 12 per SM, where
//     half of the warps would have two (5 x 400 of 64 columns 5.0 against 5.6, of 128 5.4 against 5.8), and uint8
//     rows of more than 128 columns as long as slws_run.cu gives them a warp per bag and 8 or 16 rows per step as well
//     (5 x 400 of 192 columns 29.3 against 32.2).
//   * bags of fewer than eight rows on average are one step in either kernel, and slws_run.cu has fewer warps to start
//     (12 x 100 bags of 3 rows of 64 columns 3.8 against 4.3 us, 40 x 64 4.2 against 5.2, one table of 4 bags 3.3 against 3.5).
//   * in launches of up to 384 bags per SM whose boundaries' kernel knows which tables are skewed, those are a
//     launch of their own beside that of the even tables: 13 tables, 2164 skewed 4-bit bags of 48 columns 108 -> 80 us,
//     2 x 6965 of 64 68 -> 45, 8 x 4000 of 256 177 -> 136; where no table is skewed it costs 0.3 to 0.7 us, so not with less than
//     2^17 rows (2 x 2100 even bags of 10 rows 8.4 -> 9.1).  uint8 rows of more than 64 columns only with bags of 128 rows and
//     more: 8 x 4096 of 128 144 -> 130 (10 x 4000 with bags of 12 rows on average, 78 at most, would take 62 instead of 54).
cudaError_t launch_slws(SlwsLaunch L, int align, int64_t max_segments, int64_t num_jobs, int64_t rows, cudaStream_t s) {
  const int64_t total = max_segments * num_jobs, sms = sm_count();
  const int columns = L.out_line;
  const bool four_bit = L.kind >= 2;
  // so many bags to a warp that the warps fill the SMs `times` over
  auto shape = [&](int v, int lanes, int rows, int times) {
    const int64_t slots = sms * kWarps * blocks_per_sm(four_bit ? 4 : 8, v, lanes, rows) * times;
    return SpreadShape{v, lanes, rows, (int)std::min<int64_t>(kMaxRun, std::max<int64_t>(32 / lanes, (total + slots - 1) / slots))};
  };
  if (columns % 8 != 0) return launch_slws_stream(L, align, max_segments, num_jobs, s);
  const bool streams = columns > 32 && slws_stream_takes(L, align) && !(columns > 56 && columns <= 64 && (four_bit || !L.inline_lengths)) &&
                       !(rows >= 0 && rows < total * (total <= sms * 150 ? 12 : 5));
  const int64_t small = sms * (columns <= 32 ? 12 : columns <= 64 ? 24 : streams && L.inline_lengths ? 64 : 84);
  const bool short_bags = rows >= 0 && rows < total * 8, wide_bytes = !four_bit && columns > 128;
  if (align < 4 || columns > 256 || (wide_bytes && total <= sms * 32)) return launch_slws_run(L, align, max_segments, num_jobs, s);
  if (total <= small && !short_bags && !(columns <= 128 && total > sms * 12 && total <= sms * 16)) {
    // (two bags to a warp once it has many; half the rows in flight, and more warps, where 4-bit rows fill it)
    const SpreadShape c = columns <= 64    ? shape(2, 32, 32, 1)
                          : columns <= 128 ? (total <= sms * 54 ? shape(4, 32, 32, 1) : shape(8, 16, 16, 1))
                                           : shape(8, 32, four_bit && total <= sms * 12 ? 32 : 16, 1);
    return launch_slws_spread(L, c, align, max_segments, num_jobs, s);
  }
  if (streams) return launch_slws_stream(L, align, max_segments, num_jobs, s);
  if (columns > 32 && max_segments > kInlineLengthsMax && total <= sms * 384 && (rows < 0 || rows >= 1 << 17))
    L.skip_from = four_bit || columns <= 64 ? 1 : 128;
  if (cudaError_t e = launch_slws_run(L, align, max_segments, num_jobs, s)) return e;
  if (L.skip_from == 0) return cudaSuccess;
  L.only_from = L.skip_from;
  const SpreadShape c = columns <= 64 ? shape(4, 16, 16, 1) : columns > 128 ? shape(8, 32, 16, 3) : four_bit ? shape(8, 16, 16, 3) : shape(4, 32, 32, 3);
  return launch_slws_spread(L, c, align, max_segments, num_jobs, s);
}

}  // namespace glowb200
