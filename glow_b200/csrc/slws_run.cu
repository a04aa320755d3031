// Gather-pool with fp32 accumulation: a group of lanes walks whole bags, taking the next bag of its warp's
// run whenever it has finished one.
//
// A group of `lpr` lanes (a power of two, 4..32) pools one bag at a time: lane gl owns chunks gl,
// gl + lpr, ... of 8 columns, and the rows of the bag are added in index order,
//     acc[k] = fma(w * scale, q[k], acc[k])   and   offsets = fma(w, offset, offsets)
// (the reference's CPU backend is itself compiled with fast-math, so its float result is defined only
// up to reassociation; tolerance 1e-5 relative).  Every bag is summed by one group in the same order
// whatever else the launch holds, so a table gives the same bits pooled alone, beside others, in runs,
// one bag per group, or by slws_spread.cu.
//
// Why this shape.  The kernels before it gave an evenly filled table's bags one group each -- the groups of
// a warp then wait for its longest bag -- and a skewed table's bags a whole warp each, which spent 42 warp
// instructions per 136-byte row on partly filled steps and on folding the row slots at every bag end.
// Here the groups of a warp are busy until its run of up to 32 bags is used up, and a step costs its
// arithmetic (two instructions per column pair and row) plus what all groups share.  256 even tables of 64
// columns, bound by the rate of random DRAM lines: 329 -> 310 us.  What is left to it beside slws_stream.cu:
// rows of up to 32 columns, 4-bit ones of less than 32 bytes or 57 to 64 columns, uint8 ones of more than 128 (10 x 3000 even bags
// of 256 114 us against 122), bags of a few rows, rows stored far apart, and the middle sizes that slws_spread.cu lists.
//
// Memory.  U rows per group are requested before the first is consumed, and the indices of the group's next
// step -- of its next bag, if this step ends one -- while they are on their way.  What decides is that none
// of the loads in flight is spilled: with two registers too few the same launches take twice as long.
//   * large launches: U = 4, ten blocks of 64 threads on an SM (96 registers); 4-bit rows with four chunks
//     per lane U = 8 and six blocks;
//   * a launch too small to fill the SMs: U = 16, so that a bag of 32 rows is two dependent steps instead of
//     eight (1024 bags of 64 columns: 18.3 + 3.5 us for the boundaries in a launch of their own -> 8.3 us);
//   * in between: U = 8, eight blocks.
// (The launches that slws_spread.cu takes are the smallest of rows of up to 256 columns.)
#include <climits>

#include "slws.cuh"

namespace glowb200 {
namespace {

constexpr int kThreads = 64;  // a block's SM slots stay taken until its slowest warp is done: small blocks
constexpr int kWarps = kThreads / 32;

// P chunks per lane, U rows per step.
template <int BITS, bool SO16, int ALIGN, int P, int U>
__global__ void __launch_bounds__(kThreads, U == 16 ? 4 : P == 4 ? 6 : U == 8 ? 8 : 10)
slws_run_kernel(const __grid_constant__ SlwsLaunch p, int even_run) {
  pdl_wait();
  pdl_launch_dependents();
  using R = Rows<BITS, SO16, ALIGN>;
  constexpr int KI = U / 4;  // index registers: lanes 0..3 of a group hold rows gl, gl + 4, ...
  const glowb200_slws_job *jp = p.jobs ? p.jobs + blockIdx.y : &p.single;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t segments = bags_of(p, jp);
  // (a table whose longest bag stands out: longer runs, the surplus blocks leave)
  const int64_t word = p.inline_lengths ? 0 : p.seg_begin[(int64_t)blockIdx.y * p.seg_stride + segments + 1];
  const int bags_per_warp = word != 0 ? p.skewed_run : even_run;
  const int64_t first_bag = ((int64_t)blockIdx.x * kWarps + warp) * bags_per_warp;
  if (first_bag >= segments || (p.skip_from != 0 && word >= p.skip_from)) return;  // whole warps leave together
  const int n_bags = (int)(first_bag + bags_per_warp < segments ? bags_per_warp : segments - first_bag);
  const int lpr = 1 << p.lpr_log2, gl = lane & (lpr - 1);
  const int64_t N = jp->num_indices;
  const int32_t rows = (int32_t)jp->rows;
  const int in_line = p.in_line, chunks = p.out_line >> 3;
  int32_t flags = 0;

  // ---- bag boundaries: lane l holds where bag l of the run begins, relative to the run, and how many
  // rows it has (take_run, written out: behind a call the 256 even tables above took 0.7 % longer) ----
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
    int32_t own = lane < n_bags ? lengths[fb + lane] : 0;
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
  } else if (lane < n_bags) {
    const int64_t *sb = p.seg_begin + (int64_t)blockIdx.y * p.seg_stride + first_bag + lane;
    begin = sb[0];
    len = sb[1] - begin;
    if (len < 0) { len = 0; flags |= GLOWB200_STATUS_BAD_OFFSETS; }
  }
  // Positions are 32-bit, relative to where the run begins.  (Index arrays of more than kMostRows entries are the
  // any-shape kernel's where the host can see them; here a run that long is cut short and reported.)
  const int64_t run0 = __shfl_sync(kAllLanes, begin, 0);
  int64_t rel = begin - run0;
  if (lane < n_bags && (rel + len > kMostRows || rel < INT32_MIN)) { rel = 0; len = 0; flags |= GLOWB200_STATUS_LENGTHS_OVERRUN; }
  const int32_t from_l = (int32_t)rel, len_l = (int32_t)len;

  // ---- what a group is doing: its bag, where its next row is, how many are left ----
  const bool idx64 = p.idx64 != 0, out16 = p.out16 != 0;
  const int idx_bytes = idx64 ? 8 : 4, w_bytes = out16 ? 2 : 4;
  const char *indices = reinterpret_cast<const char *>(jp->indices) + (run0 + gl) * idx_bytes;
  const char *weights = reinterpret_cast<const char *>(jp->weights) + (run0 + gl) * w_bytes;
  const unsigned leaders_before = (1u << (lane - gl)) - 1u;
  int counter = 0;  // bags of the run handed out
  int bag = -1, left = 0, pos = 0;
  struct Step {
    int n, bag;   // rows (0..U) and the bag they belong to (-1: the group has none)
    bool last;    // they end it
  };
  struct Request {     // lane gl < 4: rows gl, gl + 4, ... of the step, as loaded
    uint2 index[KI];
    uint32_t word[KI]; // of the weight, which is all of it or (fp16) the half `high` says
    bool high;
  };
  auto advance = [&](Step &s, Request &q) {
    const unsigned asking = __ballot_sync(kAllLanes, left == 0 && gl == 0);
    if (asking != 0) {
      const int mine = counter + __popc(asking & leaders_before);
      counter += __popc(asking);
      const int32_t f = __shfl_sync(kAllLanes, from_l, mine & 31), l = __shfl_sync(kAllLanes, len_l, mine & 31);
      if (left == 0) {
        const bool got = mine < n_bags;
        bag = got ? mine : -1;
        left = got ? l : 0;
        pos = f;
      }
    }
    s.n = left < U ? left : U;
    s.bag = bag;
    left -= s.n;
    s.last = bag >= 0 && left == 0;
    const char *ip = indices + (int64_t)pos * idx_bytes;
    const uintptr_t wp = reinterpret_cast<uintptr_t>(weights) + (int64_t)pos * w_bytes;
    q.high = (wp & 2) != 0;
#pragma unroll
    for (int k = 0; k < KI; k++) {
      const int take = gl < 4 ? s.n - 1 - (gl + 4 * k) : -1;
      q.index[k] = ldg_index(ip + 4 * k * idx_bytes, take, idx64);
      q.word[k] = ldg_if(reinterpret_cast<const void *>((wp & ~(uintptr_t)3) + 4 * k * w_bytes), take);
    }
    pos += s.n;
  };

  const uint8_t *data = reinterpret_cast<const uint8_t *>(jp->data) + gl * R::kBytes;
  bool has[P];
  uint64_t acc[P][4];  // pairs of columns
  float bias = 0.0f;   // sum of w * offset (and, 4-bit, minus the surplus)
#pragma unroll
  for (int c = 0; c < P; c++) {
    has[c] = c * lpr + gl < chunks;
#pragma unroll
    for (int i = 0; i < 4; i++) acc[c][i] = 0;
  }
  void *const dest0 = jp->dest;
  void *const *const dests = jp->dests;
  const int64_t dest_stride = jp->dest_stride, bags_per_dest = jp->bags_per_dest;

  Step s;
  Request q;
  advance(s, q);
  while (__any_sync(kAllLanes, s.bag >= 0)) {
    // ---- row numbers (tables have fewer than 2^31 rows; -1: nothing to add) ----
    int32_t r[KI];
    float w[KI];
#pragma unroll
    for (int k = 0; k < KI; k++) {
      r[k] = -1;
      if (gl < 4 && gl + 4 * k < s.n) {
        if (p.sharded) {
          const int64_t raw = idx64 ? (int64_t)((uint64_t)q.index[k].y << 32 | q.index[k].x) : (int64_t)(int32_t)q.index[k].x,
                        v = raw - jp->row_begin;
          if (v >= 0 && v < rows) r[k] = (int32_t)v;
          else if (raw < 0 || raw >= jp->global_rows) flags |= GLOWB200_STATUS_INDEX_OUT_OF_RANGE;  // else: another shard's row
        } else if (q.index[k].x < (uint32_t)rows && (!idx64 || q.index[k].y == 0)) {
          r[k] = (int32_t)q.index[k].x;
        } else {
          flags |= GLOWB200_STATUS_INDEX_OUT_OF_RANGE;
        }
      }
      w[k] = out16 ? __half2float(__ushort_as_half((unsigned short)(q.high ? q.word[k] >> 16 : q.word[k]))) : __uint_as_float(q.word[k]);
    }
    // ---- their loads ----
    int32_t rr[U];
    uint2 pay[U][P], tl[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      rr[u] = __shfl_sync(kAllLanes, r[u >> 2], u & 3, lpr);
      const uint8_t *row = data + (int64_t)rr[u] * in_line;
#pragma unroll
      for (int c = 0; c < P; c++)
        pay[u][c] = R::chunk(row + c * lpr * R::kBytes, in_line - (c * lpr + gl) * R::kBytes, has[c] ? rr[u] : -1);
      tl[u] = R::tail(row - gl * R::kBytes + in_line, rr[u]);
    }
    const Step now = s;
    float ww[U];
#pragma unroll
    for (int u = 0; u < U; u++) ww[u] = __shfl_sync(kAllLanes, w[u >> 2], u & 3, lpr);
    advance(s, q);
    // ---- and their sums ----
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (U > 4 && (u & 3) == 0 && u > 0 && !__any_sync(kAllLanes, now.n > u)) break;
      float scale, offset;
      R::scale_offset(tl[u], scale, offset);
      float a = ww[u] * scale * R::kUnit;
      float next = fmaf(ww[u], offset, bias);
      if (BITS == 4) next -= a;
      a = rr[u] >= 0 ? a : 0.0f;
      bias = rr[u] >= 0 ? next : bias;
#pragma unroll
      for (int c = 0; c < P; c++) R::pool(pay[u][c], a, acc[c]);
    }
    // ---- a finished bag ----
    if (now.last) {
      const int64_t b = first_bag + now.bag;
      void *base = dest0;
      int64_t dest_row = b;
      if (bags_per_dest > 0) {  // scatter over several (possibly remote) destination buffers
        const int64_t which = b < bags_per_dest ? 0 : (int64_t)((uint32_t)b / (uint32_t)bags_per_dest);
        base = dests[which];
        dest_row = b - which * bags_per_dest;
      }
      uint64_t bias2;
      asm("mov.b64 %0, {%1, %1};" : "=l"(bias2) : "f"(bias));
#pragma unroll
      for (int c = 0; c < P; c++) {
        float o[8];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          asm("add.rn.f32x2 %0, %1, %2;" : "=l"(acc[c][i]) : "l"(acc[c][i]), "l"(bias2));
          asm("mov.b64 {%0, %1}, %2;" : "=f"(o[2 * i]), "=f"(o[2 * i + 1]) : "l"(acc[c][i]));
          acc[c][i] = 0;
        }
        if (!has[c]) continue;
        const int64_t at = dest_row * dest_stride + (int64_t)(c * lpr + gl) * 8;
        if (out16) {
          __half *d = reinterpret_cast<__half *>(base) + at;
          __half2 h[4];
#pragma unroll
          for (int i = 0; i < 4; i++) h[i] = __floats2half2_rn(o[2 * i], o[2 * i + 1]);
          if ((reinterpret_cast<uintptr_t>(d) & 15u) == 0) {
            *reinterpret_cast<uint4 *>(d) = *reinterpret_cast<const uint4 *>(h);
          } else {
#pragma unroll
            for (int i = 0; i < 8; i++) d[i] = i & 1 ? __high2half(h[i / 2]) : __low2half(h[i / 2]);
          }
        } else {
          float *d = reinterpret_cast<float *>(base) + at;
          if ((reinterpret_cast<uintptr_t>(d) & 15u) == 0) {
            *reinterpret_cast<float4 *>(d) = make_float4(o[0], o[1], o[2], o[3]);
            *reinterpret_cast<float4 *>(d + 4) = make_float4(o[4], o[5], o[6], o[7]);
          } else {
#pragma unroll
            for (int i = 0; i < 8; i++) d[i] = o[i];
          }
        }
      }
      bias = 0.0f;
    }
  }
  raise_status(p.status, flags);
}

template <int BITS, bool SO16, int ALIGN>
cudaError_t launch_rows(const SlwsLaunch &L, int P, int U, dim3 grid, int bpw, cudaStream_t s) {
  if constexpr (BITS == 4) {
    if (U == 8 && P == 2) return launch_pdl(slws_run_kernel<BITS, SO16, ALIGN, 2, 8>, grid, kThreads, 0, s, L, bpw);
  }
  if (U == 8) return launch_pdl(slws_run_kernel<BITS, SO16, ALIGN, 1, 8>, grid, kThreads, 0, s, L, bpw);
  if (U == 16) {
    if (P == 1) return launch_pdl(slws_run_kernel<BITS, SO16, ALIGN, 1, 16>, grid, kThreads, 0, s, L, bpw);
    if (P == 2) return launch_pdl(slws_run_kernel<BITS, SO16, ALIGN, 2, 16>, grid, kThreads, 0, s, L, bpw);
    return launch_pdl(slws_run_kernel<BITS, SO16, ALIGN, 4, 16>, grid, kThreads, 0, s, L, bpw);
  }
  if (P == 1) return launch_pdl(slws_run_kernel<BITS, SO16, ALIGN, 1, 4>, grid, kThreads, 0, s, L, bpw);
  if (P == 2) return launch_pdl(slws_run_kernel<BITS, SO16, ALIGN, 2, 4>, grid, kThreads, 0, s, L, bpw);
  return launch_pdl(slws_run_kernel<BITS, SO16, ALIGN, 4, BITS == 4 ? 8 : 4>, grid, kThreads, 0, s, L, bpw);
}

}  // namespace

cudaError_t launch_slws_run(SlwsLaunch L, int align, int64_t max_segments, int64_t num_jobs, cudaStream_t s) {
  const int chunks = L.out_line / 8;
  const int64_t total = max_segments * num_jobs, sms = sm_count();
  auto lanes_log2 = [&](int per_lane) {
    int l = 2;  // (four lanes at least: they hold a step's indices)
    while ((per_lane << l) < chunks) l++;
    return l;
  };
  auto warps_for = [&](int bags) { return (max_segments + bags - 1) / bags; };
  // Small and medium launches are bound by the chain of steps of the longest bag, and with a warp or two per
  // scheduler by that warp's own instructions: 16 (8) rows per step, and one chunk per lane, so that a bag is
  // spread over more lanes and the bags over more warps.  A column's sum is the same either way.  (Measured
  // on launches that slws_spread.cu has taken since: 18 tables, 91 bags of up to 200 rows of 64 columns 20.8 -> 15.9 us;
  // 1024 bags of 64 columns 8.2 -> 7.0.)  Above 32 warps per SM the fewer rows in flight of more warps win.
  int P = 1, bpw = 0, U = 4;
  if (chunks <= 32) {
    L.lpr_log2 = lanes_log2(1);
    bpw = 32 >> L.lpr_log2;
    const int64_t n = warps_for(bpw) * num_jobs;
    U = n <= sms * 8 ? 16 : n <= sms * 32 ? 8 : 4;
  }
  if (U == 4) {
    P = chunks_per_lane(chunks, L.kind >= 2);
    L.lpr_log2 = lanes_log2(P);
    // A warp's run: one bag per group in small launches; up to 32 bags once that still leaves every SM two
    // dozen warps, one dozen where eight groups of a warp would wait for its longest bag.  Skewed tables (the
    // boundaries' kernel knows) even out over such runs: 702 us with runs of 8, 540 with 32.  The others
    // take them as long as the warps still fill the rounds in which they become resident, or all fit one:
    // 12 tables, 8192 bags of 64 rows of 64 columns, 1.04 rounds of runs of 32 295 us, 4.2 rounds of 8 221; 20
    // tables, 2000 skewed bags, 1.7 rounds of 8 99 us, one of 16 72.  With eight groups to a warp and the skew
    // known a bag per group is the better run even in full rounds (40 4-bit tables of 32 columns 524 -> 502 us);
    // with four the blocks that skewed tables then leave over cost more (64 of them: 569 -> 606).
    const bool wide_steps = L.kind >= 2 && P == 2;
    const int64_t resident = sms * (P == 4 ? 12 : wide_steps ? 16 : 20);
    auto filled = [&](int bags) {  // of the slots of those rounds, per cent
      const int64_t n = warps_for(bags) * num_jobs;
      return 100 * n / ((n + resident - 1) / resident * resident);
    };
    bpw = 32 >> L.lpr_log2;
    const int64_t enough = sms * (bpw >= 8 && P <= 2 ? 12 : 24);
    const int lpr = 1 << L.lpr_log2;
    int64_t best = filled(bpw);
    for (int run = 2 * bpw; run <= kMaxRun && total / run >= enough; run *= 2) {
      L.skewed_run = run;
      if (((lpr > 4 || L.inline_lengths) && filled(run) * 100 >= best * 95) || warps_for(run) * num_jobs <= resident) bpw = run;
      if (filled(run) > best) best = filled(run);
    }
    if (warps_for(bpw) * num_jobs <= sms * 8) U = 16;
    // (two 4-bit chunks are eight bytes: eight rows of them still fit the registers.  64 tables, 1000 skewed bags
    // of 64 columns: 131 -> 92 us; two uint8 chunks would make it eight rows for 20 tables 43 -> 51)
    else if (wide_steps) U = 8;
  }
  if (L.skewed_run < bpw) L.skewed_run = bpw;
  const int64_t warps = warps_for(bpw);
  const dim3 grid((unsigned)((warps + kWarps - 1) / kWarps), (unsigned)num_jobs);
  switch (L.kind) {
    case GLOWB200_UINT8_FUSED:
      if (align == 8) return launch_rows<8, false, 8>(L, P, U, grid, bpw, s);
      return align == 4 ? launch_rows<8, false, 4>(L, P, U, grid, bpw, s) : launch_rows<8, false, 1>(L, P, U, grid, bpw, s);
    case GLOWB200_UINT8_FUSED_FP16:
      return align >= 4 ? launch_rows<8, true, 4>(L, P, U, grid, bpw, s) : launch_rows<8, true, 1>(L, P, U, grid, bpw, s);
    case GLOWB200_UINT4_FUSED:
      if (align == 8) return launch_rows<4, false, 8>(L, P, U, grid, bpw, s);
      return align >= 4 ? launch_rows<4, false, 4>(L, P, U, grid, bpw, s) : launch_rows<4, false, 1>(L, P, U, grid, bpw, s);
    default:
      return align >= 4 ? launch_rows<4, true, 4>(L, P, U, grid, bpw, s) : launch_rows<4, true, 1>(L, P, U, grid, bpw, s);
  }
}

}  // namespace glowb200
