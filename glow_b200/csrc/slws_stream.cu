// Gather-pool with fp32 accumulation for launches that fill the GPU with wide rows: a warp walks the rows of a run of bags
// as one stream, 32 rows to a step, which it copies whole into shared memory a step ahead.
//
// slws_run.cu gives a bag to a group of lanes, four rows of every group on their way at a time, and holds them in
// registers: 20 warps on an SM that wait for those rows, then for the arithmetic of sixteen columns per lane and row.
// Here a row is a whole warp's, V columns to a lane, so nothing is uneven between lanes, and a step's rows lie in shared
// memory, so that 32 of them are on their way beside the 32 that are being added up, and no register is spent on
// either.  The pieces of a row are the aligned 16-byte ones that it lies across, its scale and offset among them: each
// line is asked for once.  Every column is the same chain of operations in the same order as in slws_run.cu,
//     acc[k] = fma(w * scale, q[k], acc[k])   and   offsets = fma(w, offset, offsets)
// row by row, so a bag has the same bits in either kernel.
//
// What bounds it is instructions, 25 to a row of 128 columns (12 of them its arithmetic, whose byte permutes, packed adds
// and packed multiply-adds take a scheduler two cycles each), with what latency 20 warps leave; shared memory allows no
// more.  Blocks are one warp: its slot is free as soon as its own run is done (two warps to a block: 464 -> 474 us in the
// first line below).  A ring of registers for the rows on their way did worse (529 - 1050): a warp has few counters to wait
// on, so that waiting for one row waits for most of them.  So did three steps in shared memory, and steps of 16 rows
// (530 - 630).
// Measured, us, slws_run.cu (with slws_spread.cu for skewed tables) -> this one, power-law lengths unless even:
//   uint8, 128 columns: 64 tables of 4096 bags 541 -> 465; 4 x 8192 90 -> 73; 86 x 244 114 -> 69, even 54 -> 51; 47 x 250 66 -> 42, even
//     41 -> 33; 16 x 4096 bags of 6 rows 56 -> 41; 96 columns: 20 x 3000 241 -> 165, even 174 -> 149
//   4-bit: 4 x 8192 even bags of 64 rows of 128 columns 120 -> 101; 8 x 4000 of 256 157 -> 120, even 104 -> 87
//   up to 64 columns, 32 warps of half the registers: 20 x 2000 of 64 97 -> 84, 6 x 8192 of 48 94 -> 79, even 70 -> 60; 105 x 489
//     4-bit of 48 178 -> 102; 256 even tables of 64, which the rate of random lines bounds, 316 in either
// Not better, and not taken: 4-bit rows of 64 columns (40 x 2000 98 against 113), uint8 ones where the boundaries are known
// (4 x 5000 even 22 against 25), uint8 rows of more than 128, of which shared memory holds too few (10 x 3000 even of 256 114
// against 122), and bags of a row or two (32 x 4096 of 128 36 against 38).
// Not better, and taken all the same, as the host knows neither the skew nor whether L2 holds the tables: even bags over small tables
// (50,000 rows).  4 x 8192 of 64 rows of 128 4-bit columns 93 -> 101 (from memory, 10 M rows: 120 -> 101), of uint8 ones 95 -> 99, of 56 4-bit ones with
// halves 75 -> 83 (1 M rows 89 -> 87, skewed 132 -> 116); 2 x 8192 of 16 rows of 40 columns 28 -> 34 (1 M rows 34 -> 34, skewed ones of
// 56 4-bit columns 58 -> 50).
#include <algorithm>

#include "slws.cuh"

namespace glowb200 {
namespace {

constexpr int kStep = 32;     // rows of a step: lane l knows row l
constexpr int kStages = 2;    // steps in shared memory: being added up, on its way
// Warps on an SM, by the registers they are given: 64 or 96.
constexpr int warps_per_sm(int v) { return v == 2 ? 32 : 20; }
// Pieces of a row that slws_run.cu could pool as well.  It reads the sectors that hold columns or the scale, and this kernel the
// whole row: rows stored apart (ops.pad_fused_rows) are copied with the padding between.  Even bags lose by that, skewed ones gain
// as long as the rest of the launch gains more; the lines lie where the two are about equal.  This kernel's time over slws_run.cu's (with
// slws_spread.cu), 8 x 4000 bags of 40 rows, 16 x 2000 of 20, one of 20,000 of 30 and 100 x 512 of 30, even; skewed:
//   uint8, 40 columns in 160 bytes 1.02 1.00 1.04 1.00; 0.95 0.76 1.00 0.72, in 224 1.10 1.08 1.11 1.12; 1.03 0.88 1.01 0.82, in 256 1.20 1.14 1.14 1.17; 1.06 0.87 1.06 0.85
//   uint8, 96 columns in 192 bytes 0.96 0.97 1.03 0.97; 0.85 0.68 0.85 0.66, in 256 1.10 1.08 1.05 1.09; 0.90 0.73 0.90 0.72
//   4-bit, 48 columns in 128 bytes 0.98 0.96 1.04 0.95; 0.95 0.72 1.01 0.71, in 192 1.08 1.07 1.14 1.09; 1.04 0.84 1.00 0.80, in 256 1.25 1.21 1.17 1.24; 1.11 0.91 1.10 0.90
//   4-bit, 96 columns in 192 bytes 0.98 1.02 1.03 1.04; 0.85 0.77 0.86 0.77, in 256 1.11 1.15 1.06 1.16; 0.91 0.82 0.91 0.84
//   128 with halves in 192 bytes 1.01 1.04 1.04 1.07; 1.00 0.63 0.98 0.63, in 256 1.13 1.18 1.09 1.21; 1.07 0.67 1.07 0.68
//   4-bit, 256 columns in 256 bytes 0.97 0.95 0.95 0.98; 0.82 0.56 0.91 0.67
//   uint8 with halves, whose rows the other kernels read in words, 96 columns in 256 bytes 0.92 0.93 0.93 0.91; 0.90 0.53 0.90 0.52
//   uint8, 64 columns in 128 bytes (boundaries unknown) 256 x 1024 of 32, tables of 1 M rows 0.94, of 0.5 M 1.12; 0.97; 40 x 2000 of 20 1.17; 0.88, 100 x 512 0.97;
//     0.77, in 192 16 x 2000 1.09; 1.01, 100 x 512 1.05; 0.84, in 256 1.22; 1.09, 1.18; 0.94
int most_chunks(int kind, int columns) { return columns <= 64 && kind != GLOWB200_UINT8_FUSED_FP16 ? 12 : 18; }
constexpr int kMostChunksAlone = 32;  // of any other row

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void copy_piece(uint32_t to, const uint8_t *from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
}
// 16 bytes, the first `valid` of them from global memory and the rest zero
__device__ __forceinline__ void copy_piece_part(uint32_t to, const uint8_t *from, int valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(valid) : "memory");
}

// The columns of a lane as they lie in a row.
template <int BYTES, int ALIGN>
__device__ __forceinline__ void lds_lane(uint32_t at, uint32_t *v) {
  if constexpr (BYTES == 1) {
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v[0]) : "r"(at));
  } else if constexpr (BYTES == 2) {
    uint16_t h;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(at));
    v[0] = h;
  } else if constexpr (BYTES == 4) {
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v[0]) : "r"(at));
  } else if constexpr (ALIGN == 8) {
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(at));
  } else {
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v[0]) : "r"(at));
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v[1]) : "r"(at + 4));
  }
}

// Shared memory of a warp: the rows of kStages steps, `chunks` 16-byte pieces each; {weight, where the row begins in its
// pieces (-1: it is not there)} of each; of the rows being added up {w * scale, the same, w, offset}, and where their
// columns are; and the numbers of the rows being copied.
__host__ __device__ constexpr int warp_bytes(int chunks) { return kStages * kStep * (chunks * 16 + 8) + kStep * (16 + 4 + 4); }

// acc += (q * scale + offset) * w for the columns of a word, each operation rounded on its own.  (Packed operations of two
// columns, for all their ".rn", come out fused; and a scheduler issues as many of these.)
__device__ __forceinline__ void pool_word_strict(uint32_t word, float scale, float offset, float w, uint64_t *acc, int pairs) {
#pragma unroll
  for (int i = 0; i < pairs; i++) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(acc[i]));
    auto add = [&](float sum, uint32_t selector) {
      const float q = __fadd_rn(__uint_as_float(__byte_perm(word, 0x4B000000u, selector)), -8388608.0f);
      return __fadd_rn(sum, __fmul_rn(__fadd_rn(__fmul_rn(q, scale), offset), w));
    };
    a = add(a, 0x7440 + 2 * i);
    b = add(b, 0x7441 + 2 * i);
    asm("mov.b64 %0, {%1, %2};" : "=l"(acc[i]) : "f"(a), "f"(b));
  }
}

// V columns per lane.  STRICT: uint8 rows of a width that slws_gather_any_kernel pools else, by its operations: (q * scale + offset)
// * w added up, each rounded on its own, as the reference's Interpreter has them (20 x 2000 of 100 columns 321 -> 76 us).
// CUT: the table starts off 16 bytes, and the bytes in front of it, which row 0's first piece has, are not to be read.  (An
// instance of its own: in all of them it cost 64 skewed tables of 4096 bags of 128 columns 546 -> 554 us.)
template <int BITS, bool SO16, int ALIGN, int V, bool STRICT = false, bool CUT = false>
__global__ void __launch_bounds__(32, warps_per_sm(V)) slws_stream_kernel(const __grid_constant__ SlwsLaunch p, int bags_per_warp, int chunks) {
  pdl_wait();
  pdl_launch_dependents();
  using Row = Rows<BITS, SO16, ALIGN>;
  constexpr int kBytes = V * BITS / 8, kWords = (kBytes + 3) / 4, kPairs = V / 2;
  constexpr int kPairsOfWord = kPairs < 16 / BITS ? kPairs : 16 / BITS;
  constexpr int kTail = SO16 ? 4 : 8, kGroup = V == 2 ? 4 : 8;
  extern __shared__ __align__(16) uint8_t shared[];
  const glowb200_slws_job *jp = p.jobs ? p.jobs + blockIdx.y : &p.single;
  const int lane = threadIdx.x;
  SlwsRun run;
  int32_t flags = 0;
  if (!take_run(p, jp, bags_of(p, jp), (int64_t)blockIdx.x * bags_per_warp, bags_per_warp, lane, run, flags)) return;
  const int32_t rows = (int32_t)jp->rows;
  const uint32_t in_line = (uint32_t)p.in_line;
  const int pitch = chunks * 16, stage_bytes = kStep * pitch;
  const uint32_t stages_at = smem_u32(shared);
  float2 *meta = reinterpret_cast<float2 *>(shared + kStages * stage_bytes);
  float4 *terms = reinterpret_cast<float4 *>(meta + kStages * kStep);
  uint32_t *starts = reinterpret_cast<uint32_t *>(terms + kStep);
  int32_t *numbers = reinterpret_cast<int32_t *>(starts + kStep);
  const bool idx64 = p.idx64 != 0, out16 = p.out16 != 0;
  const int idx_bytes = idx64 ? 8 : 4, w_bytes = out16 ? 2 : 4;
  const int column = lane * V;
  const bool active = column < p.out_line;
  const uint32_t lane_at = active ? lane * kBytes : 0;
  // who copies what: `per_copy` rows at a time, a lane the same piece of one of them every time
  const int per_copy = 32 / chunks, copier = lane / chunks, piece = lane - copier * chunks;
  const uintptr_t data = reinterpret_cast<uintptr_t>(jp->data);
  const uint32_t copy_to = stages_at + copier * pitch + piece * 16;
  // bytes of the lane's piece of the table's last row that are the table's
  const int32_t last_row = rows > 0 ? rows - 1 : INT32_MAX;
  const int behind = (int)(((uint32_t)last_row * in_line + (uint32_t)data) & 15u) + (int)in_line - piece * 16;
  const int last_valid = behind < 0 ? 0 : behind < 16 ? behind : 16;

  uint64_t acc[kPairs];
  float bias = 0.0f;  // sum of w * offset (and, 4-bit, minus the surplus)
#pragma unroll
  for (int i = 0; i < kPairs; i++) acc[i] = 0;

  auto put = [&](int bag) {  // the sums of a finished bag
    const int64_t bag_number = run.first_bag + bag;
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
  };

  // The bags of a run lie behind one another, unless offsets that go backwards have been reported: then each
  // is a stream of its own.
  const int after = __shfl_down_sync(kAllLanes, run.from, 1);
  const bool whole = !__any_sync(kAllLanes, lane + 1 < run.bags && run.from + run.len != after);
#pragma unroll 1
  for (int first = 0; first < run.bags; first += whole ? run.bags : 1) {
    const bool mine = whole ? lane < run.bags : lane == first;
#pragma unroll 1
    for (unsigned empty = __ballot_sync(kAllLanes, mine && run.len == 0); empty != 0; empty &= empty - 1) put(__ffs((int)empty) - 1);
    unsigned todo = __ballot_sync(kAllLanes, mine && run.len > 0);
    if (todo == 0) continue;
    const int32_t start = __shfl_sync(kAllLanes, run.from, first);
    const int32_t past = run.from - start + run.len;  // (of lanes that are `mine`)
    int32_t end = mine && run.len > 0 ? past - 1 : -1;  // the last row of the lane's bag, counted from the step being added up
    const char *indices = reinterpret_cast<const char *>(jp->indices) + (run.begin + start + lane) * idx_bytes;
    uintptr_t weights = reinterpret_cast<uintptr_t>(jp->weights) + (run.begin + start + lane) * w_bytes;
    // index and weight of the lane's row of the step that is copied next, of which there are `left` rows
    int32_t left = __shfl_sync(kAllLanes, past, whole ? run.bags - 1 : first);
    uint2 index;
    uint32_t word;
    bool high;
    auto request = [&]() {
      const int take = left - 1 - lane;
      high = (weights & 2) != 0;
      index = ldg_index(indices, take, idx64);
      word = ldg_if(reinterpret_cast<const void *>(weights & ~(uintptr_t)3), take);
      indices += kStep * idx_bytes;
      weights += kStep * w_bytes;
    };
    auto copy = [&](int stage) {
      const int32_t r = lane < left ? row_number(p, jp, rows, index, idx64, flags) : -1;
      const float w = out16 ? __half2float(__ushort_as_half((unsigned short)(high ? word >> 16 : word))) : __uint_as_float(word);
      meta[stage * kStep + lane] = make_float2(w, __int_as_float(r < 0 ? -1 : (int)(((uint32_t)r * in_line + (uint32_t)data) & 15u)));
      numbers[lane] = r;
      const bool plain = !__any_sync(kAllLanes, r < 0 || r == last_row || (CUT && r == 0));
      __syncwarp();
      const uint32_t to = copy_to + stage * stage_bytes;
      const int32_t *number = numbers + copier;
      auto from = [&](int k) {  // the lane's piece of row k
        return reinterpret_cast<const uint8_t *>((data + piece * 16 + (uint64_t)(uint32_t)number[k] * in_line) & ~(uintptr_t)15);
      };
      if (copier < per_copy) {
        if (plain) {
          int k = 0;
#pragma unroll 4
          for (; k + per_copy <= kStep; k += per_copy) copy_piece(to + k * pitch, from(k));
          if (k + copier < kStep) copy_piece(to + k * pitch, from(k));
        } else {
          // (a row that is not there is not read: as row 0 it cost a launch of bags of one row 900 us, all warps at the same lines)
          for (int k = 0; k + copier < kStep; k += per_copy) {
            if (CUT && piece == 0 && number[k] == 0) {  // (word by word)
              for (int b = (int)data & 15; b < 16; b += 4)
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(to + k * pitch + b), "r"(__ldg(reinterpret_cast<const uint32_t *>(from(k) + b))) : "memory");
            } else if (number[k] >= 0) {
              copy_piece_part(to + k * pitch, from(k), number[k] == last_row ? last_valid : 16);
            }
          }
        }
      }
      __syncwarp();  // every lane has read its rows' numbers (the lanes do not leave the copies together): the next step's may come
      left -= kStep;
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };

    request();
#pragma unroll
    for (int s = 0; s < kStages - 1; s++) {
      if (left > 0) {
        copy(s);
        request();
      }
      commit();
    }
    int stage = 0, next = kStages - 1;
#pragma unroll 1
    while (true) {
      if (left > 0) {
        copy(next);
        request();
      }
      commit();
      const unsigned ends = __reduce_or_sync(kAllLanes, (unsigned)end < (unsigned)kStep ? 1u << end : 0u);
      end -= kStep;
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
      __syncwarp();
      {
        const float2 m = meta[stage * kStep + lane];
        const int begins = __float_as_int(m.y);
        const uint32_t at = stages_at + stage * stage_bytes + lane * pitch + (begins < 0 ? 0 : begins);
        uint2 tail;
        lds_lane<kTail, ALIGN>(at + in_line - kTail, &tail.x);
        float scale, offset;
        Row::scale_offset(tail, scale, offset);
        const float a = m.x * scale * Row::kUnit;
        if constexpr (STRICT) terms[lane] = begins >= 0 ? make_float4(scale, offset, m.x, 0.0f) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        else terms[lane] = begins >= 0 ? make_float4(a, a, m.x, offset) : make_float4(0.0f, 0.0f, 0.0f, -0.0f);
        starts[lane] = at;
      }
      __syncwarp();
#pragma unroll 1
      for (int u = 0; u < kStep; u += kGroup) {
        float4 c[kGroup];
        uint32_t q[kGroup][kWords];
#pragma unroll
        for (int k = 0; k < kGroup; k++) c[k] = terms[u + k];
#pragma unroll
        for (int k = 0; k < kGroup; k += 4) {
          const uint4 at = *reinterpret_cast<const uint4 *>(starts + u + k);
          lds_lane<kBytes, ALIGN>(at.x + lane_at, q[k]);
          lds_lane<kBytes, ALIGN>(at.y + lane_at, q[k + 1]);
          lds_lane<kBytes, ALIGN>(at.z + lane_at, q[k + 2]);
          lds_lane<kBytes, ALIGN>(at.w + lane_at, q[k + 3]);
        }
        const unsigned ending = ends >> u & ((1u << kGroup) - 1u);
        auto add = [&](int k) {
          if constexpr (STRICT) {
            pool_word_strict(q[k][0], c[k].x, c[k].y, c[k].z, acc, kPairs);
          } else {
            uint64_t a2;
            asm("mov.b64 %0, {%1, %2};" : "=l"(a2) : "f"(c[k].x), "f"(c[k].y));
#pragma unroll
            for (int i = 0; i < kWords; i++) pool_word<BITS, kPairsOfWord>(q[k][i], a2, acc + i * kPairsOfWord);
            bias = fmaf(c[k].z, c[k].w, bias);
            if (BITS == 4) bias -= c[k].x;
          }
        };
        if (ending == 0) {
#pragma unroll
          for (int k = 0; k < kGroup; k++) add(k);
        } else {
#pragma unroll
          for (int k = 0; k < kGroup; k++) {
            add(k);
            if (ending >> k & 1) {
              put(__ffs((int)todo) - 1);
              todo &= todo - 1;
            }
          }
          if (todo == 0) break;
        }
      }
      if (todo == 0) break;
      __syncwarp();  // the step's pieces and terms have been read
      stage = stage + 1 == kStages ? 0 : stage + 1;
      next = next + 1 == kStages ? 0 : next + 1;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
  }
  raise_status(p.status, flags);
}

// Columns of a lane.
int columns_of(const SlwsLaunch &L) { return L.out_line <= 64 ? 2 : L.out_line <= 128 ? 4 : 8; }

template <int BITS, bool SO16, int ALIGN, bool CUT = false>
cudaError_t launch_columns(const SlwsLaunch &L, int run, int chunks, dim3 grid, cudaStream_t s) {
  auto kernel = columns_of(L) == 2 ? slws_stream_kernel<BITS, SO16, ALIGN, 2, false, CUT> : slws_stream_kernel<BITS, SO16, ALIGN, 4, false, CUT>;
  if constexpr (BITS == 8) {
    if (L.out_line % 8 != 0)
      kernel = columns_of(L) == 2 ? slws_stream_kernel<BITS, SO16, ALIGN, 2, true, CUT> : slws_stream_kernel<BITS, SO16, ALIGN, 4, true, CUT>;
  } else {
    if (columns_of(L) == 8) kernel = slws_stream_kernel<BITS, SO16, ALIGN, 8, false, CUT>;
  }
  return launch_pdl(kernel, grid, 32, warp_bytes(chunks), s, L, run, chunks);
}

// 16-byte pieces that a row lies across at most, by what the rows start on (tables of a batch start on 16 bytes: the descriptors'
// contract).
int chunks_of(const SlwsLaunch &L) {
  const uintptr_t at = (L.jobs ? 0 : reinterpret_cast<uintptr_t>(L.single.data)) | (uintptr_t)L.in_line;
  const int start = (at & 15) == 0 ? 16 : (at & 7) == 0 ? 8 : 4;
  return (L.in_line + (16 - start) + 15) / 16;
}

}  // namespace

bool slws_stream_takes(const SlwsLaunch &L, int align) {
  // (a row's pieces may reach 20 bytes into the next row)
  return align >= 4 && L.out_line % 4 == 0 && L.out_line <= (L.kind >= 2 ? 256 : 128) && L.in_line >= 32 &&
         chunks_of(L) <= (L.out_line % 8 == 0 ? most_chunks(L.kind, L.out_line) : kMostChunksAlone);
}

cudaError_t launch_slws_stream(const SlwsLaunch &L, int align, int64_t max_segments, int64_t num_jobs, cudaStream_t s) {
  // Bags to a warp: two rounds of warps where that is up to eight, three of the smallest launches whose boundaries are
  // known; that leaves a skewed table's longest run so much shorter and costs an even one little (4 x 8192 4-bit bags of 64 rows,
  // runs of 6 101 us, of 12 101, of 9 116; 16,000 skewed bags of 128, runs of 2 51, of 3 53, of 6 56).  Then six (20 x 3000 skewed of 96
  // columns 165, of 12 178), and twelve where the rounds are many (64 x 4096 of 128, runs of 6 486 us, of 12 467, of 16 464;
  // 256 x 1024 of 64 with nothing left in L2, runs of 3 337, of 6 320, of 12 316, of 32 327).
  const int chunks = chunks_of(L);
  const int64_t total = max_segments * num_jobs;
  const int64_t resident = (int64_t)sm_count() * std::min(warps_per_sm(columns_of(L)), 228 * 1024 / (warp_bytes(chunks) + 1024));
  const int64_t round = std::max<int64_t>(1, (total + resident - 1) / resident);
  const int run = (int)(round <= 16 ? (round + 1) / (round <= 6 && round > 1 && !L.inline_lengths ? 3 : 2) : round <= 40 ? 6 : 12);
  const dim3 grid((unsigned)((max_segments + run - 1) / run), (unsigned)num_jobs);
  if (!L.jobs && (reinterpret_cast<uintptr_t>(L.single.data) & 15) != 0) {
    switch (L.kind) {
      case GLOWB200_UINT8_FUSED: return launch_columns<8, false, 4, true>(L, run, chunks, grid, s);
      case GLOWB200_UINT8_FUSED_FP16: return launch_columns<8, true, 4, true>(L, run, chunks, grid, s);
      case GLOWB200_UINT4_FUSED: return launch_columns<4, false, 4, true>(L, run, chunks, grid, s);
      default: return launch_columns<4, true, 4, true>(L, run, chunks, grid, s);
    }
  }
  switch (L.kind) {
    case GLOWB200_UINT8_FUSED: return align == 8 ? launch_columns<8, false, 8>(L, run, chunks, grid, s) : launch_columns<8, false, 4>(L, run, chunks, grid, s);
    case GLOWB200_UINT8_FUSED_FP16: return launch_columns<8, true, 4>(L, run, chunks, grid, s);
    case GLOWB200_UINT4_FUSED: return align == 8 ? launch_columns<4, false, 8>(L, run, chunks, grid, s) : launch_columns<4, false, 4>(L, run, chunks, grid, s);
    default: return launch_columns<4, true, 4>(L, run, chunks, grid, s);
  }
}

}  // namespace glowb200
