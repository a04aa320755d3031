// Table-batched embedding bags: IntNBitSplitEmbeddingBags / IntNBitSplitEmbeddingWeightedBags.
//
// Reference: fwdIntNBitSplitEmbeddingWeightedBagsImpl and the row helpers of
// lib/Backends/Interpreter/InterpreterNodes.cpp:42-114, 6593-6738 (the CPU backend has no kernel
// for this node).  T tables of mixed element type (fp32, fp16, int8, int4) live in one byte
// buffer; int8 / int4 rows start with their scale and offset, rows are padded to a byte
// alignment; the request holds T*B bags, bag (t, b) = offsets[t*B+b] .. offsets[t*B+b+1], and
// the result is [B, total_dims] with table t's columns at dim_offsets[t].
//
// One launch pools every bag of every table.  blockIdx.y is the table; inside a table a group of
// lanes (as many as a row has 16-byte chunks, 8-byte ones for tables off 16-byte boundaries) owns a bag and walks its
// rows in index order, each lane keeping the sums of the columns of its own chunk: every result
// element is accumulated in the reference's order and in the result's type, with the multiply and the add
// kept apart, so results are bit-identical to the Interpreter's.  Three rows are requested before
// the first is consumed.
//
// A chunk of an fp32 or fp16 row, or of a quantized row off 16-byte boundaries, is cut from the row start, not
// from the first column: the first lane's chunk of a quantized row begins with the scale/offset header, so all
// loads stay aligned to the chunk size although the columns start 4 (or 8) bytes into the row.  Quantized rows
// at 16-byte boundaries go by columns (pool_bag_columns).
#include "common.cuh"

namespace glowb200 {
namespace {

struct SplitLaunch {
  void *dest;
  const uint8_t *dev_weights, *uvm_weights;
  int64_t dev_bytes, uvm_bytes;
  const int32_t *placements;
  const void *weights_offsets;
  const uint8_t *weights_tys;
  const int32_t *dim_offsets;
  const void *indices, *offsets;
  const void *indice_weights;
  int32_t *status;
  int64_t num_indices, bags_per_table, total_dims;
  int32_t num_tables, wo64, iw16, so_fp32, row_alignment, pooling_mode;
  int32_t first_column_ty;  // the types from here on take pool_bag_columns where the rows allow it
};

constexpr int kThreads = 128;  // (a bag of a warp ends late: small blocks hand their registers on sooner)
constexpr int kMinBlocks = 8;  // on an SM: 64 registers
// Rows in flight per lane.  Four spill under 64 registers (128-column int4 bags of 64 rows: 207 against 190 us),
// two leave more of the latency bare (210); so do 80 registers and fewer warps (211), and one group of rows being
// added up while the next is on its way measured no better (190).
constexpr int kRows = 3;

enum : int { TY_F32 = 0, TY_F16 = 1, TY_I8 = 2, TY_I4 = 3 };

// The bytes [at, at + 4*CW) of a table as CW words.  A chunk that is aligned and lies inside
// the buffer is one vector load; the last chunk of a buffer that ends with an unpadded row, and
// tables at odd addresses, are put together from single bytes (bytes past the end read as 0).
template <int CW>
__device__ __forceinline__ void load_chunk(const uint8_t *base, int64_t at, int64_t limit, bool vec, uint32_t (&q)[CW]) {
  if (vec && at + 4 * CW <= limit) {
    if constexpr (CW == 4) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(base + at));
      q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
    } else {
      const uint2 v = __ldg(reinterpret_cast<const uint2 *>(base + at));
      q[0] = v.x; q[1] = v.y;
    }
  } else {
#pragma unroll
    for (int w = 0; w < CW; w++) {
      uint32_t word = 0;
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const int64_t o = at + 4 * w + b;
        if (o < limit) word |= (uint32_t)__ldg(base + o) << (8 * b);
      }
      q[w] = word;
    }
  }
}

// N words at p (aligned to their size) if `on`, else 0: a predicate, not a branch, so that the loads of several
// rows go out together.
template <int N>
__device__ __forceinline__ void load_if(bool on, const uint8_t *p, uint32_t (&q)[N]) {
  if constexpr (N == 4) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
                 "@p ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%5];\n\t}"
                 : "=&r"(q[0]), "=&r"(q[1]), "=&r"(q[2]), "=&r"(q[3]) : "r"((int)on), "l"(p));
  } else if constexpr (N == 2) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\t"
                 "@p ld.global.nc.v2.b32 {%0, %1}, [%3];\n\t}"
                 : "=&r"(q[0]), "=&r"(q[1]) : "r"((int)on), "l"(p));
  } else {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %1, 0;\n\tmov.b32 %0, 0;\n\t@p ld.global.nc.b32 %0, [%2];\n\t}"
                 : "=&r"(q[0]) : "r"((int)on), "l"(p));
  }
}

// float(h) for the fp16 number in the low half of `h`, through the mixed-precision add of sm_100
// (adding -0 keeps every value, the sign of a zero included) instead of a conversion
// instruction: conversions issue at an eighth of the rate of adds, and this kernel would be
// bound by them.
__device__ __forceinline__ float add_f32_f16(uint16_t h, float c) {
  float d;
  asm("add.rn.f32.f16 %0, %1, %2;" : "=f"(d) : "h"(h), "f"(c));
  return d;
}
__device__ __forceinline__ float half_bits_to_float(uint32_t h) { return add_f32_f16((uint16_t)(h & 0xFFFFu), -0.0f); }
__device__ __forceinline__ uint64_t pack2f(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void unpack2f(uint64_t v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// Two floats rounded to fp16 (round to nearest even), packed {lo, hi}: one conversion for two.
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

// The sums of a lane's columns: fp32, or -- for an fp16 result -- fp16 pairs, rounded after every row as the
// reference's float16 sum is (float16::operator+, include/glow/Support/Float16.h:47-49): widened, added to in
// fp32 and rounded back.
// Slots (the elements of a lane's words) are handled in pairs: neighbours, except for nibbles, where one
// mask takes nibbles k and k + 4 of a word.
template <int TY>
__device__ __forceinline__ constexpr int slot_of(int pair, int second) {
  return TY == TY_I4 ? 8 * (pair >> 2) + (pair & 3) + 4 * second : 2 * pair + second;
}

// Adds one row's words to the sums.  Quantized elements become floats without a conversion instruction: byte
// or nibble q is merged into the mantissa of the fp16 number 1024 (0x6400 | q = 1024 + q) and 1024 is
// subtracted in the mixed-precision add.  With fp16 headers q * scale is exact in fp32 (8 + 11 significant
// bits), so one fused multiply-add gives the reference's separately rounded q * scale + offset.
// Pairs of fp32 values go through the two-lane fp32 instructions of sm_100 (each lane rounds like the scalar
// instruction, subnormals included) for the dequantising FMA and for the sums of unweighted quantized rows.
// The weight multiply and the add behind it stay scalar: issued as a two-lane multiply followed by a two-lane
// add they did not reproduce the reference's two roundings on its own unit vectors, whereas scalar
// mul.rn / add.rn are never contracted.
template <int TY, int CW, bool OUT16, bool WEIGHTED, bool SO32, int NA, int NH>
__device__ __forceinline__ void add_row(const uint32_t (&q)[CW], uint32_t header0, uint32_t header1, float w, float (&acc)[NA],
                                        uint32_t (&acch)[NH]) {
  constexpr int SLOTS = TY == TY_F32 ? CW : TY == TY_F16 ? 2 * CW : TY == TY_I8 ? 4 * CW : 8 * CW;
  constexpr int PAIRS = SLOTS / 2;
  float scale = 0.0f, offset = 0.0f;
  if constexpr (TY == TY_I8 || TY == TY_I4) {
    if constexpr (SO32) {
      scale = __uint_as_float(header0);
      offset = __uint_as_float(header1);
    } else {
      scale = half_bits_to_float(header0);
      offset = half_bits_to_float(header0 >> 16);
    }
  }
  auto dequant2 = [&](uint32_t h2, float &ta, float &tb) {  // h2 = two fp16 numbers 1024 + q
    const float fa = add_f32_f16((uint16_t)(h2 & 0xFFFFu), -1024.0f), fb = add_f32_f16((uint16_t)(h2 >> 16), -1024.0f);
    if constexpr (SO32) {
      ta = __fadd_rn(__fmul_rn(fa, scale), offset);
      tb = __fadd_rn(__fmul_rn(fb, scale), offset);
    } else {
      uint64_t v2;
      asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v2) : "l"(pack2f(fa, fb)), "l"(pack2f(scale, scale)), "l"(pack2f(offset, offset)));
      unpack2f(v2, ta, tb);
    }
  };
#pragma unroll
  for (int i = 0; i < PAIRS; i++) {
    float ta, tb;  // the values of the pair's slots in this row
    if constexpr (TY == TY_F32) {
      ta = __uint_as_float(q[2 * i]);
      tb = __uint_as_float(q[2 * i + 1]);
    } else if constexpr (TY == TY_F16) {
      ta = half_bits_to_float(q[i]);
      tb = half_bits_to_float(q[i] >> 16);
    } else if constexpr (TY == TY_I8) {
      dequant2(__byte_perm(q[i >> 1], 0x64646464u, (i & 1) ? 0x4342u : 0x4140u), ta, tb);
    } else {  // even column = low nibble, odd column = high nibble (InterpreterNodes.cpp:104-109)
      dequant2(((q[i >> 2] >> (4 * (i & 3))) & 0x000F000Fu) | 0x64006400u, ta, tb);
    }
    if constexpr (WEIGHTED) {  // (an unweighted bag multiplies by 1.0)
      ta = __fmul_rn(w, ta);
      tb = __fmul_rn(w, tb);
    }
    if constexpr (OUT16) {
      // (keeping fp32 copies of the sums and converting both ways every row was tried: half the speed)
      const float lo = add_f32_f16((uint16_t)(acch[i] & 0xFFFFu), ta);
      const float hi = add_f32_f16((uint16_t)(acch[i] >> 16), tb);
      acch[i] = pack_f16x2(lo, hi);
    } else if constexpr (!WEIGHTED && !SO32 && (TY == TY_I8 || TY == TY_I4)) {
      uint64_t s2;
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(s2) : "l"(pack2f(acc[slot_of<TY>(i, 0)], acc[slot_of<TY>(i, 1)])), "l"(pack2f(ta, tb)));
      unpack2f(s2, acc[slot_of<TY>(i, 0)], acc[slot_of<TY>(i, 1)]);
    } else {
      acc[slot_of<TY>(i, 0)] = __fadd_rn(acc[slot_of<TY>(i, 0)], ta);
      acc[slot_of<TY>(i, 1)] = __fadd_rn(acc[slot_of<TY>(i, 1)], tb);
    }
  }
}

// The sums of columns col0 .. (those below 0 or beyond the table's are nobody's), divided by the row count
// for mean pooling.
template <int TY, int SLOTS, bool OUT16, int NA, int NH>
__device__ __forceinline__ void store_sums(const float (&acc)[NA], const uint32_t (&acch)[NH], int32_t col0, int32_t num_dims,
                                           bool mean, int64_t rows, void *out_row) {
  float n = 1.0f;
  if (mean) {
    n = (float)rows;
    if (OUT16) n = __half2float(__float2half_rn(n));
  }
#pragma unroll
  for (int i = 0; i < SLOTS / 2; i++) {
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int slot = slot_of<TY>(i, e);
      const int32_t c = col0 + slot;
      if (c < 0 || c >= num_dims) continue;
      if constexpr (OUT16) {
        const __half h = __ushort_as_half((unsigned short)((acch[i] >> (16 * e)) & 0xFFFFu));
        reinterpret_cast<__half *>(out_row)[c] = mean ? __float2half_rn(__fdiv_rn(__half2float(h), n)) : h;
      } else {
        reinterpret_cast<float *>(out_row)[c] = mean ? __fdiv_rn(acc[slot], n) : acc[slot];
      }
    }
  }
}

// Pools the bag [begin, end) of one table for the lanes of one group.
//   TY   element type of the table; CW words per lane chunk (2 or 4); SO32: fp32 row headers
//   gl / lpr  lane within the group / lanes of the group
template <int TY, int CW, bool OUT16, bool WEIGHTED, bool SO32, typename IdxT>
__device__ __forceinline__ int32_t pool_bag(const SplitLaunch &p, const uint8_t *base, int64_t limit, int64_t table_at,
                                            int32_t row_bytes, int32_t touched, int32_t num_dims, int32_t max_row, bool vec,
                                            int64_t begin, int64_t end, int gl, int lpr, void *out_row) {
  constexpr int CB = 4 * CW;                                           // chunk bytes
  constexpr int SLOTS = TY == TY_F32 ? CW : TY == TY_F16 ? 2 * CW : TY == TY_I8 ? 4 * CW : 8 * CW;
  constexpr int PAIRS = SLOTS / 2;
  constexpr int H = (TY == TY_I8 || TY == TY_I4) ? (SO32 ? 8 : 4) : 0;  // header bytes of a row
  const IdxT *indices = reinterpret_cast<const IdxT *>(p.indices);
  int32_t flags = 0;
  for (int32_t cbase = 0; cbase < touched; cbase += lpr * CB) {
    const int32_t at = cbase + gl * CB;          // byte of the row this lane's chunk starts at
    const bool has = at < touched;
    // column of slot 0 (negative inside the header)
    const int32_t col0 = TY == TY_F32 ? at / 4 : TY == TY_F16 ? at / 2 : TY == TY_I8 ? at - H : 2 * (at - H);
    float acc[OUT16 ? 1 : SLOTS];      // fp32 result: the sums
    uint32_t acch[OUT16 ? PAIRS : 1];  // fp16 result: the sums as fp16 pairs {slot_a, slot_b}
#pragma unroll
    for (int s = 0; s < (OUT16 ? 1 : SLOTS); s++) acc[s] = 0.0f;
#pragma unroll
    for (int s = 0; s < (OUT16 ? PAIRS : 1); s++) acch[s] = 0u;

    // The indices (and weights) of the next kRows rows are requested while the current rows are
    // in flight: an index fetch and the row fetch that depends on it would otherwise add their
    // latencies in every trip of the loop.  A row is kept as a 32-bit number: -2 none, -1 refused.
    int32_t next_r[kRows];
    float next_w[kRows];
    auto request = [&](int64_t j) {
#pragma unroll
      for (int u = 0; u < kRows; u++) {
        next_r[u] = -2;
        next_w[u] = 1.0f;
        if (j + u < end) {
          const int64_t r = (int64_t)indices[j + u];
          next_r[u] = (r < 0 || r > max_row) ? -1 : (int32_t)r;
          if constexpr (WEIGHTED)
            next_w[u] = p.iw16 ? __half2float(reinterpret_cast<const __half *>(p.indice_weights)[j + u])
                               : reinterpret_cast<const float *>(p.indice_weights)[j + u];
        }
      }
    };
    request(begin);
    for (int64_t j = begin; j < end; j += kRows) {
      bool live[kRows];
      float w[kRows];
      uint32_t q[kRows][CW];
      uint32_t hdr[kRows][2] = {};
#pragma unroll
      for (int u = 0; u < kRows; u++) {
        w[u] = next_w[u];
        live[u] = next_r[u] >= 0 && has;
        if (next_r[u] == -1) flags |= GLOWB200_STATUS_INDEX_OUT_OF_RANGE;
        if (!live[u]) continue;
        const int64_t row_at = table_at + (int64_t)next_r[u] * row_bytes;
        load_chunk<CW>(base, row_at + at, limit, vec, q[u]);
        if constexpr (TY == TY_I8 || TY == TY_I4) {
          // all lanes of the group read the same header word(s): one transaction
          if (vec) {
            hdr[u][0] = __ldg(reinterpret_cast<const uint32_t *>(base + row_at));
            hdr[u][1] = SO32 ? __ldg(reinterpret_cast<const uint32_t *>(base + row_at + 4)) : 0u;
          } else {
            uint32_t h2[2];
            load_chunk<2>(base, row_at, limit, false, h2);
            hdr[u][0] = h2[0];
            hdr[u][1] = h2[1];
          }
        }
      }
      request(j + kRows);
#pragma unroll
      for (int u = 0; u < kRows; u++) {
        if (!live[u]) continue;
        add_row<TY, CW, OUT16, WEIGHTED, SO32>(q[u], hdr[u][0], hdr[u][1], w[u], acc, acch);
      }
    }

    if (!has) continue;
    store_sums<TY, SLOTS, OUT16>(acc, acch, col0, num_dims, p.pooling_mode == 1 && end > begin, end - begin, out_row);
  }
  return flags;
}

// The same for quantized rows at 16-byte boundaries whose chunks are cut from the first column instead: a lane's
// LW words are all columns, where chunks from the row start give the first lane a header and the last one
// little more than that (five 16-byte chunks for the 68 bytes of a 128-column int4 row: 160 slots for 128
// columns).  Behind a 4-byte header a lane's four words are three of its aligned 16 bytes and one more load.
// What bounds it is the arithmetic -- four instructions per element is its least (widen and add for the sum, half
// a pack, subtract, half an FMA, extract) -- and the rows' latency, which 27 warps of three rows do not hide.
// 65,536 bags of Poisson(64) int4 rows of 128 columns, fp16 result: 282 us by row chunks and loads in branches, 190 so.
template <int TY, int LW, bool OUT16, bool WEIGHTED, bool SO32, typename IdxT>
__device__ __forceinline__ int32_t pool_bag_columns(const SplitLaunch &p, const uint8_t *table,
                                                    int32_t row_bytes, int32_t touched, int32_t num_dims, int32_t max_row,
                                                    int64_t begin, int64_t end, int gl, int lpr, void *out_row) {
  constexpr int H = SO32 ? 8 : 4, SLOTS = (TY == TY_I8 ? 4 : 8) * LW;
  const IdxT *indices = reinterpret_cast<const IdxT *>(p.indices) + begin;
  // (longer bags do not come here; without the minimum the compiler spills in this loop)
  const int32_t count = (int32_t)(end - begin < 0x7FFFFFF0ll ? end - begin : 0x7FFFFFF0ll);
  int32_t flags = 0;
  for (int32_t word0 = gl * LW; H + 4 * (word0 - gl * LW) < touched; word0 += lpr * LW) {
    const int32_t at = H + 4 * word0;   // byte of the row the lane's words start at
    const bool has = at < touched;
    const bool more = at + 4 * (LW == 4 && SO32 ? 2 : LW - 1) < touched;  // the second load has something to bring
    float acc[OUT16 ? 1 : SLOTS];
    uint32_t acch[OUT16 ? SLOTS / 2 : 1];
#pragma unroll
    for (int s = 0; s < (OUT16 ? 1 : SLOTS); s++) acc[s] = 0.0f;
#pragma unroll
    for (int s = 0; s < (OUT16 ? SLOTS / 2 : 1); s++) acch[s] = 0u;
    int32_t next_r[kRows];  // -2 none, -1 refused
    float next_w[kRows];
    auto request = [&](int32_t j) {
#pragma unroll
      for (int u = 0; u < kRows; u++) {
        next_r[u] = -2;
        next_w[u] = 1.0f;
        if (j + u < count) {
          const IdxT r = indices[j + u];
          next_r[u] = (r < 0 || r > (IdxT)max_row) ? -1 : (int32_t)r;
          if constexpr (WEIGHTED)
            next_w[u] = p.iw16 ? __half2float(reinterpret_cast<const __half *>(p.indice_weights)[begin + j + u])
                               : reinterpret_cast<const float *>(p.indice_weights)[begin + j + u];
        }
      }
    };
    request(0);
    for (int32_t j = 0; j < count; j += kRows) {
      bool live[kRows];
      float w[kRows];
      uint32_t q[kRows][LW], hdr[kRows][2] = {};
#pragma unroll
      for (int u = 0; u < kRows; u++) {
        w[u] = next_w[u];
        live[u] = next_r[u] >= 0 && has;
        if (next_r[u] == -1) flags |= GLOWB200_STATUS_INDEX_OUT_OF_RANGE;
        const uint8_t *row = table + (int64_t)next_r[u] * row_bytes;
        if constexpr (SO32) {
          load_if<2>(live[u], row, hdr[u]);
#pragma unroll
          for (int k = 0; k < LW; k += 2)
            load_if<2>(live[u] && (k == 0 || more), row + at + 4 * k, *reinterpret_cast<uint32_t (*)[2]>(&q[u][k]));
        } else {
          load_if<1>(live[u], row, *reinterpret_cast<uint32_t (*)[1]>(&hdr[u][0]));
          if constexpr (LW == 4) {
            uint32_t v[4];
            load_if<4>(live[u], row + at - 4, v);
            q[u][0] = v[1]; q[u][1] = v[2]; q[u][2] = v[3];
          } else {
            load_if<1>(live[u], row + at, *reinterpret_cast<uint32_t (*)[1]>(&q[u][0]));
          }
          load_if<1>(live[u] && more, row + at + 4 * (LW - 1), *reinterpret_cast<uint32_t (*)[1]>(&q[u][LW - 1]));
        }
      }
      request(j + kRows);
#pragma unroll
      for (int u = 0; u < kRows; u++)
        if (live[u]) add_row<TY, LW, OUT16, WEIGHTED, SO32>(q[u], hdr[u][0], hdr[u][1], w[u], acc, acch);
    }
    if (has)
      store_sums<TY, SLOTS, OUT16>(acc, acch, (TY == TY_I8 ? 4 : 8) * word0, num_dims, p.pooling_mode == 1 && end > begin, end - begin,
                                   out_row);
  }
  return flags;
}

// A table as the lanes of one group see it.
struct TableRows {
  const uint8_t *base;
  int64_t limit, table_at;
  int32_t row_bytes, touched, num_dims, dim_start, table, max_row, gl, lpr;
  bool vec;
};

template <bool COLUMNS, int TY, int CW, bool OUT16, bool WEIGHTED, bool SO32, typename IdxT>
__device__ __forceinline__ int32_t pool_bags(const SplitLaunch &p, const TableRows &r, int64_t first, int64_t step) {
  const IdxT *offsets = reinterpret_cast<const IdxT *>(p.offsets) + (int64_t)r.table * p.bags_per_table;
  int32_t flags = 0;
  for (int64_t b = first; b < p.bags_per_table; b += step) {
    int64_t begin = (int64_t)offsets[b];
    int64_t end = (int64_t)offsets[b + 1];
    if (begin < 0 || end < begin || end > p.num_indices) {
      if (end >= begin) flags |= GLOWB200_STATUS_BAD_OFFSETS;  // a start above its end is an empty bag
      begin = end = 0;
    }
    void *out_row = reinterpret_cast<char *>(p.dest) + ((size_t)(b * p.total_dims + r.dim_start)) * (OUT16 ? 2 : 4);
    if constexpr (COLUMNS)
      flags |= pool_bag_columns<TY, CW, OUT16, WEIGHTED, SO32, IdxT>(p, r.base + r.table_at, r.row_bytes, r.touched, r.num_dims,
                                                                     r.max_row, begin, end, r.gl, r.lpr, out_row);
    else
      flags |= pool_bag<TY, CW, OUT16, WEIGHTED, SO32, IdxT>(p, r.base, r.limit, r.table_at, r.row_bytes, r.touched, r.num_dims, r.max_row, r.vec,
                                                             begin, end, r.gl, r.lpr, out_row);
  }
  return flags;
}

struct SplitTable {
  int32_t dim_start, num_dims, ty, placement;
  bool supported;
};
// (int2 rows and tables placed in device-only memory are not supported by the reference
// either, InterpreterNodes.cpp:6696, 6704: the table's columns stay 0)
__device__ __forceinline__ SplitTable split_table(const SplitLaunch &p, int t) {
  SplitTable d;
  d.dim_start = p.dim_offsets[t];
  d.num_dims = p.dim_offsets[t + 1] - d.dim_start;
  d.ty = p.weights_tys[t];
  d.placement = p.placements[t];
  d.supported = d.ty <= TY_I4 && d.placement != 0 && d.dim_start >= 0 && (int64_t)d.dim_start + d.num_dims <= p.total_dims &&
                d.num_dims <= (1 << 27);
  return d;
}

// The columns no table writes are 0 (the reference clears the result first, InterpreterNodes.cpp:6672).  The
// blocks behind the last table look for them, each for the bags of its turn -- a fill of the whole result was a launch
// of its own, 4 us of 16 MB.  Where the offsets ascend, as they do in earnest, those are the columns in front of the first
// table, behind the last one and of the tables that are not supported; a search through all tables for every column
// (1000 tables of 64: 18 ms) is left for offsets that do not.
template <bool OUT16>
__device__ __forceinline__ void clear_uncovered(const SplitLaunch &p) {
  auto clear = [&](int64_t b, int64_t c) {
    if constexpr (OUT16) reinterpret_cast<uint16_t *>(p.dest)[b * p.total_dims + c] = 0;
    else reinterpret_cast<float *>(p.dest)[b * p.total_dims + c] = 0.0f;
  };
  bool in_order = true;
  for (int t = threadIdx.x; t < p.num_tables; t += kThreads) in_order = in_order && p.dim_offsets[t] <= p.dim_offsets[t + 1];
  if (__syncthreads_and(in_order)) {
    __shared__ int32_t from[kThreads], to[kThreads];
    for (int first = -1; first <= p.num_tables; first += kThreads) {
      const int t = first + (int)threadIdx.x;  // -1: in front of the first table, num_tables: behind the last
      int64_t a = 0, b = 0;
      if (t <= p.num_tables) {
        a = t < 0 ? 0 : p.dim_offsets[t];
        b = t == p.num_tables ? p.total_dims : p.dim_offsets[t + 1];
        if (t >= 0 && t < p.num_tables && split_table(p, t).supported) b = a;
      }
      from[threadIdx.x] = (int32_t)(a > 0 ? a : 0);
      to[threadIdx.x] = (int32_t)(b < p.total_dims ? b : p.total_dims);
      if (__syncthreads_or(from[threadIdx.x] < to[threadIdx.x])) {
        for (int i = 0; i < kThreads; i++)
          if (from[i] < to[i])
            for (int64_t bag = blockIdx.x; bag < p.bags_per_table; bag += gridDim.x)
              for (int c = from[i] + (int)threadIdx.x; c < to[i]; c += kThreads) clear(bag, c);
      }
      __syncthreads();
    }
    return;
  }
  for (int64_t c = (int64_t)blockIdx.x * kThreads + threadIdx.x; c < p.total_dims; c += (int64_t)gridDim.x * kThreads) {
    bool covered = false;
    for (int t = 0; t < p.num_tables && !covered; t++) {
      const SplitTable d = split_table(p, t);
      covered = d.supported && c >= d.dim_start && c < (int64_t)d.dim_start + d.num_dims;
    }
    if (covered) continue;
    for (int64_t b = 0; b < p.bags_per_table; b++) clear(b, c);
  }
}

template <bool OUT16, typename IdxT>
__global__ void __launch_bounds__(kThreads, kMinBlocks) split_embedding_bags_kernel(const __grid_constant__ SplitLaunch p) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.y;
  if (t == p.num_tables) return clear_uncovered<OUT16>(p);
  const SplitTable d = split_table(p, t);
  const int32_t num_dims = d.num_dims;
  if (num_dims <= 0) return;
  if (!d.supported) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && p.status != nullptr) atomicOr(p.status, GLOWB200_STATUS_UNSUPPORTED_TABLE);
    return;
  }
  const int ty = d.ty, so = p.so_fp32 ? 4 : 2;
  const int32_t unpadded = ty == TY_F32 ? num_dims * 4 : ty == TY_F16 ? num_dims * 2
                         : ty == TY_I8 ? num_dims + 2 * so : num_dims / 2 + 2 * so;
  const int32_t row_bytes = (unpadded + p.row_alignment - 1) / p.row_alignment * p.row_alignment;
  // bytes of a row the reference touches: the last column of an int4 row with an odd column
  // count sits in the byte after the counted payload (column d reads byte d / 2)
  const int32_t touched = ty == TY_I4 ? (num_dims + 1) / 2 + 2 * so : unpadded;
  const uint8_t *base = d.placement == 3 ? p.dev_weights : p.uvm_weights;
  const int64_t limit = d.placement == 3 ? p.dev_bytes : p.uvm_bytes;
  const int64_t table_at = p.wo64 ? reinterpret_cast<const int64_t *>(p.weights_offsets)[t]
                                  : (int64_t)reinterpret_cast<const int32_t *>(p.weights_offsets)[t];
  // 16-byte chunks where the table allows them (rows at 16-byte boundaries), else 8-byte chunks.
  // A bag takes as many lanes as its rows have chunks (32 at most; wider rows take several
  // passes), not a power of two: a 132-byte row is 9 lanes, three bags to a warp.
  const uint64_t addr = reinterpret_cast<uintptr_t>(base) + (uint64_t)table_at;
  const bool wide = (addr % 16) == 0 && (row_bytes % 16) == 0;
  // rows whose touched bytes all lie inside the buffer (InterpreterNodes.cpp:6720): 0 .. max_row
  int64_t max_row = -1;
  if (table_at >= 0 && table_at + touched <= limit) max_row = (limit - touched - table_at) / row_bytes;
  if (max_row > 0x7FFFFFFEll) max_row = 0x7FFFFFFEll;
  // (a buffer that does not end on a 16-byte boundary may cut the last row's pieces short)
  const bool columns = wide && ty >= p.first_column_ty && table_at + max_row * row_bytes + (touched + 15) / 16 * 16 <= limit;
  // Words of columns per lane: four, but two of int4 rows with an fp32 result (32 fp32 sums per lane spill: 12.9
  // against 16.0 G rows/s) and of int4 rows that are no longer.
  const bool pairs = ty == TY_I4 && (!OUT16 || num_dims <= 16);
  const bool vec = wide || ((addr % 8) == 0 && (row_bytes % 8) == 0);
  const int cb = columns ? (pairs ? 8 : 16) : wide ? 16 : 8;
  const int chunks = ((columns ? touched - 2 * so : touched) + cb - 1) / cb;
  int lpr = chunks > 32 ? 32 : chunks;
  // Rows of a little more than half a warp (17 chunks: a 260-byte row) would leave the other
  // half idle: half as many lanes then walk the bag twice, one half of the row per pass, when that
  // puts over 2.4 times as many bags into the warp.
  if (chunks <= 32 && 32 / ((chunks + 1) / 2) * 5 > 32 / lpr * 12) lpr = (chunks + 1) / 2;
  const int bags_per_warp = 32 / lpr;
  const int lane = threadIdx.x & 31;
  if (lane >= bags_per_warp * lpr) return;
  const int gl = lane % lpr;
  const int64_t first = ((int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5)) * bags_per_warp + lane / lpr;
  const int64_t step = (int64_t)gridDim.x * (kThreads / 32) * bags_per_warp;
  const TableRows rows{base, limit, table_at, row_bytes, touched, num_dims, d.dim_start, t, (int32_t)max_row, gl, lpr, vec};
  int32_t flags = 0;
#define GLOWB200_POOL2(COLUMNS, TY, CW, SO32)                                                                         \
  do {                                                                                                               \
    if (p.indice_weights != nullptr) flags = pool_bags<COLUMNS, TY, CW, OUT16, true, SO32, IdxT>(p, rows, first, step); \
    else flags = pool_bags<COLUMNS, TY, CW, OUT16, false, SO32, IdxT>(p, rows, first, step);                          \
  } while (0)
#define GLOWB200_POOLQ(COLUMNS, TY, CW) \
  do { if (p.so_fp32) GLOWB200_POOL2(COLUMNS, TY, CW, true); else GLOWB200_POOL2(COLUMNS, TY, CW, false); } while (0)
  switch (ty) {
    case TY_F32: if (wide) GLOWB200_POOL2(false, TY_F32, 4, false); else GLOWB200_POOL2(false, TY_F32, 2, false); break;
    case TY_F16: if (wide) GLOWB200_POOL2(false, TY_F16, 4, false); else GLOWB200_POOL2(false, TY_F16, 2, false); break;
    case TY_I8: if (columns) GLOWB200_POOLQ(true, TY_I8, 4); else GLOWB200_POOLQ(false, TY_I8, 2); break;
    default:
      if (columns && !pairs) {
        if constexpr (OUT16) GLOWB200_POOLQ(true, TY_I4, 4);
      } else if (columns) {
        GLOWB200_POOLQ(true, TY_I4, 2);
      } else {
        GLOWB200_POOLQ(false, TY_I4, 2);
      }
      break;
  }
#undef GLOWB200_POOLQ
#undef GLOWB200_POOL2
  if (p.status != nullptr && flags != 0) atomicOr(p.status, flags);
}

}  // namespace
}  // namespace glowb200

using namespace glowb200;

extern "C" int glowb200_int_nbit_split_embedding_bags(
    void *dest, const void *dev_weights, int64_t dev_weights_bytes, const void *uvm_weights,
    int64_t uvm_weights_bytes, const int32_t *weights_placements, const void *weights_offsets,
    int weights_offsets_are_int64, const uint8_t *weights_tys, const int32_t *dim_offsets, int64_t num_tables,
    int64_t total_dims, const void *indices, const void *offsets, int indices_are_int64, int64_t num_indices,
    int64_t bags_per_table, int pooling_mode, const void *indice_weights, int indice_weights_are_fp16,
    int out_is_fp16, int scale_offset_is_fp32, int row_alignment, int32_t *status, glowb200_stream_t stream) {
  GLOWB200_REQUIRE(num_tables >= 0 && num_tables <= 65535, "num_tables must be in [0, 65535]");
  GLOWB200_REQUIRE(bags_per_table >= 0 && bags_per_table < (1ll << 31), "bags_per_table out of range");
  GLOWB200_REQUIRE(total_dims >= 0 && total_dims < (1ll << 31) && num_indices >= 0, "total_dims / num_indices out of range");
  GLOWB200_REQUIRE(pooling_mode >= 0 && pooling_mode <= 2, "pooling_mode must be 0 (sum), 1 (mean) or 2 (none)");
  GLOWB200_REQUIRE(row_alignment > 0 && row_alignment <= 4096, "row_alignment must be in [1, 4096]");
  GLOWB200_REQUIRE(dev_weights_bytes >= 0 && uvm_weights_bytes >= 0, "negative weights size");
  if (bags_per_table == 0 || total_dims == 0) return GLOWB200_OK;
  GLOWB200_REQUIRE(dest != nullptr, "dest is NULL");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (num_tables == 0) {
    GLOWB200_CUDA_OK(cudaMemsetAsync(dest, 0, (size_t)(bags_per_table * total_dims) * (out_is_fp16 ? 2 : 4), s));
    return GLOWB200_OK;
  }
  GLOWB200_REQUIRE(weights_placements != nullptr && weights_offsets != nullptr && weights_tys != nullptr &&
                       dim_offsets != nullptr && offsets != nullptr,
                   "NULL table description or offsets");
  GLOWB200_REQUIRE(num_indices == 0 || indices != nullptr, "indices is NULL");
  SplitLaunch L{};
  L.dest = dest;
  L.dev_weights = reinterpret_cast<const uint8_t *>(dev_weights);
  L.uvm_weights = reinterpret_cast<const uint8_t *>(uvm_weights);
  L.dev_bytes = dev_weights != nullptr ? dev_weights_bytes : 0;
  L.uvm_bytes = uvm_weights != nullptr ? uvm_weights_bytes : 0;
  L.placements = weights_placements;
  L.weights_offsets = weights_offsets;
  L.weights_tys = weights_tys;
  L.dim_offsets = dim_offsets;
  L.indices = indices;
  L.offsets = offsets;
  L.indice_weights = indice_weights;
  L.status = status;
  L.num_indices = num_indices;
  L.bags_per_table = bags_per_table;
  L.total_dims = total_dims;
  L.wo64 = weights_offsets_are_int64 ? 1 : 0;
  L.iw16 = indice_weights_are_fp16 ? 1 : 0;
  L.so_fp32 = scale_offset_is_fp32 ? 1 : 0;
  L.row_alignment = row_alignment;
  L.pooling_mode = pooling_mode;
  L.num_tables = (int32_t)num_tables;
  // (pool_bag_columns counts the rows of a bag in 32 bits; a long bag in pieces cost its loop 2 to 15 %)
  L.first_column_ty = num_indices <= 0x7FFFFFF0ll ? TY_I8 : TY_I4 + 1;
  // A warp takes 8 bags of rows of 4 lanes; the blocks of tables with wider rows walk on, those of narrower ones
  // are in part not needed and leave at once.  Few bags: a block for every 8, so that no row is so wide that its
  // bags would wait for one another while SMs idle (8 tables, 64 bags of 20 int8 rows of 128 columns: 17 -> 12 us).
  int64_t blocks = (bags_per_table + 7) / 8;
  if (blocks * num_tables > 2048) blocks = (bags_per_table + 31) / 32;
  const dim3 grid((unsigned)blocks, (unsigned)num_tables + (num_tables < 65535 ? 1 : 0));
  if (num_tables == 65535)  // no block row left for the columns without a table
    GLOWB200_CUDA_OK(cudaMemsetAsync(dest, 0, (size_t)(bags_per_table * total_dims) * (out_is_fp16 ? 2 : 4), s));
  if (out_is_fp16)
    GLOWB200_CUDA_OK(indices_are_int64 ? launch_pdl(split_embedding_bags_kernel<true, int64_t>, grid, kThreads, 0, s, L)
                                       : launch_pdl(split_embedding_bags_kernel<true, int32_t>, grid, kThreads, 0, s, L));
  else
    GLOWB200_CUDA_OK(indices_are_int64 ? launch_pdl(split_embedding_bags_kernel<false, int64_t>, grid, kThreads, 0, s, L)
                                       : launch_pdl(split_embedding_bags_kernel<false, int32_t>, grid, kThreads, 0, s, L));
  GLOWB200_CUDA_OK(cudaGetLastError());
  return GLOWB200_OK;
}
