// DLRM feature interaction: for every sample, the dot products of all pairs among the bottom-MLP
// output and the pooled embedding vectors, concatenated behind the bottom-MLP output.
//
// The reference builds this from generic nodes -- Concat, Reshape to [B, n, D], BatchMatMul with
// its own transpose, then a flatten (tests/unittests/RecommendationSystemTest.cpp:640-680) -- and
// has no kernel of its own for it.  The benchmark's model keeps only the strictly-lower triangle
// of the n x n product (n = tables + 1, pairs (i, j) with j < i in row-major order, the DLRM
// convention): out[b] = [ v_0 (D values) | v_1.v_0 | v_2.v_0 | v_2.v_1 | v_3.v_0 | ... ].
// One block per sample keeps the n vectors in shared memory; a dot product is a sequential fp32
// FMA chain over the D components.  The result can be written as fp32 or already quantized to
// int8 (Quantize fused: nearbyintf(x / scale + offset), clipped).
#include "common.cuh"

namespace glowb200 {
namespace {

__global__ void __launch_bounds__(256) pairwise_dot_kernel(const float *__restrict__ dense, int64_t ld_dense,
                                                           const float *__restrict__ pooled, int64_t ld_pooled, int tables,
                                                           int D, float *__restrict__ out_f, int8_t *__restrict__ out_q,
                                                           int64_t ld_out, float q_scale, int32_t q_offset) {
  pdl_wait();               // (launched as a programmatic dependent of the pooling kernel)
  pdl_launch_dependents();  // a contraction that follows may set up now (it waits for this kernel before its loads)
  extern __shared__ float v[];  // [n][D + 1]
  const int n = tables + 1, pitch = D + 1;
  const int64_t b = blockIdx.x;
  for (int i = threadIdx.x; i < n * D; i += blockDim.x) {
    const int r = i / D, k = i - r * D;
    v[r * pitch + k] = r == 0 ? dense[b * ld_dense + k] : pooled[b * ld_pooled + (int64_t)(r - 1) * D + k];
  }
  __syncthreads();
  auto emit = [&](int64_t col, float x) {
    if (out_q) {
      const float t = __fadd_rn(__fdiv_rn(x, q_scale), (float)q_offset);
      const float c = fminf(fmaxf(nearbyintf(t), -2147483648.0f), 2147483520.0f);
      out_q[b * ld_out + col] = (int8_t)clip_i8((int32_t)c);
    } else {
      out_f[b * ld_out + col] = x;
    }
  };
  for (int k = threadIdx.x; k < D; k += blockDim.x) emit(k, v[k]);
  const int pairs = n * (n - 1) / 2;
  for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
    // p -> (i, j), j < i, row-major over the strictly-lower triangle
    int i = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)p)) * 0.5f);
    while (i * (i - 1) / 2 > p) i--;
    while ((i + 1) * i / 2 <= p) i++;
    const int j = p - i * (i - 1) / 2;
    const float *a = v + i * pitch, *c = v + j * pitch;
    float acc = 0.0f;
    for (int k = 0; k < D; k++) acc = fmaf(a[k], c[k], acc);
    emit(D + p, acc);
  }
}

// The same result from R x R register tiles (D a multiple of 4): a thread owns the dots of rows
// bi + r*nb against rows bj + s*nb (r, s < R, nb = ceil(n / R), bj <= bi) and walks k four at a time with 16-byte
// shared-memory loads -- with R = 4, 8 loads feed 64 FMAs instead of 2 loads per FMA, which is what bounded
// the kernel above.  Every dot still is the sequential FMA chain over k = 0..D-1, so the bits are
// the same.  Rows are padded by 4 floats (D + 4, an odd number of 16-byte units for D a multiple of 8) so that
// the neighbouring rows a warp reads fall into different banks.
// What bounds it, for many vectors, is the copying and the sums in turn: 45 us of one and 67 of the other for 4096 samples of
// 65 x 128, where a multiply-add of three registers takes a scheduler 1.5 to 1.9 clocks.  Vectors come by asynchronous
// copies, without a register on the way (133 -> 114 us), and more blocks fit an SM when they are smaller
// (108).  Not better: 8 x 4 tiles over a transposed copy with packed multiply-adds (138), 6 x 6, 7 x 7 and 8 x 8 tiles of
// several samples to a block (124 - 146), two buffers and a block that goes on (122 - 136).
// Few vectors have few tiles -- 28 of 4 x 4 for 27
// vectors, the rest of the block idle -- and go in 2 x 2 tiles with no more warps than those fill: 128 samples of
// 27 x 64 5.4 -> 3.3 us, 4096 samples 35 -> 21, 2048 of 17 x 32 15.0 -> 5.4.
// The quantized result takes the reciprocal of its scale; next to a tie, and for offsets far outside int8, the division decides.
template <int R, int THREADS, int BLOCKS>
__global__ void __launch_bounds__(THREADS, BLOCKS) pairwise_dot_tiled_kernel(const float *__restrict__ dense, int64_t ld_dense,
                                                                             const float *__restrict__ pooled, int64_t ld_pooled,
                                                                             int tables, int D, float *__restrict__ out_f,
                                                                             int8_t *__restrict__ out_q, int64_t ld_out, float q_scale,
                                                                             int32_t q_offset, float limit, int vec_in) {
  pdl_wait();               // (launched as a programmatic dependent of the pooling kernel)
  pdl_launch_dependents();  // a contraction that follows may set up now (it waits for this kernel before its loads)
  extern __shared__ __align__(16) float v[];  // [R * ceil(n / R)][D + 4]; rows beyond n are zero
  const int n = tables + 1, pitch = D + 4, nb = (n + R - 1) / R;
  const int64_t b = blockIdx.x;
  if (vec_in) {
    const int q = D >> 2;
    for (int i = threadIdx.x; i < nb * R * q; i += blockDim.x) {
      const int r = i / q, k = (i - r * q) * 4;
      if (r >= n)
        *reinterpret_cast<float4 *>(v + r * pitch + k) = make_float4(0.f, 0.f, 0.f, 0.f);
      else
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(v + r * pitch + k)),
                     "l"(r == 0 ? dense + b * ld_dense + k : pooled + b * ld_pooled + (int64_t)(r - 1) * D + k)
                     : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    for (int i = threadIdx.x; i < nb * R * D; i += blockDim.x) {
      const int r = i / D, k = i - r * D;
      v[r * pitch + k] = r >= n ? 0.0f : (r == 0 ? dense[b * ld_dense + k] : pooled[b * ld_pooled + (int64_t)(r - 1) * D + k]);
    }
  }
  __syncthreads();
  const float inverse = __fdiv_rn(1.0f, q_scale), shift = (float)q_offset;
  auto emit = [&](int64_t col, float x) {
    if (out_q) {
      bool sure = true;
      int32_t q = quantize_by_reciprocal(x, inverse, shift, limit, sure);
      if (!sure) q = (int32_t)fminf(fmaxf(nearbyintf(__fadd_rn(__fdiv_rn(x, q_scale), shift)), -2147483648.0f), 2147483520.0f);
      out_q[b * ld_out + col] = (int8_t)clip_i8(q);
    } else {
      out_f[b * ld_out + col] = x;
    }
  };
  for (int k = threadIdx.x; k < D; k += blockDim.x) emit(k, v[k]);
  const int tiles = nb * (nb + 1) / 2;
  for (int t = threadIdx.x; t < tiles; t += blockDim.x) {
    // t -> (bi, bj), bj <= bi, row-major over the lower triangle of tiles
    int bi = (int)((sqrtf(1.0f + 8.0f * (float)t) - 1.0f) * 0.5f);
    while (bi * (bi + 1) / 2 > t) bi--;
    while ((bi + 1) * (bi + 2) / 2 <= t) bi++;
    const int bj = t - bi * (bi + 1) / 2;
    // the tile's rows are bi + r*nb against bj + s*nb (strided, not adjacent): neighbouring
    // threads then read neighbouring rows, which the odd pitch / 4 spreads over all banks
    const float *a = v + bi * pitch, *c = v + bj * pitch;
    const int tile_step = nb * pitch;
    float acc[R][R];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int s = 0; s < R; s++) acc[r][s] = 0.0f;
    for (int k = 0; k < D; k += 4) {
      float4 x[R], y[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        x[r] = *reinterpret_cast<const float4 *>(a + r * tile_step + k);
        y[r] = *reinterpret_cast<const float4 *>(c + r * tile_step + k);
      }
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int s = 0; s < R; s++) {
          acc[r][s] = fmaf(x[r].x, y[s].x, acc[r][s]);
          acc[r][s] = fmaf(x[r].y, y[s].y, acc[r][s]);
          acc[r][s] = fmaf(x[r].z, y[s].z, acc[r][s]);
          acc[r][s] = fmaf(x[r].w, y[s].w, acc[r][s]);
        }
    }
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int s = 0; s < R; s++) {
        // a dot product is symmetric: the tile of two different residue classes holds every
        // pair between them once; the diagonal tile holds each pair twice and keeps one
        const int i = bi + r * nb, j = bj + s * nb;
        const int hi = i > j ? i : j, lo = i > j ? j : i;
        if (hi < n && lo < hi && (bi != bj || i > j)) emit(D + hi * (hi - 1) / 2 + lo, acc[r][s]);
      }
  }
}

}  // namespace
}  // namespace glowb200

using namespace glowb200;

extern "C" int glowb200_pairwise_dot_interaction(const float *dense, int64_t ld_dense, const float *pooled,
                                                 int64_t ld_pooled, int64_t batch, int64_t tables, int64_t dim,
                                                 float *out_f32, int8_t *out_i8, int64_t ld_out, float quant_scale,
                                                 int32_t quant_offset, glowb200_stream_t stream) {
  GLOWB200_REQUIRE(batch >= 0 && tables >= 0 && dim > 0 && tables < 4096 && dim <= 4096 && batch < (1ll << 31),
                   "bad sizes");
  if (batch == 0) return GLOWB200_OK;
  GLOWB200_REQUIRE(dense && (tables == 0 || pooled) && ((out_f32 != nullptr) != (out_i8 != nullptr)),
                   "need dense, pooled and exactly one of the two outputs");
  const int64_t n = tables + 1, width = dim + n * (n - 1) / 2;
  GLOWB200_REQUIRE(ld_out >= width && ld_dense >= dim && ld_pooled >= tables * dim, "row pitch smaller than the row");
  cudaStream_t cs = reinterpret_cast<cudaStream_t>(stream);
  auto tiles_of = [&](int64_t r) { return ((n + r - 1) / r) * ((n + r - 1) / r + 1) / 2; };
  const int R = tiles_of(4) >= 80 ? 4 : 2;  // (66 tiles -- 41 vectors -- still gain from the smaller ones)
  const size_t tiled_smem = (size_t)((n + R - 1) / R * R) * (dim + 4) * sizeof(float);
  if ((dim % 4) == 0 && tiled_smem <= 200 * 1024) {
    const int64_t warps = (tiles_of(R) + 31) / 32;
    const int vec_in = (reinterpret_cast<uintptr_t>(dense) % 16 == 0) && (ld_dense % 4 == 0) &&
                       (tables == 0 || (reinterpret_cast<uintptr_t>(pooled) % 16 == 0 && ld_pooled % 4 == 0));
    // Blocks of 160 threads once six of them to an SM -- where its shared memory holds six -- fill it more than twice (4096 samples of
    // 65 x 128: 108 us against 114; of 49 x 64 51 against 53; 16,384 of 57 x 96 270 against 296); fewer samples are copied and summed faster by
    // larger ones (512 samples: 18.4 against 27), and so are vectors of which fewer blocks fit (4096 of 65 x 160 143 us against 154, of
    // 65 x 256 239 against 249).
    const bool many = R == 4 && tiles_of(4) <= 160 && batch >= 2 * 6 * (int64_t)sm_count() && 6 * (tiled_smem + 1024) <= 228 * 1024;
    auto kernel = many ? pairwise_dot_tiled_kernel<4, 160, 6> : R == 4 ? pairwise_dot_tiled_kernel<4, 256, 4> : pairwise_dot_tiled_kernel<2, 256, 4>;
    const unsigned threads = many ? 160 : R == 4 ? 256 : 32 * (unsigned)(warps < 2 ? 2 : warps > 8 ? 8 : warps);
    if (tiled_smem > 48 * 1024)
      GLOWB200_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tiled_smem));
    GLOWB200_CUDA_OK(launch_pdl(kernel, (unsigned)batch, threads, tiled_smem, cs, dense, ld_dense, pooled, ld_pooled,
                                (int)tables, (int)dim, out_f32, out_i8, ld_out, quant_scale, quant_offset, reciprocal_limit(quant_offset), vec_in));
    return GLOWB200_OK;
  }
  const size_t smem = (size_t)n * (dim + 1) * sizeof(float);
  GLOWB200_REQUIRE(smem <= 200 * 1024, "tables x dim too large for one block's shared memory");
  if (smem > 48 * 1024)
    GLOWB200_CUDA_OK(cudaFuncSetAttribute(pairwise_dot_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GLOWB200_CUDA_OK(launch_pdl(pairwise_dot_kernel, (unsigned)batch, 256, smem, reinterpret_cast<cudaStream_t>(stream), dense, ld_dense,
                              pooled, ld_pooled, (int)tables, (int)dim, out_f32, out_i8, ld_out, quant_scale, quant_offset));
  return GLOWB200_OK;
}
