// Pieces shared by the block-FP8 GEMM kernels: parameter block, output-row stores, tensor-map
// construction and the device status word.
#pragma once
#include "common.cuh"

namespace b200 {

struct GemmParams {
  const float* sa;
  const float* sb;
  void* out;
  int64_t sa_stride_m, sa_stride_g, sb_stride_n, sb_stride_g, ldo;
  int M, N, K;
  int out_dtype;
  int* status;
  // grouped (per-expert) form only: rows [expert_offsets[e], +problem_sizes[3e]) of A/out belong to
  // expert e, whose weights are rows [e*N, (e+1)*N) of B and whose weight scales start at sb + e*sb_stride_e
  const int32_t* expert_offsets;
  const int32_t* problem_sizes;
  int64_t sb_stride_e;
  int num_experts;
  // split-K form (dense, small M): the k-blocks of a tile are divided among split_k CTAs, each writing
  // fp32 partial sums to partial[split][M][N]; a second kernel adds them in split order
  int split_k;
  int kb_per_split;
  float* partial;
  // tail split (dense, 128-row-tile kernel): tiles [0, tail_first) are whole; each tile from tail_first on -- the ones
  // that would form a mostly empty last wave -- is divided among split_k CTAs.  partial_tiles != 0: partial sums are
  // whole tiles, partial[(tile - tail_first) * split_k + split][128][tile_n]
  int tail_first;
  int partial_tiles;
  const void* bias; // [N] in the output type, added to the rounded product; or nullptr
  int prefetch_w;   // != 0: the kernel before this one in the stream is this library's own and triggered after its wait, so
                    // weights may be fetched ahead of the wait
  int tile_n;       // tile width of the 128-row-tile kernel, 128 or 256
  // activation scales given as packed UE8M0 exponent bytes (four k-blocks per 32-bit word) instead of fp32:
  // element (m, kb) is byte kb % 4 of the word at sa[(kb / 4) * sa_stride_g + m * sa_stride_m]
  int sa_ue8m0;
};


// A fresh slot of the current device's status ring for one launch, or nullptr on error.
int* gemm_status_ptr();
// The device's sticky error code as mirrored in pinned host memory (0 = none); no synchronisation.
int gemm_sticky_status();
// 2-D tensor map over a row-major [rows, cols] byte matrix with leading dimension ld, box =
// box_rows x 128 bytes, 128-byte swizzle, zero fill outside the matrix.
int make_map_u8_2d(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int64_t ld, int box_rows);

// The dense fp32-promotion GEMM behind the C entry points (gemm.cu).  split_k 0: the library's own schedule, as far as the
// workspace allows; sa_ue8m0: packed exponent activation scales; bias and prefetch_w as in GemmParams.
int dense_mm(const void* a, int64_t lda, const void* b, int64_t ldb, const float* sa, int64_t sa_stride_m,
             int64_t sa_stride_g, const float* sb, int64_t sb_stride_n, int64_t sb_stride_g, void* out, int64_t ldo,
             int out_dtype, int64_t M, int64_t N, int64_t K, int split_k, void* workspace, size_t workspace_bytes,
             void* stream, int sa_ue8m0, const void* bias, int prefetch_w);

// Whether a linear with power-of-two scales on both sides runs on dense_mm rather than the block-scaling kernel.
bool packed_promotes(int64_t M, int64_t N, int64_t K);

#if defined(__CUDACC__)
// Row-tile prefix table of the grouped form, by the whole CTA: per-expert counts, then a warp's running sum.
__device__ __forceinline__ void build_tile_table(int* tile_start, const int32_t* problem_sizes, int num_experts, int tile_rows) {
  for (int e = threadIdx.x; e < num_experts; e += blockDim.x)
    tile_start[e + 1] = (max(problem_sizes[e * 3], 0) + tile_rows - 1) / tile_rows;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int carry = 0;
    for (int base = 0; base < num_experts; base += 32) {
      int v = (base + lane < num_experts) ? tile_start[base + lane + 1] : 0;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= off) v += u;
      }
      if (base + lane < num_experts) tile_start[base + lane + 1] = carry + v;
      carry += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) tile_start[0] = 0;
  }
  __syncthreads();
}

// Activation scale of (row, k-block), fp32 or packed UE8M0.  The representation is a template argument so
// that a stager's batch of loads stays a straight line of independent loads: with a run-time test inside
// every load the compiler serialised them and the stager fell behind the tensor pipe.
template <bool UE8M0>
__device__ __forceinline__ float load_sa(const GemmParams& p, int64_t row, int kb) {
  if constexpr (UE8M0) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(p.sa);
    const uint32_t word = __ldg(w + static_cast<int64_t>(kb >> 2) * p.sa_stride_g + row * p.sa_stride_m);
    return __uint_as_float(((word >> (8 * (kb & 3))) & 0xffu) << 23);   // 2 ** (byte - 127); byte 0 -> 0
  } else {
    return __ldg(p.sa + row * p.sa_stride_m + static_cast<int64_t>(kb) * p.sa_stride_g);
  }
}

__device__ __forceinline__ uint32_t pack2(__nv_bfloat16*, float a, float b) {
  __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&t);
}
__device__ __forceinline__ uint32_t pack2(__half*, float a, float b) {
  __half2 t = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&t);
}
__device__ __forceinline__ __nv_bfloat16 cvt1(__nv_bfloat16*, float a) { return __float2bfloat16_rn(a); }
__device__ __forceinline__ __half cvt1(__half*, float a) { return __float2half_rn(a); }
__device__ __forceinline__ float cvt1(float*, float a) { return a; }

// 32 bytes to a 32-byte-aligned address in one store: a warp that writes one row per lane then fills whole sectors.
__device__ __forceinline__ void st_global_32(void* dst, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// Store NCOLS consecutive outputs of one row; `valid` = columns left before N.
template <int NCOLS, typename OutT>
__device__ __forceinline__ void store_row(OutT* dst, const float (&acc)[NCOLS], int valid, bool vec_ok) {
  if (vec_ok && valid >= NCOLS) {
#pragma unroll
    for (int c = 0; c < NCOLS; c += 8) {
      uint4 v;
      v.x = pack2(dst, acc[c + 0], acc[c + 1]);
      v.y = pack2(dst, acc[c + 2], acc[c + 3]);
      v.z = pack2(dst, acc[c + 4], acc[c + 5]);
      v.w = pack2(dst, acc[c + 6], acc[c + 7]);
      *reinterpret_cast<uint4*>(dst + c) = v;
    }
  } else {
#pragma unroll
    for (int c = 0; c < NCOLS; ++c)
      if (c < valid) dst[c] = cvt1(dst, acc[c]);
  }
}
template <int NCOLS>
__device__ __forceinline__ void store_row(float* dst, const float (&acc)[NCOLS], int valid, bool vec_ok) {
  if (vec_ok && valid >= NCOLS) {
#pragma unroll
    for (int c = 0; c < NCOLS; c += 4)
      *reinterpret_cast<float4*>(dst + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
  } else {
#pragma unroll
    for (int c = 0; c < NCOLS; ++c)
      if (c < valid) dst[c] = acc[c];
  }
}

// One thread's row segment of the output, `cols` of NCOLS columns from (m, n0) on, 16 columns at a time: 32-byte stores
// where the row allows them (full sectors: 60 cycles per k-block of a 128 x 256 tile less than 16-byte ones).  The bias
// is added to the value rounded to the output type, as `out += bias` does.
template <int NCOLS, typename OutT>
__device__ __forceinline__ void store_out(OutT* out, const OutT* bias, int64_t m, int n0, int64_t ldo, float (&acc)[NCOLS], int cols) {
  OutT* dst = out + m * ldo + n0;
  if (bias != nullptr) {
#pragma unroll
    for (int c = 0; c < NCOLS; ++c)
      if (c < cols) acc[c] = static_cast<float>(cvt1(dst, acc[c])) + static_cast<float>(bias[n0 + c]);
  }
  const bool vec16 = ((ldo * sizeof(OutT)) & 15) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  const bool vec32 = ((ldo * sizeof(OutT)) & 31) == 0 && (reinterpret_cast<uintptr_t>(out) & 31u) == 0;
#pragma unroll
  for (int c = 0; c < NCOLS; c += 16) {
    if (c >= cols) break;
    if constexpr (sizeof(OutT) == 2) {
      if (vec32 && cols - c >= 16) {
        uint32_t v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = pack2(dst, acc[c + 2 * i], acc[c + 2 * i + 1]);
        st_global_32(dst + c, v);
        continue;
      }
    }
    store_row<16>(dst + c, reinterpret_cast<const float(&)[16]>(acc[c]), cols - c, vec16);
  }
}

#endif  // __CUDACC__

}  // namespace b200
