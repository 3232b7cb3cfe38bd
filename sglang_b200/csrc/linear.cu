// The whole block-FP8 linear and the whole fused expert layer behind one C call each: the caller allocates the output
// and one workspace, everything in between -- activation codes and scales, split-K partial sums, routing tables,
// expert intermediates -- is laid out in that workspace here and enqueued on the caller's stream.  A decode-size layer
// is a few microseconds of device work per kernel, so what bounds it is the host: one call replaces a Python-level
// allocation, argument check and foreign call per kernel.
#include <algorithm>

#include "gemm_common.cuh"

namespace b200 {

// moe_glue.cu: weighted un-permute sum with fp32 routing weights, each rounded to `dtype` first (what the separate
// conversion pass stored)
int unpermute_sum_f32_factors(const void* input, void* output, const int32_t* permutation, const float* factors, int64_t m,
                              int64_t topk, int64_t row_len, int dtype, cudaStream_t stream);
// quant.cu: every token quantised once, codes and scales stored to the rows of its experts
int quant_to_rows(const void* x, int dtype, const int32_t* row_of, int topk, void* q, void* s, int64_t M, int64_t K,
                  int64_t s_ld, bool ue8m0, cudaStream_t stream);

namespace {

constexpr float kFp8Max = 448.0f;
constexpr float kQuantEps = 1e-10f;

inline size_t align_up(size_t v) { return (v + 255) & ~size_t(255); }
inline int64_t align4(int64_t v) { return (v + 3) / 4 * 4; }

// Bump allocation over the caller's workspace; with a null base it only counts.
struct Arena {
  uint8_t* base;
  size_t used = 0;
  explicit Arena(void* p) : base(static_cast<uint8_t*>(p)) {}
  template <typename T = uint8_t>
  T* take(size_t count) {
    T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
    used += align_up(count * sizeof(T));
    return p;
  }
};

// out[m, n] = T(float(out[m, n]) + float(bias[n])): the bias is added to the rounded product, as `out += bias` does.
template <typename T>
__global__ void __launch_bounds__(256) bias_add_kernel(T* __restrict__ out, const T* __restrict__ bias, int64_t M, int N,
                                                       int64_t ldo) {
  pdl_start();
  const int n2 = N >> 1;
  const int64_t total = M * n2;
  for (int64_t i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
    const int64_t m = i / n2;
    const int n = static_cast<int>(i - m * n2) * 2;
    T* dst = out + m * ldo + n;
    dst[0] = static_cast<T>(static_cast<float>(dst[0]) + static_cast<float>(bias[n]));
    dst[1] = static_cast<T>(static_cast<float>(dst[1]) + static_cast<float>(bias[n + 1]));
  }
}

int bias_add(void* out, const void* bias, int64_t M, int64_t N, int64_t ldo, int dtype, cudaStream_t st) {
  if (N % 2 != 0) return B200_ERR_BAD_SHAPE;
  const int64_t blocks = std::min<int64_t>((M * (N / 2) + 255) / 256, 16LL * sm_count());
  if (dtype == B200_DT_BF16)
    launch_pdl(bias_add_kernel<__nv_bfloat16>, static_cast<unsigned>(blocks), 256, 0, st, static_cast<__nv_bfloat16*>(out),
               static_cast<const __nv_bfloat16*>(bias), M, static_cast<int>(N), ldo);
  else
    launch_pdl(bias_add_kernel<__half>, static_cast<unsigned>(blocks), 256, 0, st, static_cast<__half*>(out),
               static_cast<const __half*>(bias), M, static_cast<int>(N), ldo);
  B200_CUDA_TRY(cudaGetLastError());
  return B200_OK;
}

struct LinearPlan {
  uint8_t* q;
  void* s;
  int64_t s_ld;        // column-major scales: stride between k-groups (fp32) or packed words
  void* partial;
  size_t partial_bytes;
};
LinearPlan plan_linear(Arena& a, int64_t M, int64_t N, int64_t K, int scale_mode) {
  const bool ue8m0 = scale_mode != 0;
  LinearPlan p;
  const int64_t groups = K / 128;
  p.q = a.take<uint8_t>(static_cast<size_t>(M) * K);
  p.s_ld = align4(M);
  p.s = a.take<uint32_t>(static_cast<size_t>(p.s_ld) * (ue8m0 ? (groups + 3) / 4 : groups));
  p.partial_bytes = scale_mode != 2 || packed_promotes(M, N, K) ? b200_fp8_blockwise_scaled_mm_workspace_bytes(M, N, K) : 0;
  p.partial = p.partial_bytes ? a.take<uint8_t>(p.partial_bytes) : nullptr;
  return p;
}

}  // namespace
}  // namespace b200

extern "C" size_t b200_fp8_linear_workspace_bytes(int64_t M, int64_t N, int64_t K, int scale_mode) {
  using namespace b200;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  Arena a(nullptr);
  plan_linear(a, M, N, K, scale_mode);
  return a.used;
}

extern "C" int b200_fp8_linear(const void* x, int dtype, const void* w, int64_t ldw, const float* ws, int64_t ws_stride_n,
                               int64_t ws_stride_g, const void* bias, void* out, int64_t ldo, int64_t M, int64_t N,
                               int64_t K, int scale_mode, void* workspace, size_t workspace_bytes, void* stream) {
  using namespace b200;
  if (M < 0 || N <= 0 || K <= 0 || K % 128 != 0) return B200_ERR_BAD_SHAPE;
  if (M == 0) return B200_OK;
  if (dtype != B200_DT_BF16 && dtype != B200_DT_F16) return B200_ERR_BAD_DTYPE;
  if (!x || !w || !ws || !out || !workspace) return B200_ERR_NULL_PTR;
  if (!aligned16(workspace)) return B200_ERR_MISALIGNED;
  if (scale_mode < 0 || scale_mode > 2) return B200_ERR_UNSUPPORTED;
  Arena a(workspace);
  const LinearPlan p = plan_linear(a, M, N, K, scale_mode);
  if (workspace_bytes < a.used) return B200_ERR_TOO_LARGE;
  int rc;
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (scale_mode == 0)
    rc = b200_per_token_group_quant_fp8(x, dtype, p.q, static_cast<float*>(p.s), M, K, 128, 1, p.s_ld, kQuantEps, -kFp8Max,
                                        kFp8Max, stream);
  else
    rc = b200_per_token_group_quant_fp8_ue8m0(x, dtype, p.q, static_cast<uint32_t*>(p.s), M, K, p.s_ld, kQuantEps, -kFp8Max,
                                              kFp8Max, stream);
  if (rc != B200_OK) return rc;
  if (scale_mode == 2 && !packed_promotes(M, N, K)) {
    rc = b200_fp8_blockwise_scaled_mm_pow2(p.q, K, w, ldw, static_cast<uint32_t*>(p.s), 1, p.s_ld, ws, ws_stride_n,
                                           ws_stride_g, out, ldo, dtype, M, N, K, stream);
    return rc == B200_OK && bias ? bias_add(out, bias, M, N, ldo, dtype, st) : rc;
  }
  // the kernel before is the quantiser launched above: weights may be fetched while it runs
  return dense_mm(p.q, K, w, ldw, static_cast<const float*>(p.s), 1, p.s_ld, ws, ws_stride_n, ws_stride_g, out, ldo, dtype,
                  M, N, K, 0, p.partial, p.partial_bytes, stream, scale_mode != 0, bias, 1);
}

namespace b200 {
namespace {

struct ExpertPlan {
  int32_t *offsets, *ps1, *ps2, *a_map, *c_map;
  uint8_t* prep_scratch;
  size_t prep_bytes;
  uint8_t *rep_q, *inter_q, *c1, *c2;
  uint32_t *rep_s, *inter_s;           // fp32 scales or packed exponent words
};

ExpertPlan plan_experts(Arena& a, int64_t m, int64_t k, int64_t n, int topk, int E, bool ue8m0) {
  ExpertPlan p;
  const int64_t R = m * topk, gk = k / 128, gn = n / 128;
  p.offsets = a.take<int32_t>(E + 1);
  p.ps1 = a.take<int32_t>(3 * E);
  p.ps2 = a.take<int32_t>(3 * E);
  p.a_map = a.take<int32_t>(R);
  p.c_map = a.take<int32_t>(R);
  p.prep_bytes = b200_moe_prepare_scratch_bytes(R, E);
  p.prep_scratch = a.take(p.prep_bytes);
  p.rep_q = a.take(R * k);
  p.inter_q = a.take(R * n);
  if (ue8m0) {
    p.rep_s = a.take<uint32_t>(align4(R) * ((gk + 3) / 4));
    p.inter_s = a.take<uint32_t>(align4(R) * ((gn + 3) / 4));
    p.c1 = nullptr;
  } else {
    p.rep_s = a.take<uint32_t>(R * gk);
    p.inter_s = a.take<uint32_t>(R * gn);
    p.c1 = a.take(2 * R * 2 * n);
  }
  p.c2 = a.take(2 * R * k);
  return p;
}

}  // namespace
}  // namespace b200

extern "C" size_t b200_fused_experts_fp8_workspace_bytes(int64_t m, int64_t k, int64_t n, int topk, int num_experts,
                                                         int scale_ue8m0) {
  using namespace b200;
  if (m <= 0 || k <= 0 || n <= 0 || topk <= 0 || num_experts <= 0) return 0;
  Arena a(nullptr);
  plan_experts(a, m, k, n, topk, num_experts, scale_ue8m0 != 0);
  return a.used;
}

extern "C" int b200_fused_experts_fp8(const void* x, int dtype, const void* w13, const void* w2, const float* w13_scale,
                                      const float* w2_scale, const float* topk_weights, const int32_t* topk_ids,
                                      int64_t m, int64_t k, int64_t n, int topk, int num_experts, int32_t* expert_offsets,
                                      int32_t* problem_sizes1, int32_t* problem_sizes2, void* out, int scale_ue8m0,
                                      void* workspace, size_t workspace_bytes, void* stream) {
  using namespace b200;
  if (m < 0 || k <= 0 || n <= 0 || topk <= 0 || num_experts <= 0 || k % 128 != 0 || n % 128 != 0)
    return B200_ERR_BAD_SHAPE;
  if (m == 0) return B200_OK;
  if (dtype != B200_DT_BF16 && dtype != B200_DT_F16) return B200_ERR_BAD_DTYPE;
  if (!x || !w13 || !w2 || !w13_scale || !w2_scale || !topk_weights || !topk_ids || !out || !workspace)
    return B200_ERR_NULL_PTR;
  if (!aligned16(workspace)) return B200_ERR_MISALIGNED;
  Arena a(workspace);
  ExpertPlan p = plan_experts(a, m, k, n, topk, num_experts, scale_ue8m0 != 0);
  if (workspace_bytes < a.used) return B200_ERR_TOO_LARGE;
  if (expert_offsets) p.offsets = expert_offsets;
  if (problem_sizes1) p.ps1 = problem_sizes1;
  if (problem_sizes2) p.ps2 = problem_sizes2;
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t R = m * topk, gk = k / 128, gn = n / 128;
  const int E = num_experts;
  int rc = b200_moe_prepare(topk_ids, m, topk, E, static_cast<int>(n), static_cast<int>(k), p.offsets, nullptr, p.ps1,
                            p.ps2, p.a_map, p.c_map, p.prep_scratch, p.prep_bytes, stream);
  if (rc != B200_OK) return rc;
  if (scale_ue8m0) {
    const int64_t ld_r = align4(R);
    const int wn = static_cast<int>((gn + 3) / 4);
    rc = quant_to_rows(x, dtype, p.c_map, topk, p.rep_q, p.rep_s, m, k, ld_r, true, st);
    if (rc != B200_OK) return rc;
    if (gn % 4 != 0) B200_CUDA_TRY(cudaMemsetAsync(p.inter_s + (wn - 1) * ld_r, 0, ld_r * sizeof(uint32_t), st));
    rc = b200_fp8_blockwise_scaled_grouped_mm_pow2_silu_quant(
        p.rep_q, k, R, w13, k, p.rep_s, 1, ld_r, -1, w13_scale, 2 * gn * gk, gk, 1, p.inter_q, n, p.inter_s, ld_r, dtype,
        p.offsets, p.ps1, 3, nullptr, E, E, n, k, stream);
    if (rc == B200_OK)
      rc = b200_fp8_blockwise_scaled_grouped_mm_pow2(p.inter_q, n, R, w2, n, p.inter_s, 1, ld_r, -1, w2_scale, gk * gn, gn,
                                                     1, p.c2, k, dtype, p.offsets, p.ps1, 3, nullptr, E, E, k, n, stream);
  } else {
    float* inter_s = reinterpret_cast<float*>(p.inter_s);
    rc = quant_to_rows(x, dtype, p.c_map, topk, p.rep_q, p.rep_s, m, k, 0, false, st);
    if (rc == B200_OK)
      rc = b200_fp8_blockwise_scaled_grouped_mm(p.rep_q, k, w13, k, reinterpret_cast<float*>(p.rep_s), gk, 1, w13_scale,
                                                2 * gn * gk, gk, 1, p.c1, 2 * n, dtype, p.offsets, p.ps1, E, R, 2 * n, k,
                                                stream);
    if (rc == B200_OK)
      rc = b200_silu_mul_per_token_group_quant_fp8(p.c1, dtype, p.inter_q, inter_s, R, n, gn, 1, kQuantEps, -kFp8Max,
                                                   kFp8Max, stream);
    if (rc == B200_OK)
      rc = b200_fp8_blockwise_scaled_grouped_mm(p.inter_q, n, w2, n, inter_s, gn, 1, w2_scale, gk * gn, gn, 1, p.c2, k,
                                                dtype, p.offsets, p.ps2, E, R, k, n, stream);
  }
  if (rc != B200_OK) return rc;
  return unpermute_sum_f32_factors(p.c2, out, p.c_map, topk_weights, m, topk, k, dtype, st);
}
