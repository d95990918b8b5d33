// Entry of the dequantizing GEMM (kernel: hq_dq_gemm.cuh, plan and launch: hq_dq_launch.cuh, instances:
// hq_dq_gemm_*.cu) and the scale tables its block-FP8 form reads.
#include "hq_common.cuh"
#include "hq_kernels.h"

namespace hq {

// ---- block-FP8 scale preparation (once per layer) -------------------------------------
// scales [groups = E*NB][KB] -> tile_scale[group] = max_kb scale, rel_scale[group][kb] = scale / tile_scale.
__global__ void __launch_bounds__(128) fp8_scale_prepare_kernel(const float* __restrict__ scales, int64_t n_groups,
                                                                int kb, float* __restrict__ tile_scale,
                                                                float* __restrict__ rel_scale) {
  const int64_t grp = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (grp >= n_groups) return;
  const int lane = threadIdx.x & 31;
  float m = 0.f;
  for (int i = lane; i < kb; i += 32) m = fmaxf(m, scales[grp * kb + i]);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
  if (lane == 0) tile_scale[grp] = m;
  for (int i = lane; i < kb; i += 32) rel_scale[grp * kb + i] = m > 0.f ? scales[grp * kb + i] / m : 0.f;
}

int32_t launch_fp8_scale_prepare(const float* scales, int64_t n_groups, int kb, float* tile_scale, float* rel_scale,
                                 cudaStream_t stream) {
  if (n_groups == 0) return HQ_OK;
  fp8_scale_prepare_kernel<<<(unsigned)((n_groups + 3) / 4), 128, 0, stream>>>(scales, n_groups, kb, tile_scale,
                                                                             rel_scale);
  return cudaGetLastError() == cudaSuccess ? HQ_OK : HQ_ERR_CUDA;
}

bool grouped_gemm_supported(int format, int64_t n, int64_t k) {
  if (format < HQ_FMT_Q8_0 || format > HQ_FMT_Q3_K) return false;
  if (k % 64 != 0) return false;
  if (format == HQ_FMT_FP8_BLOCK && k % 128 != 0) return false;
  return n >= 1;
}

int32_t launch_grouped_gemm(const GroupedParams& p, int64_t rows, cudaStream_t stream) {
  if (p.x_dtype != HQ_DT_F16) return HQ_ERR_FORMAT;   // activations are copied into the operand tiles as f16
  if (rows <= 0) return HQ_OK;
  const uintptr_t w = reinterpret_cast<uintptr_t>(p.w) | reinterpret_cast<uintptr_t>(p.w_up);
  // 16-byte (Q6_K, Q3_K, Q2_K: 4-byte) pieces of the rows are copied as they lie
  const bool narrow = p.format == HQ_FMT_Q6_K || p.format == HQ_FMT_Q3_K || p.format == HQ_FMT_Q2_K;
  if ((w & (narrow ? 3u : 15u)) != 0) return HQ_ERR_ALIGN;
  switch (p.format) {
    case HQ_FMT_Q8_0: return launch_dq<HQ_FMT_Q8_0>(p, rows, stream);
    case HQ_FMT_Q4_K: return launch_dq<HQ_FMT_Q4_K>(p, rows, stream);
    case HQ_FMT_FP8_BLOCK: return launch_dq<HQ_FMT_FP8_BLOCK>(p, rows, stream);
    case HQ_FMT_MXFP4: return launch_dq<HQ_FMT_MXFP4>(p, rows, stream);
    case HQ_FMT_Q6_K: return launch_dq<HQ_FMT_Q6_K>(p, rows, stream);
    case HQ_FMT_Q5_K: return launch_dq<HQ_FMT_Q5_K>(p, rows, stream);
    case HQ_FMT_Q4_0: return launch_dq<HQ_FMT_Q4_0>(p, rows, stream);
    case HQ_FMT_Q5_0: return launch_dq<HQ_FMT_Q5_0>(p, rows, stream);
    case HQ_FMT_Q4_1: return launch_dq<HQ_FMT_Q4_1>(p, rows, stream);
    case HQ_FMT_Q5_1: return launch_dq<HQ_FMT_Q5_1>(p, rows, stream);
    case HQ_FMT_Q2_K: return launch_dq<HQ_FMT_Q2_K>(p, rows, stream);
    case HQ_FMT_Q3_K: return launch_dq<HQ_FMT_Q3_K>(p, rows, stream);
    default: return HQ_ERR_FORMAT;
  }
}

template <int FMT>
static bool plan_query(int format, const GroupedParams& p, int64_t rows, int32_t* out) {
  if (format == FMT) return dq_plan_query<FMT>(p, rows, out);
  if constexpr (FMT < HQ_FMT_Q3_K) return plan_query<FMT + 1>(format, p, rows, out);
  return false;
}

}  // namespace hq

// Test aid, not part of the public header: the plan of a call with `rows` activation rows (or assignments, with more than one
// expert), `gated` = a gate and an up bank.  Eight words as in dq_plan_query; 0 = there is one.
extern "C" int32_t hq_dq_gemm_plan(int32_t format, int64_t n, int64_t k, int32_t n_experts, int32_t gated, int64_t rows,
                                   int32_t* out) {
  hq::GroupedParams p{};
  static const int32_t some_bounds = 0;
  p.format = format;
  p.n = (int)n;
  p.k = (int)k;
  p.n_experts = n_experts;
  p.m = (int)rows;
  p.w_up = gated ? out : nullptr;
  p.expert_bounds = n_experts > 1 ? &some_bounds : nullptr;
  return rows > 0 && hq::grouped_gemm_supported(format, n, k) && hq::plan_query<HQ_FMT_Q8_0>(format, p, rows, out)
             ? HQ_OK : HQ_ERR_SHAPE;
}
