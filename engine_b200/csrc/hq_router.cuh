// MoE router of one token row by one warp, shared by the router kernel and the kernel that routes and dispatches small
// calls: score (raw / softmax / sigmoid) -> optional selection bias -> top-k by (selection DESC, expert id ASC) ->
// weights (score / softmax over the selected logits / sigmoid of the selected logits) -> optional renormalisation,
// output scale and per-expert scale.
//
// A lane holds experts lane, lane + 32, ... in registers.  Selection scores become unsigned keys of the same order, so a
// round of the arg-max is two warp reductions (largest key, lowest expert that has it) instead of ten shuffles over
// scores re-read from shared memory.  Every sum is a fixed-order shuffle tree: the same logits give the same bits.
#pragma once
#include <math_constants.h>

#include "hq_common.cuh"
#include "hq_kernels.h"

namespace hq {

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, m));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}
// f32 -> unsigned with the order of the numbers (-0 as +0); never 0, which marks a consumed expert
__device__ __forceinline__ uint32_t order_key(float v) {
  const uint32_t b = __float_as_uint(v + 0.f);
  return (b & 0x80000000u) ? ~b : b | 0x80000000u;
}

// groups_sm: n_experts floats of shared memory of this warp, read with n_group > 1 only; ids_sm: if given, the ids go there too
template <int NV>
__device__ __forceinline__ void route_row(const RouterCall& c, int64_t row, int lane, float* groups_sm, uint32_t* ids_sm = nullptr) {
  const hq_router_args& a = c.a;
  const int E = a.n_experts;
  float raw[NV], score[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int e = lane + 32 * i;
    float v = -CUDART_INF_F;
    if (e < E) {
      v = load_as_float(c.logits, c.dtype, row * E + e);
      if (a.clamp_logits) v = fminf(fmaxf(v, a.clamp_min), a.clamp_max);
      if (v != v) v = -CUDART_INF_F;
    }
    raw[i] = v;
  }
  if (a.score_mode == HQ_SCORE_SOFTMAX) {
    float m = -CUDART_INF_F;
#pragma unroll
    for (int i = 0; i < NV; ++i) m = fmaxf(m, raw[i]);
    m = warp_max(m);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      score[i] = expf(raw[i] - m);
      if (lane + 32 * i < E) s += score[i];
    }
    s = warp_sum(s);
#pragma unroll
    for (int i = 0; i < NV; ++i) score[i] = score[i] / s;
  } else {
#pragma unroll
    for (int i = 0; i < NV; ++i) score[i] = a.score_mode == HQ_SCORE_SIGMOID ? 1.f / (1.f + expf(-raw[i])) : raw[i];
  }
  uint32_t key[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int e = lane + 32 * i;
    float v = score[i];
    if (a.selection_bias != nullptr && e < E) v += a.selection_bias[e];
    if (v != v) v = -CUDART_INF_F;
    key[i] = e < E ? order_key(v) : 0u;
    if (c.n_group > 1 && e < E) groups_sm[e] = v;
  }

  // Group-limited selection (DeepSeek): experts form n_group contiguous groups; a group's score is the sum of its
  // two best selection scores (group_mode 0, "noaux_tc") or its best one (1, "group_limited_greedy"); only the
  // topk_group best groups stay selectable, the selection score of every other expert becomes 0
  // (hanzo-engine/src/models/deepseek3.rs:623-690).  Lane g scores group g; ties go to the lower group.
  if (c.n_group > 1) {
    __syncwarp();
    const int gs = E / c.n_group;
    uint32_t gkey = 0u;
    if (lane < c.n_group) {
      float t1 = -CUDART_INF_F, t2 = -CUDART_INF_F;
      for (int e = lane * gs; e < (lane + 1) * gs; ++e) {
        const float v = groups_sm[e];
        if (v > t1) { t2 = t1; t1 = v; }
        else if (v > t2) t2 = v;
      }
      const float g = c.group_mode == 0 ? t1 + t2 : t1;
      // a group score that is not a number orders below every other one
      gkey = g == g ? order_key(g) : 1u;
    }
    uint32_t keep = 0;
    for (int r = 0; r < c.topk_group; ++r) {
      const uint32_t best = __reduce_max_sync(0xffffffffu, gkey);
      const int g = __ffs(__ballot_sync(0xffffffffu, gkey == best)) - 1;
      keep |= 1u << g;
      if (lane == g) gkey = 0u;
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int e = lane + 32 * i;
      if (e < E && ((keep >> (e / gs)) & 1u) == 0u) key[i] = order_key(0.f);
    }
  }

  // k rounds of arg-max; ties go to the lower expert id.  Lane j keeps the j-th result.
  float my_w = 0.f;
  uint32_t my_id = 0;
  for (int r = 0; r < a.top_k; ++r) {
    uint32_t bk = 0u;
    int bi = 0;
    float bo = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (key[i] > bk) {
        bk = key[i];
        bi = i;
        bo = a.weight_mode == HQ_WEIGHT_SCORE ? score[i] : raw[i];
      }
    const uint32_t best = __reduce_max_sync(0xffffffffu, bk);
    const uint32_t e = __reduce_min_sync(0xffffffffu, bk == best ? (uint32_t)(lane + 32 * bi) : 0xffffffffu);
    const float out = __shfl_sync(0xffffffffu, bo, (int)(e & 31u));
    if (lane == r) { my_w = out; my_id = e; }
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (lane + 32 * i == (int)e) key[i] = 0u;
  }
  if (a.weight_mode == HQ_WEIGHT_SIGMOID) my_w = 1.f / (1.f + expf(-my_w));
  const bool mine = lane < a.top_k;
  if (a.weight_mode == HQ_WEIGHT_SOFTMAX) {
    const float m = warp_max(mine ? my_w : -CUDART_INF_F);
    const float ex = mine ? expf(my_w - m) : 0.f;
    const float s = warp_sum(ex);
    my_w = ex / s;
  }
  if (a.renormalize) {
    float s = warp_sum(mine ? my_w : 0.f);
    if (a.norm_min > 0.f) s = fmaxf(s, a.norm_min);
    my_w = my_w / s;
  }
  if (a.output_scale != 1.0f) my_w *= a.output_scale;
  if (mine) {
    if (a.expert_scale != nullptr) my_w *= a.expert_scale[my_id];
    c.weights[row * a.top_k + lane] = my_w;
    if (ids_sm != nullptr) ids_sm[row * a.top_k + lane] = my_id;
    c.ids[row * a.top_k + lane] = my_id;
  }
}

}  // namespace hq
