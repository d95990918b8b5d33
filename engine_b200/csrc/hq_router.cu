// Router kernel: one warp per token row (route_row), four rows per block.
//
// What bounds it: latency of one row (its logits from memory, top_k rounds of two warp reductions); at 4,096 rows of 128
// experts every row is in flight at once.  HBM bytes per row: E * sizeof(logit) + k * 8.
#include "hq_router.cuh"

namespace hq {

constexpr int kRouterWarps = 4;

template <int NV>
__global__ void __launch_bounds__(kRouterWarps * 32) router_kernel(const RouterCall c) {
  extern __shared__ float rsm[];
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * kRouterWarps + warp;
  if (row < c.n_rows) route_row<NV>(c, row, lane, rsm + (size_t)warp * c.a.n_experts);
}

int32_t launch_router(const RouterCall& c, cudaStream_t stream) {
  if (c.n_rows == 0) return HQ_OK;
  const size_t smem = c.n_group > 1 ? (size_t)kRouterWarps * c.a.n_experts * sizeof(float) : 0;
  const dim3 grid((unsigned)((c.n_rows + kRouterWarps - 1) / kRouterWarps));
  auto kern = c.a.n_experts <= 64    ? router_kernel<2>
              : c.a.n_experts <= 128 ? router_kernel<4>
              : c.a.n_experts <= 256 ? router_kernel<8>
              : c.a.n_experts <= 512 ? router_kernel<16>
                                     : router_kernel<32>;
  return launch_pdl(kern, grid, kRouterWarps * 32, smem, stream, 1, c);
}

}  // namespace hq
