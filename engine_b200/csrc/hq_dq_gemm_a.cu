// Instances of the dequantizing GEMM (hq_dq_gemm.cuh): Q4_K Q5_K Q8_0.
#include "hq_dq_launch.cuh"

namespace hq {
template int32_t launch_dq<HQ_FMT_Q4_K>(const GroupedParams&, int64_t, cudaStream_t);
template bool dq_plan_query<HQ_FMT_Q4_K>(const GroupedParams&, int64_t, int32_t*);
template int32_t launch_dq<HQ_FMT_Q5_K>(const GroupedParams&, int64_t, cudaStream_t);
template bool dq_plan_query<HQ_FMT_Q5_K>(const GroupedParams&, int64_t, int32_t*);
template int32_t launch_dq<HQ_FMT_Q8_0>(const GroupedParams&, int64_t, cudaStream_t);
template bool dq_plan_query<HQ_FMT_Q8_0>(const GroupedParams&, int64_t, int32_t*);
}  // namespace hq
