// Instances of the dequantizing GEMM (hq_dq_gemm.cuh): Q6_K Q3_K Q2_K.
#include "hq_dq_launch.cuh"

namespace hq {
template int32_t launch_dq<HQ_FMT_Q6_K>(const GroupedParams&, int64_t, cudaStream_t);
template bool dq_plan_query<HQ_FMT_Q6_K>(const GroupedParams&, int64_t, int32_t*);
template int32_t launch_dq<HQ_FMT_Q3_K>(const GroupedParams&, int64_t, cudaStream_t);
template bool dq_plan_query<HQ_FMT_Q3_K>(const GroupedParams&, int64_t, int32_t*);
template int32_t launch_dq<HQ_FMT_Q2_K>(const GroupedParams&, int64_t, cudaStream_t);
template bool dq_plan_query<HQ_FMT_Q2_K>(const GroupedParams&, int64_t, int32_t*);
}  // namespace hq
