// Instances of the dequantizing GEMM (hq_dq_gemm.cuh): FP8_BLOCK MXFP4 Q4_0.
#include "hq_dq_launch.cuh"

namespace hq {
template int32_t launch_dq<HQ_FMT_FP8_BLOCK>(const GroupedParams&, int64_t, cudaStream_t);
template bool dq_plan_query<HQ_FMT_FP8_BLOCK>(const GroupedParams&, int64_t, int32_t*);
template int32_t launch_dq<HQ_FMT_MXFP4>(const GroupedParams&, int64_t, cudaStream_t);
template bool dq_plan_query<HQ_FMT_MXFP4>(const GroupedParams&, int64_t, int32_t*);
template int32_t launch_dq<HQ_FMT_Q4_0>(const GroupedParams&, int64_t, cudaStream_t);
template bool dq_plan_query<HQ_FMT_Q4_0>(const GroupedParams&, int64_t, int32_t*);
}  // namespace hq
