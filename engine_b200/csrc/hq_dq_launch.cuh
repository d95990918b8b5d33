// Host side of the dequantizing GEMM: the plan of a launch and the launch itself.
#pragma once
#include "hq_dq_gemm.cuh"
#include "hq_gemv_shared.cuh"

namespace hq {

bool f8_encode_2d(CUtensorMap* map, CUtensorMapDataType type, const void* base, uint64_t inner, uint64_t rows,
                  uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_rows, CUtensorMapSwizzle swz);
// a [rows, 64 * blocks] matrix of 16-bit elements as (64 columns, rows, column blocks): a box is `box_rows` rows of
// `box_blocks` column blocks, one block behind the other in shared memory, each of 128-byte swizzled rows
bool encode_column_blocks(CUtensorMap* map, const void* base, uint64_t blocks, uint64_t rows, uint64_t row_stride_bytes,
                          uint32_t box_rows, uint32_t box_blocks);

// Cycles of one 64-k step of a tile, fitted to sweeps of tile widths on this part: the instructions that expand 128 x 64
// weights, then half a cycle per token column.  A tile costs a start-up; without a second accumulator buffer its
// epilogue is not hidden either.
constexpr double kDqTileCycles = 1000.0, kDqSplitCycles = 2500.0, kDqDrainCycles = 24.0, kDqGatedDrainCycles = 56.0;

template <int FMT>
double dq_step_cycles(int tokens) {
  const double expand = FMT == HQ_FMT_Q6_K || FMT == HQ_FMT_Q3_K ? 740.0
                        : FMT == HQ_FMT_FP8_BLOCK || FMT == HQ_FMT_MXFP4 ? 410.0 : 500.0;
  return expand + 0.5 * tokens;
}

template <int FMT>
bool dq_smem_plan(DqPlan& pl, int n_experts, bool expert_indexed) {
  using T = DqTraits<FMT>;
  pl.nbuf = pl.tn <= 192 ? 2 : 1;
  pl.subs = pl.tn <= 64 ? 4 : 2;
  const int stage = pl.subs * pl.tn * 128;
  pl.cpc = (pl.tn + pl.kslices - 1) / pl.kslices;
  const int recv = pl.kslices > 1 ? pl.kslices * pl.cpc * 512 : 0;
  const int pref = expert_indexed ? (2 * (n_experts + 1) * 4 + 15) & ~15 : 16;
  const int rows = 2 * kDqMaxTokens * 4;
  const int fixed = rows + pref + kDqNumBars * 8 + 16 + 1024;
  pl.ns = (512 - pl.nbuf * pl.tn) / (32 * pl.subs);
  if (pl.ns > 4) pl.ns = 4;
  // two slots at least: a group of expanding warps meets every stage (subs = 4) or, dq_walk_steps sees to it, every second one
  // (subs = 2), so its slot is never two uses behind, which one parity bit could not tell from none
  const int min_ns = 2;
  for (;; --pl.ns) {
    if (pl.ns < min_ns) return false;
    pl.nr = (kDqSmem - fixed - recv - pl.ns * stage) / T::STAGE;
    if (pl.nr >= (pl.ns > min_ns ? 3 : 2)) break;
  }
  if (pl.nr > kDqMaxRaw) pl.nr = kDqMaxRaw;
  pl.ns_magic = pl.ns == 3 ? 0x55555556u : pl.ns == 2 ? 0x80000000u : 0x40000000u;
  pl.off_raw = pl.ns * stage;
  pl.off_recv = pl.off_raw + pl.nr * T::STAGE;
  pl.off_rows = pl.off_recv + recv;
  pl.off_pref = pl.off_rows + rows;
  pl.off_bar = pl.off_pref + pref;
  pl.smem = pl.off_bar + kDqNumBars * 8 + 16 + 1024;
  return true;
}

// lets the kernel have its shared memory, once per device
template <int FMT, bool ODD>
bool dq_kernel_ready() {
  static bool done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  if (dev < 64 && done[dev]) return true;
  if (cudaFuncSetAttribute(dq_gemm_kernel<FMT, ODD>, cudaFuncAttributeMaxDynamicSharedMemorySize, kDqSmem) != cudaSuccess)
    return false;
  if (dev < 64) done[dev] = true;
  return true;
}

// CTA clusters of `s` CTAs (one per SM) the device can hold at once
template <int FMT>
int dq_max_clusters(int s) {
  static int cached[64][9] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return 1;
  if (cached[dev][s] == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(s * (sm_count() / s)));
    cfg.blockDim = dim3(DqTraits<FMT>::THREADS);
    cfg.dynamicSmemBytes = kDqSmem - 1024;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)s;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    // (without the attribute the query fails, and the answer would be the guess below for good)
    if (!dq_kernel_ready<FMT, false>() ||
        cudaOccupancyMaxActiveClusters(&n, dq_gemm_kernel<FMT, false>, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = sm_count() / s * 3 / 4;
      if (n < 1) n = 1;
    }
    cached[dev][s] = n;
  }
  return cached[dev][s];
}

// Dense calls: the token-tile width and the number of K slices with the smallest estimated time.  Expert-indexed
// calls: the tile width for the average rows of an expert (plus one standard deviation of a random assignment).
template <int FMT>
bool dq_plan(const GroupedParams& p, int64_t rows, DqPlan& best, int& grid) {
  const bool two = p.w_up != nullptr, experts = p.expert_bounds != nullptr;
  const int n_nt = two ? (p.n + 63) / 64 : (p.n + 127) / 128;
  const int nrs = (p.k + 255) / 256;
  const int sms = sm_count();
  double best_cost = -1.0;
  for (int tn = 16; tn <= kDqMaxTokens; tn += 16) {
    DqPlan pl{};
    int64_t tiles;
    int tokens;
    if (experts) {
      const double avg = (double)rows / p.n_experts, hi = avg + sqrt(avg);
      pl.tn = tn;
      const int nt = hi <= tn ? 1 : (int)((hi + tn - 1) / tn);
      tiles = (int64_t)nt * p.n_experts;
      tokens = ((int)(avg / nt) + 16) & ~15;
      if (tokens > tn) tokens = tn;
    } else {
      const int n_tt = (int)((rows + tn - 1) / tn);
      pl.rows_per_tile = (int)((rows + n_tt - 1) / n_tt);
      pl.n_tt = (int)((rows + pl.rows_per_tile - 1) / pl.rows_per_tile);
      pl.tn = (pl.rows_per_tile + 15) & ~15;
      if (pl.tn != tn) continue;
      tiles = pl.n_tt;
      tokens = tn;
    }
    for (int s = 1; s <= 8 && s <= nrs; ++s) {
      if (s > 1 && (experts || tn > 128)) break;
      if ((s - 1) * ((nrs + s - 1) / s) >= nrs) continue;      // a slice would be empty
      pl.kslices = s;
      if (!dq_smem_plan<FMT>(pl, p.n_experts, experts)) continue;
      const int64_t slots = s == 1 ? sms : dq_max_clusters<FMT>(s);
      const int64_t items = tiles * n_nt;
      const double waves = experts ? (double)(items + slots - 1) / slots : (double)((items + slots - 1) / slots);
      const double drain = pl.nbuf == 2 ? 0.0 : (two ? kDqGatedDrainCycles : kDqDrainCycles) * tokens;
      const double cost = waves * (4.0 * ((nrs + s - 1) / s) * dq_step_cycles<FMT>(tokens) + kDqTileCycles + drain +
                                   (s > 1 ? kDqSplitCycles : 0.0));
      if (best_cost < 0.0 || cost < best_cost * 0.999) {
        best_cost = cost;
        best = pl;
        grid = (int)(items < slots ? items : slots) * s;
        if (experts) grid = sms;
      }
    }
  }
  return best_cost >= 0.0;
}

template <int FMT>
bool dq_plan_query(const GroupedParams& p, int64_t rows, int32_t* out) {
  DqPlan pl{};
  int grid = 0;
  if (!dq_plan<FMT>(p, rows, pl, grid)) return false;
  const int32_t v[8] = {pl.tn, pl.subs, pl.ns, pl.nr, pl.nbuf, pl.kslices, grid, pl.smem};
  for (int i = 0; i < 8; ++i) out[i] = v[i];
  return true;
}

template <int FMT, bool ODD>
int32_t launch_dq_plan(const GroupedParams& p, DqPlan& pl, int grid, int64_t rows, cudaStream_t stream) {
  if (!dq_kernel_ready<FMT, ODD>()) return HQ_ERR_CUDA;
  using T = DqTraits<FMT>;
  CUtensorMap tm_w{}, tm_wu{};
  DqTokenMaps tm_x{};
  pl.raw_tma = T::WIDE || (p.w_row_bytes % 16 == 0 && (reinterpret_cast<uintptr_t>(p.w) & 15u) == 0 &&
                           (reinterpret_cast<uintptr_t>(p.w_up) & 15u) == 0);
  if (pl.raw_tma) {
    const uint64_t wrows = (uint64_t)p.n_experts * (uint64_t)p.n;
    const CUtensorMapSwizzle swz = T::SWZ ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE;
    const uint32_t box_rows = p.w_up != nullptr ? 64 : 128;
    if constexpr (T::BOXES == 2) {
      const uint64_t blocks = (uint64_t)p.w_row_bytes / 128;
      if (!encode_column_blocks(&tm_w, p.w, blocks, wrows, (uint64_t)p.w_row_bytes, box_rows, 2) ||
          (p.w_up != nullptr && !encode_column_blocks(&tm_wu, p.w_up, blocks, wrows, (uint64_t)p.w_row_bytes, box_rows, 2)))
        return HQ_ERR_CUDA;
    } else if (!f8_encode_2d(&tm_w, CU_TENSOR_MAP_DATA_TYPE_UINT16, p.w, (uint64_t)p.w_row_bytes / 2, wrows,
                             (uint64_t)p.w_row_bytes, T::PITCH / 2, box_rows, swz) ||
               (p.w_up != nullptr && !f8_encode_2d(&tm_wu, CU_TENSOR_MAP_DATA_TYPE_UINT16, p.w_up, (uint64_t)p.w_row_bytes / 2,
                                                   wrows, (uint64_t)p.w_row_bytes, T::PITCH / 2, box_rows, swz))) {
      return HQ_ERR_CUDA;
    }
  }
  pl.x_tma = p.x_rows == nullptr;
  if (pl.x_tma) {
    const int first = p.expert_bounds != nullptr ? 16 : pl.tn;
    for (int box = first; box <= pl.tn; box += 16)
      if (!encode_column_blocks(&tm_x.m[(box - first) / 16], p.x, (uint64_t)p.k / 64, (uint64_t)rows, (uint64_t)p.x_stride * 2,
                                (uint32_t)box, (uint32_t)pl.subs))
        return HQ_ERR_CUDA;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(DqTraits<FMT>::THREADS);
  cfg.dynamicSmemBytes = (size_t)pl.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)pl.kslices;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pl.kslices > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, dq_gemm_kernel<FMT, ODD>, tm_w, tm_wu, tm_x, p, pl) == cudaSuccess ? HQ_OK : HQ_ERR_CUDA;
}

template <int FMT>
int32_t launch_dq(const GroupedParams& p, int64_t rows, cudaStream_t stream) {
  DqPlan pl{};
  int grid = 0;
  if (!dq_plan<FMT>(p, rows, pl, grid)) return HQ_ERR_SHAPE;
  if (grid <= 0) return HQ_OK;
  // The GGML types have whole raw stages only (K % 256 == 0), which is an even number of operand stages.  So have all K slices
  // but the last.
  if constexpr (FMT == HQ_FMT_FP8_BLOCK || FMT == HQ_FMT_MXFP4) {
    const int per = ((p.k + 255) / 256 + pl.kslices - 1) / pl.kslices;
    if (dq_odd_on_two_slots(pl.subs, pl.ns, p.k / 64 - 4 * per * (pl.kslices - 1)))
      return launch_dq_plan<FMT, true>(p, pl, grid, rows, stream);
  }
  return launch_dq_plan<FMT, false>(p, pl, grid, rows, stream);
}

}  // namespace hq
