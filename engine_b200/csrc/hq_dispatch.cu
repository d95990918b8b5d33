// Token -> expert dispatch tables: a stable counting sort of the flat assignment index t*top_k+s by expert id, built
// without output atomics so the permutation is identical on every run (the reference's CUDA scatter orders rows by
// atomic arrival; its host grouping is the stable order reproduced here).
//
// One launch of one block, or of a cluster of eight, 1024 threads each.  Every warp owns a contiguous run of
// assignments: it counts them into its own histogram row (shared memory), the rows become exclusive prefixes over the
// warps, the blocks of a cluster read each other's totals through distributed shared memory, a block-wide scan turns
// the totals into expert bounds, and every warp scatters its run with its own running positions.  Inside 32 assignments
// the rank among equal experts comes from a match mask and a popcount.  So no pass over global memory stands between
// counting and scattering, and no warp waits for another while it scatters.
//
// What bounds it: latency.  Three launches (count, scan over all chunks in one block, scatter whose warps took turns)
// took 26 us for 4,096 tokens x 8 of 128 experts and 13 us for one token.  Bytes: T*k*4 read twice (the second time
// from L2) + T*k*12 written.
//
// With few tokens the router runs in the same block first (route_dispatch_kernel): a launch and a trip through memory
// less on the shortest path of a MoE layer.
#include <atomic>

#include "hq_router.cuh"

namespace hq {

constexpr int kDispatchThreads = 1024;
constexpr int kDispatchCluster = 8;
// assignments up to which one block does it all: its 32 warps walk 128 each, as long as a cluster's start takes
constexpr int64_t kDispatchOneBlock = 4096;

struct DispatchCall {
  const uint32_t* ids;
  int total, top_k, n_experts, tile_rows, rows_at;
  int32_t *bounds, *sorted_assign, *sorted_token, *inv_perm, *ws;
};

static __device__ __forceinline__ uint32_t cluster_peer(const void* p, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
static __device__ __forceinline__ int32_t lds_cluster(uint32_t addr) {
  int32_t v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// Few assignments (kDispatchSmall): every thread compares its own, or its expert, with all of them.  No histogram, no scan: two
// steps of the block instead of six, 1 us instead of 4.3 for one token's tables.  ids_sm: the assignments' experts, filled up
// to a multiple of four with 0xFFFFFFFF; keys_sm: as many words.
constexpr int kDispatchSmall = 256;
static_assert((2 * kDispatchSmall + 2 * 32) * 4 <= kDispatchStatic, "few_sm, warp_rows and warp_tiles");
static __device__ __forceinline__ void dispatch_few(const DispatchCall& c, const uint32_t* ids_sm, uint32_t* keys_sm) {
  const int tid = threadIdx.x, E = c.n_experts, quads = (c.total + 3) >> 2;
  const uint4* ids4 = reinterpret_cast<const uint4*>(ids_sm);
  uint32_t e = 0xFFFFFFFFu;
  int pos = 0, at = 0, n = 0;
  if (tid < kDispatchSmall) {
    if (tid < c.total) {
      e = ids_sm[tid];
      for (int q = 0; q < quads; ++q) {
        const uint4 v = ids4[q];
        const uint32_t o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          pos += o[j] < e ? 1 : 0;
          n += o[j] == e ? 1 : 0;
          at += o[j] == e && 4 * q + j < tid ? 1 : 0;
        }
      }
      pos += at;
      // ids outside [0, n_experts) are skipped, as in dispatch_block
      if (e < (uint32_t)E) {
        c.sorted_assign[pos] = tid;
        c.sorted_token[pos] = tid / c.top_k;
        c.inv_perm[tid] = pos;
      } else {
        c.inv_perm[tid] = -1;
      }
    }
    // the assignments that start a work item, by sorted row
    const bool first = e < (uint32_t)E && at % c.tile_rows == 0;
    if (tid < 4 * quads) keys_sm[tid] = first ? (uint32_t)pos : 0xFFFFFFFFu;
    if (!first) e = 0xFFFFFFFFu;
  } else {
    for (int x = tid - kDispatchSmall; x <= E; x += kDispatchThreads - kDispatchSmall) {
      int less = 0;
      for (int q = 0; q < quads; ++q) {
        const uint4 v = ids4[q];
        less += (v.x < (uint32_t)x ? 1 : 0) + (v.y < (uint32_t)x ? 1 : 0) + (v.z < (uint32_t)x ? 1 : 0) + (v.w < (uint32_t)x ? 1 : 0);
      }
      c.bounds[x] = less;
      if (x == E) c.ws[1] = less;
    }
  }
  __syncthreads();
  if (tid > kDispatchSmall || (tid < kDispatchSmall && e >= (uint32_t)E)) return;
  const uint32_t key = tid == kDispatchSmall ? 0xFFFFFFFFu : (uint32_t)pos;
  int before = 0;
  const uint4* keys4 = reinterpret_cast<const uint4*>(keys_sm);
  for (int q = 0; q < quads; ++q) {
    const uint4 v = keys4[q];
    before += (v.x < key ? 1 : 0) + (v.y < key ? 1 : 0) + (v.z < key ? 1 : 0) + (v.w < key ? 1 : 0);
  }
  if (tid == kDispatchSmall) {
    c.ws[0] = before;
    c.ws[kHeaderRowsAt] = c.rows_at;
  } else {
    put_decode_item(c.ws, c.rows_at, before, (int32_t)e, pos, min(c.tile_rows, n - at));
  }
}

// smem: hist [rows][E], then five arrays of [E] (all int32)
static __device__ __forceinline__ void dispatch_block(const DispatchCall& c, int rows, int rank, int n_ranks, int32_t* sm) {
  const int E = c.n_experts;
  int32_t* hist = sm;
  int32_t* tot = hist + rows * E;       // this block's totals, read by the other blocks
  int32_t* base = tot + E;              // an expert's first sorted row that belongs to this block
  int32_t* start = base + E;            // ... to any
  int32_t* count = start + E;
  int32_t* tile0 = count + E;           // first work item of an expert
  __shared__ int32_t warp_rows[32], warp_tiles[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // this warp's run, whole groups of 32
  const int groups = (c.total + 31) >> 5, owners = n_ranks * rows;
  const int per = (groups + owners - 1) / owners * 32;
  const int lo = warp < rows ? min(c.total, (rank * rows + warp) * per) : 0;
  const int hi = warp < rows ? min(c.total, lo + per) : 0;
  for (int i = tid; i < rows * E; i += kDispatchThreads) hist[i] = 0;
  __syncthreads();
  int32_t* mine = hist + (warp < rows ? warp : 0) * E;
  for (int i0 = lo; i0 < hi; i0 += 128) {
    uint32_t e[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) e[j] = i0 + 32 * j + lane < hi ? c.ids[i0 + 32 * j + lane] : 0xFFFFFFFFu;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (e[j] < (uint32_t)E) atomicAdd(&mine[e[j]], 1);   // integer counts: order does not matter
  }
  __syncthreads();
  // rows of the histogram -> exclusive prefixes over the warps
  for (int e = tid; e < E; e += kDispatchThreads) {
    int32_t run = 0;
#pragma unroll 8
    for (int w = 0; w < rows; ++w) {
      const int32_t n = hist[w * E + e];
      hist[w * E + e] = run;
      run += n;
    }
    tot[e] = run;
  }
  if (n_ranks > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  // totals over the blocks; exclusive scan over the experts, four neighbours per thread
  int32_t all[4], before[4], rsum = 0, tsum = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int e = 4 * tid + j;
    all[j] = before[j] = 0;
    if (e < E) {
      if (n_ranks == 1) {
        all[j] = tot[e];
      } else {
#pragma unroll
        for (int r = 0; r < kDispatchCluster; ++r) {
          const int32_t n = lds_cluster(cluster_peer(&tot[e], (uint32_t)r));
          all[j] += n;
          if (r < rank) before[j] += n;
        }
      }
    }
    rsum += all[j];
    tsum += (all[j] + c.tile_rows - 1) / c.tile_rows;
  }
  // the others may leave once every block has read the totals (waited for at the end)
  if (n_ranks > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  int32_t rv = rsum, tv = tsum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int32_t a = __shfl_up_sync(0xffffffffu, rv, d), b = __shfl_up_sync(0xffffffffu, tv, d);
    if (lane >= d) { rv += a; tv += b; }
  }
  if (lane == 31) { warp_rows[warp] = rv; warp_tiles[warp] = tv; }
  __syncthreads();
  int32_t r0 = rv - rsum, t0 = tv - tsum, r_all = 0, t_all = 0;
#pragma unroll 8
  for (int w = 0; w < 32; ++w) {
    if (w < warp) { r0 += warp_rows[w]; t0 += warp_tiles[w]; }
    r_all += warp_rows[w];
    t_all += warp_tiles[w];
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int e = 4 * tid + j;
    if (e < E) {
      base[e] = r0 + before[j];
      start[e] = r0;
      count[e] = all[j];
      tile0[e] = t0;
      if (rank == 0) c.bounds[e] = r0;
      r0 += all[j];
      t0 += (all[j] + c.tile_rows - 1) / c.tile_rows;
    }
  }
  if (rank == 0 && tid == 0) {
    c.bounds[E] = r_all;
    c.ws[0] = t_all;
    c.ws[kHeaderRowsAt] = c.rows_at;
    c.ws[1] = r_all;
  }
  __syncthreads();
  // stable scatter of this warp's run
  for (int i0 = lo; i0 < hi; i0 += 32) {
    const int i = i0 + lane;
    const uint32_t e = i < hi ? c.ids[i] : 0xFFFFFFFFu;
    const bool routed = e < (uint32_t)E;
    const uint32_t peers = __match_any_sync(0xffffffffu, e);
    const int before_me = __popc(peers & ((1u << lane) - 1u));
    if (routed) {
      const int pos = base[e] + mine[e] + before_me;
      c.sorted_assign[pos] = i;
      c.sorted_token[pos] = i / c.top_k;
      c.inv_perm[i] = pos;
    } else if (i < hi) {
      // ids outside [0, n_experts) are skipped (padding slots such as -1): they get no sorted row and their
      // inverse-map entry says so, which the weighted reduce reads as "contributes nothing"
      c.inv_perm[i] = -1;
    }
    __syncwarp();
    if (routed && before_me == 0) mine[e] += __popc(peers);
    __syncwarp();
  }
  // work items: a warp per expert, lanes over its items
  for (int e = rank * 32 + warp; e < E; e += 32 * n_ranks) {
    const int r = start[e], n = count[e];
    for (int i = lane; i * c.tile_rows < n; i += 32)
      put_decode_item(c.ws, c.rows_at, tile0[e] + i, e, r + i * c.tile_rows, min(c.tile_rows, n - i * c.tile_rows));
  }
  if (n_ranks > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(kDispatchThreads) dispatch_kernel(const DispatchCall c, int rows, int n_ranks) {
  extern __shared__ int32_t dsm[];
  __shared__ __align__(16) uint32_t few_sm[2 * kDispatchSmall];
  pdl_launch_dependents();
  pdl_wait();
  if (c.total <= kDispatchSmall) {
    if (threadIdx.x < kDispatchSmall) few_sm[threadIdx.x] = threadIdx.x < c.total ? c.ids[threadIdx.x] : 0xFFFFFFFFu;
    __syncthreads();
    dispatch_few(c, few_sm, few_sm + kDispatchSmall);
    return;
  }
  dispatch_block(c, rows, (int)blockIdx.x, n_ranks, dsm);
}

// router of up to kRouteDispatchRows rows (one warp each), then their tables, in one block
template <int NV>
__global__ void __launch_bounds__(kDispatchThreads) route_dispatch_kernel(const RouterCall rc, const DispatchCall c, int rows) {
  extern __shared__ int32_t dsm[];
  pdl_launch_dependents();
  pdl_wait();
  __shared__ __align__(16) uint32_t few_sm[2 * kDispatchSmall];
  const int warp = threadIdx.x >> 5;
  const bool few = c.total <= kDispatchSmall;
  const int pad = c.total + kDispatchThreads - 1 - (int)threadIdx.x;      // the last three threads fill up the ids
  if (few && threadIdx.x >= kDispatchThreads - 3 && pad < kDispatchSmall) few_sm[pad] = 0xFFFFFFFFu;
  if (warp < rc.n_rows)
    route_row<NV>(rc, warp, threadIdx.x & 31, reinterpret_cast<float*>(dsm) + warp * c.n_experts, few ? few_sm : nullptr);
  __syncthreads();       // the ids, written by this block, are read back by other warps of it
  if (few) dispatch_few(c, few_sm, few_sm + kDispatchSmall);
  else dispatch_block(c, rows, 0, 1, dsm);
}

template <typename K>
static bool allow_smem(K kern, size_t bytes) {
  static std::atomic<size_t> have[64];
  int dev = 0;
  if (!dispatch_asks_for_smem((int64_t)bytes)) return true;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  if (dev < 64 && have[dev].load(std::memory_order_relaxed) >= bytes) return true;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDispatchDynamic) != cudaSuccess) return false;
  if (dev < 64) have[dev].store((size_t)kDispatchDynamic, std::memory_order_relaxed);
  return true;
}

static DispatchCall dispatch_call(const uint32_t* ids, int64_t n_tokens, int top_k, int n_experts, int32_t* bounds,
                                  int32_t* sorted_assign, int32_t* sorted_token, int32_t* inv_perm, int32_t* ws) {
  const DispatchLayout l = dispatch_layout(n_tokens, top_k, n_experts);
  return DispatchCall{ids, (int)(n_tokens * top_k), top_k, n_experts, l.tile_rows, (int)l.rows_at, bounds, sorted_assign,
                      sorted_token, inv_perm, ws};
}

int32_t launch_dispatch(const uint32_t* ids, int64_t n_tokens, int top_k, int n_experts, int32_t* bounds,
                        int32_t* sorted_assign, int32_t* sorted_token, int32_t* inv_perm, int32_t* ws,
                        cudaStream_t stream) {
  const DispatchCall c = dispatch_call(ids, n_tokens, top_k, n_experts, bounds, sorted_assign, sorted_token, inv_perm, ws);
  const int rows = dispatch_rows(n_experts), n_ranks = c.total <= kDispatchOneBlock ? 1 : kDispatchCluster;
  const size_t smem = (size_t)dispatch_smem(n_experts);
  if (!allow_smem(dispatch_kernel, smem)) return HQ_ERR_CUDA;
  return launch_pdl(dispatch_kernel, dim3((unsigned)n_ranks), kDispatchThreads, smem, stream, n_ranks, c, rows, n_ranks);
}

int32_t launch_route_dispatch(const RouterCall& rc, int32_t* bounds, int32_t* sorted_assign, int32_t* sorted_token,
                              int32_t* inv_perm, int32_t* ws, cudaStream_t stream) {
  const DispatchCall c = dispatch_call(rc.ids, rc.n_rows, rc.a.top_k, rc.a.n_experts, bounds, sorted_assign, sorted_token,
                                       inv_perm, ws);
  const int rows = dispatch_rows(c.n_experts);
  const size_t smem = (size_t)dispatch_smem(c.n_experts);
  auto run = [&](auto kern) {
    if (!allow_smem(kern, smem)) return (int32_t)HQ_ERR_CUDA;
    return launch_pdl(kern, dim3(1), kDispatchThreads, smem, stream, 1, rc, c, rows);
  };
  if (c.n_experts <= 64) return run(route_dispatch_kernel<2>);
  if (c.n_experts <= 128) return run(route_dispatch_kernel<4>);
  if (c.n_experts <= 256) return run(route_dispatch_kernel<8>);
  return HQ_ERR_SHAPE;
}

// ---- variant for callers that cannot allocate ------------------------------------------------------
// Some hosts have no way to hand this library a workspace: every byte of device memory is already owned by
// their own pool (a serving engine that sizes its KV cache to whatever is free), or the call is made from
// a place where asking the CUDA runtime for memory is not allowed.  For them the work-item
// lists live in a fixed array inside the library image.  It is sized for kNoAllocMaxAssignments
// assignments and kNoAllocMaxExperts experts (about 100 KB), exists once per GPU that loads the library
// and is shared by every call: two calls that overlap on the GPU (different streams, or graphs replayed
// concurrently) race on it.  Nothing in it has to start at zero -- every word that is read is written
// first by the same call.
constexpr int kNoAllocMaxAssignments = 65536;
constexpr int kNoAllocMaxExperts = 512;
constexpr int64_t kNoAllocWords = dispatch_words_up_to(kNoAllocMaxAssignments, kNoAllocMaxExperts);
static __device__ __align__(256) int32_t g_noalloc_scratch[kNoAllocWords];

int32_t launch_dispatch_noalloc(const uint32_t* ids, int64_t n_tokens, int top_k, int n_experts, int32_t* bounds,
                                int32_t* sorted_assign, int32_t* sorted_token, int32_t* inv_perm,
                                cudaStream_t stream) {
  if (n_tokens * top_k > kNoAllocMaxAssignments || n_experts > kNoAllocMaxExperts) return HQ_ERR_TOO_LARGE;
  const DispatchLayout l = dispatch_layout(n_tokens, top_k, n_experts);
  if (l.total_words > kNoAllocWords) return HQ_ERR_TOO_LARGE;
  // The array's name is only a host-side handle; kernels need its device address, which differs per device.
  // Looked up on the first call made with a given device current (a plain runtime query, no allocation).
  // The cache is written by whichever host thread gets there first; every writer stores the same value.
  static std::atomic<int32_t*> dev_ptr[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return HQ_ERR_CUDA;
  int32_t* scratch = dev_ptr[dev].load(std::memory_order_acquire);
  if (scratch == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || p == nullptr) return HQ_ERR_CUDA;
    scratch = static_cast<int32_t*>(p);
    dev_ptr[dev].store(scratch, std::memory_order_release);
  }
  return launch_dispatch(ids, n_tokens, top_k, n_experts, bounds, sorted_assign, sorted_token, inv_perm, scratch,
                         stream);
}

}  // namespace hq
