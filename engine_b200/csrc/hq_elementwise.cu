// Memory-bound helpers around the expert GEMMs: weighted un-permute/reduce,
// FP8 quantizers (1x128 activation groups, 128x128 weight blocks), gated
// activations.  All are single-pass: each input byte is read once, each output
// byte written once, accumulation in f32.
#include <cuda_fp8.h>

#include "hq_common.cuh"
#include "hq_kernels.h"

namespace hq {

// ---- out[t,:] = sum_s w[t,s] * y[row(t,s),:] (+ addend[t,:]) ----------------------
// One CTA per (token, slab of at most 256 x 8 elements); slots are added in slot order, so the f32 sum is reproducible.  Bytes:
// T*k*H*sizeof(y) read + T*H*sizeof(out) written, which bounds it: the rows of four slots are in flight per thread, and
// the eight results leave in one store.  With eight slots in flight a thread of 16-bit rows holds 55 registers in place of 40, and
// what is in flight per SM is no more; a block covers an equal share of a row, as no block of 256 has a half-empty last one
// then.  bf16, 4,096 x 8 x 7,168: 132 -> 116 us (528 MB: 77), 8,192 x 4 x 2,880: 69 -> 52 (236 MB: 35).
template <typename TO>
__device__ __forceinline__ void store8(TO* p, const float (&v)[8]) {
  if constexpr (sizeof(TO) == 4) {
    reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (std::is_same<TO, __half>::value) {
        w[i] = pack_half2(v[2 * i], v[2 * i + 1]);
      } else {
        const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t*>(&b);
      }
    }
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}
// vec: rows, out and addend can be read and written eight elements at a time.
template <typename TY, typename TO>
__global__ void __launch_bounds__(256) weighted_reduce_kernel(const TY* __restrict__ y, const float* __restrict__ w,
                                                              const int32_t* __restrict__ row_map,
                                                              const TO* __restrict__ addend, TO* __restrict__ out,
                                                              int top_k, int64_t hidden, int vec) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t t = blockIdx.x;
  const int64_t h0 = ((int64_t)blockIdx.y * blockDim.x + threadIdx.x) * 8;
  if (h0 >= hidden) return;
  const float* wt = w + t * top_k;
  // sorted row of slot s; < 0: a slot without a row (skipped id), adds nothing
  auto row_of = [&](int s) { return row_map != nullptr ? (int64_t)__ldg(row_map + t * top_k + s) : t * top_k + s; };
  if (vec) {
    constexpr int U = 4;                                // slots in flight
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    for (int s0 = 0; s0 < top_k; s0 += U) {
      uint4 v[U][sizeof(TY) / 2];
      float ws[U];
      bool live[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t row = s0 + u < top_k ? row_of(s0 + u) : -1;
        live[u] = row >= 0;
        if (live[u]) {
          load8(y + row * hidden + h0, v[u]);
          ws[u] = __ldg(wt + s0 + u);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (live[u]) {
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i] = fmaf(ws[u], elem8<TY>(v[u], i), acc[i]);
        }
    }
    if (addend) {
      uint4 a[sizeof(TO) / 2];
      load8(addend + t * hidden + h0, a);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += elem8<TO>(a, i);
    }
    store8(out + t * hidden + h0, acc);
    return;
  }
  for (int i = 0; i < 8 && h0 + i < hidden; ++i) {
    float r = 0.f;
    for (int s = 0; s < top_k; ++s) {
      const int64_t row = row_of(s);
      if (row >= 0) r = fmaf(wt[s], to_float<TY>(y[row * hidden + h0 + i]), r);
    }
    if (addend) r += to_float<TO>(addend[t * hidden + h0 + i]);
    if constexpr (sizeof(TO) == 4) out[t * hidden + h0 + i] = r;
    else if constexpr (std::is_same<TO, __half>::value) out[t * hidden + h0 + i] = __float2half_rn(r);
    else out[t * hidden + h0 + i] = __float2bfloat16_rn(r);
  }
}

template <typename TY, typename TO>
static int32_t launch_wr(const void* y, const float* w, const int32_t* row_map, const void* addend, void* out,
                         int64_t n_tokens, int top_k, int64_t hidden, cudaStream_t stream) {
  const uintptr_t bits = reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(addend);
  const int vec = hidden % 8 == 0 && (bits & 15u) == 0;
  // blocks of equal width that cover a row
  const int64_t lanes = (hidden + 7) / 8;
  const unsigned slabs = (unsigned)((lanes + 255) / 256);
  const int threads = (int)((lanes + slabs * 32 - 1) / (slabs * 32)) * 32;
  return launch_pdl(weighted_reduce_kernel<TY, TO>, dim3((unsigned)n_tokens, slabs), threads, 0, stream, 1, (const TY*)y, w, row_map,
                    (const TO*)addend, (TO*)out, top_k, hidden, vec);
}
int32_t launch_weighted_reduce(const void* y, int y_dtype, const float* w, const int32_t* row_map,
                               const void* addend, void* out, int out_dtype, int64_t n_tokens, int top_k,
                               int64_t hidden, cudaStream_t stream) {
  if (n_tokens == 0) return HQ_OK;
#define HQ_WR(TYC, TY, TOC, TO) \
  if (y_dtype == TYC && out_dtype == TOC) return launch_wr<TY, TO>(y, w, row_map, addend, out, n_tokens, top_k, hidden, stream);
  HQ_WR(HQ_DT_F32, float, HQ_DT_F32, float)
  HQ_WR(HQ_DT_F32, float, HQ_DT_BF16, __nv_bfloat16)
  HQ_WR(HQ_DT_F32, float, HQ_DT_F16, __half)
  HQ_WR(HQ_DT_BF16, __nv_bfloat16, HQ_DT_F32, float)
  HQ_WR(HQ_DT_BF16, __nv_bfloat16, HQ_DT_BF16, __nv_bfloat16)
  HQ_WR(HQ_DT_F16, __half, HQ_DT_F32, float)
  HQ_WR(HQ_DT_F16, __half, HQ_DT_F16, __half)
  HQ_WR(HQ_DT_F16, __half, HQ_DT_BF16, __nv_bfloat16)
  HQ_WR(HQ_DT_BF16, __nv_bfloat16, HQ_DT_F16, __half)
#undef HQ_WR
  return HQ_ERR_FORMAT;
}

// ---- FP8 e4m3 -------------------------------------------------------------------
__device__ __forceinline__ uint8_t f32_to_e4m3(float v) {
  return (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ float e4m3_to_f32(uint8_t c) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)c, __NV_E4M3);
  return __half2float(*reinterpret_cast<const __half*>(&h));
}

// one warp per group of 128 values; lane owns 4 consecutive values
__global__ void __launch_bounds__(256) fp8_vector_quant_kernel(const void* __restrict__ x, int dtype,
                                                               int64_t n_groups, uint8_t* __restrict__ codes,
                                                               float* __restrict__ scales) {
  const int64_t grp = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (grp >= n_groups) return;
  const int lane = threadIdx.x & 31;
  const int64_t base = grp * 128 + lane * 4;
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = load_as_float(x, dtype, base + i);
  float m = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
  const float scale = m > 0.f ? __fdiv_rn(m, 448.f) : 1e-12f;
  uint32_t packed = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float q = fminf(fmaxf(__fdiv_rn(v[i], scale), -448.f), 448.f);
    packed |= (uint32_t)f32_to_e4m3(q) << (8 * i);
  }
  *reinterpret_cast<uint32_t*>(codes + base) = packed;
  if (lane == 0) scales[grp] = scale;
}

__global__ void __launch_bounds__(256) fp8_vector_dequant_kernel(const uint8_t* __restrict__ codes,
                                                                 const float* __restrict__ scales, int64_t n,
                                                                 void* __restrict__ out, int dtype) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  store_from_float(out, dtype, i, e4m3_to_f32(codes[i]) * scales[i / 128]);
}

// one CTA per (by x bx) block
__global__ void __launch_bounds__(256) fp8_block_quant_kernel(const void* __restrict__ w, int dtype, int64_t rows,
                                                              int64_t cols, int by, int bx,
                                                              uint8_t* __restrict__ codes,
                                                              float* __restrict__ scales) {
  const int64_t r0 = (int64_t)blockIdx.y * by, c0 = (int64_t)blockIdx.x * bx;
  const int nr = (int)min((int64_t)by, rows - r0), nc = (int)min((int64_t)bx, cols - c0);
  __shared__ float red[8];
  float m = 0.f;
  for (int i = threadIdx.x; i < nr * nc; i += blockDim.x)
    m = fmaxf(m, fabsf(load_as_float(w, dtype, (r0 + i / nc) * cols + c0 + i % nc)));
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  m = red[0];
  for (int i = 1; i < 8; ++i) m = fmaxf(m, red[i]);
  const float scale = m > 0.f ? __fdiv_rn(m, 448.f) : 1e-12f;
  if (threadIdx.x == 0) scales[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = scale;
  for (int i = threadIdx.x; i < nr * nc; i += blockDim.x) {
    const int64_t idx = (r0 + i / nc) * cols + c0 + i % nc;
    const float q = fminf(fmaxf(__fdiv_rn(load_as_float(w, dtype, idx), scale), -448.f), 448.f);
    codes[idx] = f32_to_e4m3(q);
  }
}

__global__ void __launch_bounds__(256) fp8_block_dequant_kernel(const uint8_t* __restrict__ codes,
                                                                const float* __restrict__ scales, int64_t rows,
                                                                int64_t cols, int by, int bx, int64_t sc_cols,
                                                                void* __restrict__ out, int dtype) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * cols) return;
  const int64_t r = i / cols, c = i % cols;
  store_from_float(out, dtype, i, e4m3_to_f32(codes[i]) * scales[(r / by) * sc_cols + c / bx]);
}

int32_t launch_fp8_vector_quant(const void* x, int x_dtype, int64_t n, uint8_t* codes, float* scales,
                                cudaStream_t stream) {
  const int64_t groups = n / 128;
  if (groups == 0) return HQ_OK;
  fp8_vector_quant_kernel<<<(unsigned)((groups + 7) / 8), 256, 0, stream>>>(x, x_dtype, groups, codes, scales);
  return cudaGetLastError() == cudaSuccess ? HQ_OK : HQ_ERR_CUDA;
}
// four consecutive elements starting at element index i (a multiple of 4; rows are 16-byte aligned)
__device__ __forceinline__ void load4_as_float(const void* p, int dtype, int64_t i, float (&v)[4]) {
  if (dtype == HQ_DT_F32) {
    const float4 t = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + i);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else {
    const uint2 t = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(p) + i);
    if (dtype == HQ_DT_BF16) {
      v[0] = __uint_as_float(t.x << 16); v[1] = __uint_as_float(t.x & 0xFFFF0000u);
      v[2] = __uint_as_float(t.y << 16); v[3] = __uint_as_float(t.y & 0xFFFF0000u);
    } else {
      const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&t.x));
      const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&t.y));
      v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
  }
}

// The same 1 x 128 quantizer over rows that are looked up first (token order -> expert-sorted order).  Feeds the
// FP8 expert GEMM, whose operand boxes need whole sorted rows.  A warp quantizes U x 256 columns of a row, the eight warps of a
// block the same columns of eight rows: a lane owns 8 consecutive values of each 256, a 128-column group is 16 lanes.
// Latency bounds it: the chain row number -> values -> maximum -> codes, so all U loads are issued before anything is used
// (the type is a template argument: a branch on it between the loads had them one after the other), a division per group and
// not per value, no 64-bit division for the item.  4,096 x 7,168 bf16: 32.6 -> 24.8 us
// (88 MB: 13 us), 32 rows 2.3 -> 1.5.
template <typename T, int U>
__global__ void __launch_bounds__(256) fp8_quant_rows_kernel(const T* __restrict__ x, int64_t x_stride,
                                                             const int32_t* __restrict__ row_map,
                                                             const int32_t* __restrict__ n_valid, int64_t n_rows,
                                                             int kgroups, int spans, uint8_t* __restrict__ codes,
                                                             float* __restrict__ scales) {
  pdl_launch_dependents();
  pdl_wait();
  const unsigned eight = blockIdx.x / (unsigned)spans;
  const int span = (int)(blockIdx.x - eight * (unsigned)spans);
  const int64_t row = (int64_t)eight * 8 + (threadIdx.x >> 5);
  const int64_t limit = n_valid != nullptr ? min((int64_t)*n_valid, n_rows) : n_rows;   // rows the map is defined for
  if (row >= limit) return;
  const int lane = threadIdx.x & 31;
  const int64_t src_row = row_map != nullptr ? (int64_t)row_map[row] : row;
  const int k = kgroups * 128, c0 = span * (256 * U) + lane * 8;
  uint4 raw[U][sizeof(T) / 2];
#pragma unroll
  for (int j = 0; j < U; ++j)
    if (c0 + 256 * j < k) load8(x + src_row * x_stride + c0 + 256 * j, raw[j]);
#pragma unroll
  for (int j = 0; j < U; ++j) {
    const int col = c0 + 256 * j;
    const bool in = col < k;                          // the same for the 16 lanes of a group
    float v[8], m = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i] = in ? elem8<T>(raw[j], i) : 0.f;
      m = fmaxf(m, fabsf(v[i]));
    }
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
    if (!in) continue;
    const float scale = m > 0.f ? __fdiv_rn(m, 448.f) : 1e-12f;
    const DivideBy by = divide_by(scale);
    if (by.fast) {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = by.quick(v[i]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = __fdiv_rn(v[i], scale);
    }
    uint32_t packed[2];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = fminf(fmaxf(v[i], -448.f), 448.f);
#pragma unroll
    for (int h = 0; h < 2; ++h)
      packed[h] = (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(v[4 * h], v[4 * h + 1]), __NV_SATFINITE, __NV_E4M3) |
                  ((uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(v[4 * h + 2], v[4 * h + 3]), __NV_SATFINITE, __NV_E4M3) << 16);
    *reinterpret_cast<uint2*>(codes + row * k + col) = make_uint2(packed[0], packed[1]);
    if ((lane & 15) == 0) scales[row * kgroups + col / 128] = scale;
  }
}
template <typename T, int U>
static int32_t launch_fq(const void* x, int64_t x_stride, const int32_t* row_map, const int32_t* n_valid, int64_t n_rows, int64_t k,
                         uint8_t* codes, float* scales, cudaStream_t stream) {
  const int spans = (int)((k + 256 * U - 1) / (256 * U));
  return launch_pdl(fp8_quant_rows_kernel<T, U>, dim3((unsigned)((n_rows + 7) / 8 * spans)), 256, 0, stream, 1, (const T*)x, x_stride,
                    row_map, n_valid, n_rows, (int)(k / 128), spans, codes, scales);
}
int32_t launch_fp8_quant_rows(const void* x, int x_dtype, int64_t x_stride, const int32_t* row_map,
                              const int32_t* n_valid, int64_t n_rows, int64_t k, uint8_t* codes, float* scales,
                              cudaStream_t stream) {
  if (n_rows == 0) return HQ_OK;
  // four loads a warp where that leaves half of the chip's warps (64 an SM) or more something to do.  One load against four, bf16:
  // 512 x 7,168 (14,336 loads) 4.9 us against 5.8, 1,024 x 7,168 (28,672) 8.9 against 8.2, 4,096 x 7,168 30.8 against 24.8
  const bool wide = n_rows * (k / 256) >= 2 * (int64_t)sm_count() * 64;
#define HQ_FQ(T) \
  return wide ? launch_fq<T, 4>(x, x_stride, row_map, n_valid, n_rows, k, codes, scales, stream) \
              : launch_fq<T, 1>(x, x_stride, row_map, n_valid, n_rows, k, codes, scales, stream)
  if (x_dtype == HQ_DT_F32) HQ_FQ(float);
  if (x_dtype == HQ_DT_F16) HQ_FQ(__half);
  HQ_FQ(__nv_bfloat16);
#undef HQ_FQ
}

int32_t launch_fp8_vector_dequant(const uint8_t* codes, const float* scales, int64_t n, void* out, int out_dtype,
                                  cudaStream_t stream) {
  if (n == 0) return HQ_OK;
  fp8_vector_dequant_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(codes, scales, n, out, out_dtype);
  return cudaGetLastError() == cudaSuccess ? HQ_OK : HQ_ERR_CUDA;
}
int32_t launch_fp8_block_quant(const void* w, int w_dtype, int64_t rows, int64_t cols, int by, int bx,
                               uint8_t* codes, float* scales, cudaStream_t stream) {
  if (rows == 0 || cols == 0) return HQ_OK;
  dim3 grid((unsigned)((cols + bx - 1) / bx), (unsigned)((rows + by - 1) / by));
  fp8_block_quant_kernel<<<grid, 256, 0, stream>>>(w, w_dtype, rows, cols, by, bx, codes, scales);
  return cudaGetLastError() == cudaSuccess ? HQ_OK : HQ_ERR_CUDA;
}
int32_t launch_fp8_block_dequant(const uint8_t* codes, const float* scales, int64_t rows, int64_t cols, int by,
                                 int bx, void* out, int out_dtype, cudaStream_t stream) {
  if (rows == 0 || cols == 0) return HQ_OK;
  const int64_t n = rows * cols;
  fp8_block_dequant_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(codes, scales, rows, cols, by, bx,
                                                                           (cols + bx - 1) / bx, out, out_dtype);
  return cudaGetLastError() == cudaSuccess ? HQ_OK : HQ_ERR_CUDA;
}

// ---- dtype conversion (hosts holding bf16 / f32 activations cast once before a prefill-sized call) -------
// Eight elements per thread (16-byte accesses on the 16-bit side).  A finite value beyond the f16 range is clamped
// to +-65504 instead of becoming inf, and the call says so through the status word: the tensor-core kernels
// multiply in f16, which the reference's bf16 / f32 activation paths do not, so the caller has to know.
__global__ void __launch_bounds__(256) convert_kernel(const void* __restrict__ src, int src_dtype,
                                                      void* __restrict__ dst, int dst_dtype, int64_t n, int vec_ok,
                                                      int32_t* __restrict__ status) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i0 >= n) return;
  float v[8];
  const bool full = vec_ok && i0 + 8 <= n;
  if (full) {
    load4_as_float(src, src_dtype, i0, *reinterpret_cast<float(*)[4]>(&v[0]));
    load4_as_float(src, src_dtype, i0 + 4, *reinterpret_cast<float(*)[4]>(&v[4]));
  } else {
    for (int j = 0; j < 8; ++j) v[j] = i0 + j < n ? load_as_float(src, src_dtype, i0 + j) : 0.f;
  }
  if (dst_dtype == HQ_DT_F16 && src_dtype != HQ_DT_F16) {
    bool clamped = false;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float a = fabsf(v[j]);
      if (a > 65504.f && a <= 3.4028235e38f) {       // finite and out of range (inf / NaN pass through)
        v[j] = copysignf(65504.f, v[j]);
        clamped = true;
      }
    }
    if (clamped) report_status(status, HQ_DEV_F16_RANGE, 900);
  }
  if (full && dst_dtype != HQ_DT_F32) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (dst_dtype == HQ_DT_F16) {
        w[j] = pack_half2(v[2 * j], v[2 * j + 1]);
      } else {
        __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        w[j] = *reinterpret_cast<uint32_t*>(&b);
      }
    }
    *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(dst) + i0) = make_uint4(w[0], w[1], w[2], w[3]);
  } else if (full) {
    float4* o = reinterpret_cast<float4*>(reinterpret_cast<float*>(dst) + i0);
    o[0] = make_float4(v[0], v[1], v[2], v[3]);
    o[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    for (int j = 0; j < 8 && i0 + j < n; ++j) store_from_float(dst, dst_dtype, i0 + j, v[j]);
  }
}

int32_t launch_convert(const void* src, int src_dtype, void* dst, int dst_dtype, int64_t n, int32_t* status,
                       cudaStream_t stream) {
  if (n == 0) return HQ_OK;
  const int64_t threads = (n + 7) / 8;
  const int vec_ok = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0;
  return launch_pdl(convert_kernel, dim3((unsigned)((threads + 255) / 256)), 256, 0, stream, 1, src, src_dtype, dst, dst_dtype,
                    n, vec_ok, status);
}

// a finite value beyond the f16 range is clamped to +-65504 (inf / NaN pass through)
__device__ __forceinline__ uint4 f32x8_to_f16x8(float (&v)[8], bool& clamped) {
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float a = fabsf(v[j]);
    if (a > 65504.f && a <= 3.4028235e38f) {
      v[j] = copysignf(65504.f, v[j]);
      clamped = true;
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) w[j] = pack_half2(v[2 * j], v[2 * j + 1]);
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ uint4 bf16x8_to_f16x8(uint4 r, bool& clamped) {
  float v[8] = {__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xFFFF0000u), __uint_as_float(r.y << 16),
                __uint_as_float(r.y & 0xFFFF0000u), __uint_as_float(r.z << 16), __uint_as_float(r.z & 0xFFFF0000u),
                __uint_as_float(r.w << 16), __uint_as_float(r.w & 0xFFFF0000u)};
  return f32x8_to_f16x8(v, clamped);
}

// Rows x[row_map[r]] as f16 in the order of the map (expert-sorted rows for the dequantizing GEMM, which then copies its
// token tiles as whole boxes instead of gathering 16-byte pieces).  Rows at or past *n_valid are left unwritten.  Bytes:
// rows * k * 2 written; the sources are re-read through L2, once per slot of a token.
__global__ void __launch_bounds__(256) gather_rows_f16_kernel(const void* __restrict__ x, int dtype, int64_t x_stride,
                                                              const int32_t* __restrict__ row_map,
                                                              const int32_t* __restrict__ n_valid, int64_t n_rows, int k8,
                                                              uint16_t* __restrict__ out, int32_t* __restrict__ status) {
  pdl_launch_dependents();
  pdl_wait();
  // a warp per row, four 8-element chunks of it in flight per lane
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= n_rows || (n_valid != nullptr && row >= (int64_t)*n_valid)) return;
  const int64_t src = (int64_t)row_map[row] * x_stride;
  uint16_t* const dst = out + row * ((int64_t)k8 * 8);
  bool clamped = false;
  for (int c0 = threadIdx.x & 31; c0 < k8; c0 += 128) {
    if (dtype != HQ_DT_F32) {
      uint4 v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (c0 + 32 * i < k8) v[i] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(x) + src) + c0 + 32 * i);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (c0 + 32 * i < k8) {
          if (dtype == HQ_DT_BF16) v[i] = bf16x8_to_f16x8(v[i], clamped);
          *(reinterpret_cast<uint4*>(dst) + c0 + 32 * i) = v[i];
        }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (c0 + 32 * i < k8) {
          float v[8];
          load4_as_float(x, dtype, src + 8 * (c0 + 32 * i), *reinterpret_cast<float(*)[4]>(&v[0]));
          load4_as_float(x, dtype, src + 8 * (c0 + 32 * i) + 4, *reinterpret_cast<float(*)[4]>(&v[4]));
          *(reinterpret_cast<uint4*>(dst) + c0 + 32 * i) = f32x8_to_f16x8(v, clamped);
        }
    }
  }
  if (clamped) report_status(status, HQ_DEV_F16_RANGE, 901);
}

int32_t launch_gather_rows_f16(const void* x, int dtype, int64_t x_stride, const int32_t* row_map, const int32_t* n_valid,
                               int64_t n_rows, int64_t k, void* out, int32_t* status, cudaStream_t stream) {
  if (n_rows == 0) return HQ_OK;
  return launch_pdl(gather_rows_f16_kernel, dim3((unsigned)((n_rows + 7) / 8)), 256, 0, stream, 1, x, dtype, x_stride, row_map,
                    n_valid, n_rows, (int)(k / 8), (uint16_t*)out, status);
}

// ---- gated activations --------------------------------------------------------------
__device__ __forceinline__ float gated_act(float g, float u, const hq_act_args& a) {
  if (a.act == HQ_ACT_GPTOSS) {
    g = fminf(g, a.limit);
    u = fminf(fmaxf(u, -a.limit), a.limit);
    return (u + 1.f) * (g / (1.f + expf(-a.alpha * g)));
  }
  if (a.has_limit) {
    g = fminf(g, a.limit);
    u = fminf(fmaxf(u, -a.limit), a.limit);
  }
  return (g / (1.f + expf(-g))) * u;
}

__global__ void __launch_bounds__(256) gated_act_kernel(const void* __restrict__ gate, const void* __restrict__ up,
                                                        int dtype, int64_t n, int interleaved, hq_act_args a,
                                                        void* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float g, u;
  if (interleaved) {
    g = load_as_float(gate, dtype, 2 * i);
    u = load_as_float(gate, dtype, 2 * i + 1);
  } else {
    g = load_as_float(gate, dtype, i);
    u = load_as_float(up, dtype, i);
  }
  store_from_float(out, dtype, i, gated_act(g, u, a));
}

int32_t launch_gated_act(const void* gate, const void* up, int dtype, int64_t n, int interleaved,
                         const hq_act_args& act, void* out, cudaStream_t stream) {
  if (n == 0) return HQ_OK;
  gated_act_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(gate, up, dtype, n, interleaved, act, out);
  return cudaGetLastError() == cudaSuccess ? HQ_OK : HQ_ERR_CUDA;
}

// Gated activation of a [rows, 2 * width] matrix {gate | up} followed by the 1 x 128 FP8 quantizer: the expert
// intermediate goes to the FP8 down projection without a 16-bit round trip through memory.
__global__ void __launch_bounds__(256) fp8_gated_quant_rows_kernel(const void* __restrict__ gu, int dtype,
                                                                   int64_t n_rows, int width, hq_act_args act,
                                                                   uint8_t* __restrict__ codes,
                                                                   float* __restrict__ scales) {
  const int kgroups = width / 128;
  const int64_t grp = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (grp >= n_rows * kgroups) return;
  const int lane = threadIdx.x & 31;
  const int64_t row = grp / kgroups;
  const int g = (int)(grp - row * kgroups);
  const int64_t src = row * 2 * width + g * 128 + lane * 4;
  float gv[4], uv[4], v[4];
  load4_as_float(gu, dtype, src, gv);
  load4_as_float(gu, dtype, src + width, uv);
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = gated_act(gv[i], uv[i], act);
  float m = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
  const float scale = m > 0.f ? __fdiv_rn(m, 448.f) : 1e-12f;
  uint32_t packed = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float q = fminf(fmaxf(__fdiv_rn(v[i], scale), -448.f), 448.f);
    packed |= (uint32_t)f32_to_e4m3(q) << (8 * i);
  }
  *reinterpret_cast<uint32_t*>(codes + grp * 128 + lane * 4) = packed;
  if (lane == 0) scales[grp] = scale;
}

int32_t launch_fp8_gated_quant_rows(const void* gu, int dtype, int64_t n_rows, int64_t width, const hq_act_args& act,
                                    uint8_t* codes, float* scales, cudaStream_t stream) {
  const int64_t groups = n_rows * (width / 128);
  if (groups == 0) return HQ_OK;
  fp8_gated_quant_rows_kernel<<<(unsigned)((groups + 7) / 8), 256, 0, stream>>>(gu, dtype, n_rows, (int)width, act,
                                                                               codes, scales);
  return cudaGetLastError() == cudaSuccess ? HQ_OK : HQ_ERR_CUDA;
}

}  // namespace hq
