// Expansion of the quantized weight formats to f16 operands of the tensor cores, and the tcgen05 wrappers, shared by
// the translation units of the dequantizing GEMM (hq_dq_gemm.cuh).
#pragma once
#include "hq_common.cuh"
#include "hq_kernels.h"

namespace hq {

constexpr int kTileM = 128;   // weight rows per tile (tensor-memory lanes)

// ---- tcgen05 wrappers -----------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory operand descriptor: K-major tile of 128-byte rows, 128-byte swizzle,
// 8-row groups 1024 bytes apart, descriptor version 1 (sm_100).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);         // start address, 16-byte units
  d |= (uint64_t)1 << 16;                              // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;                    // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                              // descriptor version
  d |= (uint64_t)2 << 61;                              // SWIZZLE_128B
  return d;
}
// kind::f16 instruction descriptor: f32 accumulate, f16 x f16, both K-major, M = 128
// (both operands must have the same 16-bit format: f16 weights beside bf16 activations in one instruction
// raise an illegal-instruction error on B200, so bf16 activations are converted while their tile is written)
__device__ __forceinline__ uint32_t make_idesc_f16(int tile_n) {
  return (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(tile_n >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
}
// byte offset of 16-byte chunk `c` (0..7) of row `r` inside a swizzled K-major operand tile of 64 f16 columns
__device__ __forceinline__ uint32_t swz(int r, int c) {
  return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4));
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- expansion of 16 consecutive weights: the raw fields picked out of a block (hq_dq_gemm.cuh) -> eight f16 pairs in
// natural k order
struct RawA {
  uint4 hdr;          // Q8_0, Q4_0 ..: .x = fifth payload word, .y = m (f16 bits); Q6_K: words of high bits; Q3_K: of hmask
  uint4 q;            // FP8: 16 codes; MXFP4: .x/.y = 8 nibble bytes; else payload words
  uint32_t aux;       // FP8: relative block scale (f32 bits); MXFP4: e8m0 byte; Q8_0, Q4_0 ..: d (f16 bits) | shift << 16
                      // [| half block << 24]; Q6_K, Q3_K: bit pair [| hmask bit << 8]
  uint4 ext;          // Q6_K, Q3_K: .x / .y = fifth words of q / hdr, .z = d (f16 bits) | scale << 16, .w = shifts (of q |
                      // of hdr << 8); Q5_0 / Q5_1: .x = the 16 fifth bits of this half block
};

// Q4_K, Q5_K, Q2_K: w = d * s * code - dmin * m with the integer scale s and minimum m of the sub-block.  A code byte
// becomes the f16 number p = 1024 + code with one permute (bytes {code, 0x64}); s * code = fma(p, s, -1024 s) is an
// exact f16 integer (at most 63 x 31), d multiplies it as it is stored, and dmin * m is split into a leading f16 and its
// remainder: w carries only the two roundings of weight-sized quantities.
struct AffineH2 {
  __half2 s, cs, d, mh, ml;
};
__device__ __forceinline__ AffineH2 make_affine(uint32_t d_dmin, uint32_t s, uint32_t m) {
  AffineH2 r;
  const __half2 one = __halves2half2(__ushort_as_half(0x6400), __ushort_as_half(0x6400));   // 1024
  const uint32_t sb = (s * 0x00010001u) | 0x64006400u;
  r.s = __hsub2(*reinterpret_cast<const __half2*>(&sb), one);
  r.cs = __hneg2(__hmul2(r.s, one));
  const uint32_t db = __byte_perm(d_dmin, 0u, 0x1010);
  r.d = *reinterpret_cast<const __half2*>(&db);
  const float m1 = -half_bits_to_float(d_dmin >> 16) * (__uint_as_float(0x4B000000u | m) - 8388608.f);
  const __half mh = __float2half_rn(m1);
  r.mh = __half2half2(mh);
  r.ml = __float2half2_rn(m1 - __half2float(mh));
  return r;
}
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t b) { return *reinterpret_cast<const __half2*>(&b); }
// The same of two sub-blocks at a time, their scales and minima the bytes of s4 / m4 that `pick` (a permute selector that pairs
// each with 0x64) names: words {d | dmin, ...} -> {d twice, scales, minus the minima, their remainders}, a sub-block per half.
// HIGH: the second sub-block's codes come 16 times too large, as high nibbles where they lie, and its scale is a sixteenth.
// All exact but the rounding of dmin * m to its leading part, as in make_affine; 11 instructions instead of 2 x 15.
template <bool HIGH>
__device__ __forceinline__ void affine_pair(uint32_t* w, uint32_t s4, uint32_t m4, uint32_t pick) {
  const __half2 one = bits_h2(0x64006400u);      // 1024
  __half2 s = __hsub2(bits_h2(__byte_perm(s4, 0x64646464u, pick)), one);
  if (HIGH) s = __hmul2(s, bits_h2(0x2C003C00u));      // 1, 1 / 16
  const __half2 m = __hsub2(bits_h2(__byte_perm(m4, 0x64646464u, pick)), one);
  const __half2 dmin = __hneg2(bits_h2(__byte_perm(w[0], 0u, 0x3232)));
  const __half2 mh = __hmul2(dmin, m);
  w[0] = __byte_perm(w[0], 0u, 0x1010);
  w[1] = h2_bits(s);
  w[2] = h2_bits(mh);
  w[3] = h2_bits(__hfma2(dmin, m, __hneg2(mh)));
}
__device__ __forceinline__ AffineH2 affine_of(const uint32_t* w, int i) {
  const uint32_t pick = i ? 0x3232u : 0x1010u;
  AffineH2 r;
  r.s = bits_h2(__byte_perm(w[1], 0u, pick));
  r.cs = __hmul2(r.s, bits_h2(0xE400E400u));      // -1024
  r.d = bits_h2(w[0]);
  r.mh = bits_h2(__byte_perm(w[2], 0u, pick));
  r.ml = bits_h2(__byte_perm(w[3], 0u, pick));
  return r;
}
// four code bytes -> two f16 pairs
__device__ __forceinline__ void affine4(const AffineH2& a, uint32_t codes, uint32_t& o01, uint32_t& o23) {
  uint32_t p01 = __byte_perm(codes, 0x64646464u, 0x4140);
  uint32_t p23 = __byte_perm(codes, 0x64646464u, 0x4342);
  __half2 w01 = __hfma2(*reinterpret_cast<__half2*>(&p01), a.s, a.cs);
  __half2 w23 = __hfma2(*reinterpret_cast<__half2*>(&p23), a.s, a.cs);
  w01 = __hadd2(__hfma2(w01, a.d, a.mh), a.ml);
  w23 = __hadd2(__hfma2(w23, a.d, a.mh), a.ml);
  o01 = *reinterpret_cast<uint32_t*>(&w01);
  o23 = *reinterpret_cast<uint32_t*>(&w23);
}
// the 6-bit scales (s) and minima (m) of sub-blocks 4 hi .. 4 hi + 3 of a Q4_K / Q5_K header, four to a word
__device__ __forceinline__ void k_scales(uint32_t y, uint32_t z, uint32_t w, bool hi, uint32_t& s, uint32_t& m) {
  s = hi ? (w & 0x0F0F0F0Fu) | ((y >> 2) & 0x30303030u) : y & 0x3F3F3F3Fu;
  m = hi ? ((w >> 4) & 0x0F0F0F0Fu) | ((z >> 2) & 0x30303030u) : z & 0x3F3F3F3Fu;
}

// Q8_0: w = d * q.  Bytes q + 128 become the f16 pair (1024 + u0, 1024 + u1) with one permute, 1152 is subtracted
// exactly, and the product with the block's f16 d is rounded once to f16 (relative error <= 2^-11 per weight).
__device__ __forceinline__ void emit_q8_0(const RawA& r, uint32_t (&out)[8]) {
  const uint32_t sh = (r.aux >> 16) & 31u;          // 0 or 16
  const uint32_t raw[5] = {r.q.x, r.q.y, r.q.z, r.q.w, r.hdr.x};
  const uint32_t d16 = r.aux & 0xFFFFu;
  const uint32_t dd = d16 | (d16 << 16);
  const __half2 d2 = *reinterpret_cast<const __half2*>(&dd);
  const uint32_t off = 0x64806480u;                  // f16 1152 twice
  const __half2 o2 = *reinterpret_cast<const __half2*>(&off);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w = __funnelshift_r(raw[i], raw[i + 1], sh) ^ 0x80808080u;
    uint32_t p01 = __byte_perm(w, 0x64646464u, 0x4140);
    uint32_t p23 = __byte_perm(w, 0x64646464u, 0x4342);
    __half2 w01 = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&p01), o2), d2);
    __half2 w23 = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&p23), o2), d2);
    out[2 * i] = *reinterpret_cast<uint32_t*>(&w01);
    out[2 * i + 1] = *reinterpret_cast<uint32_t*>(&w23);
  }
}

// Q6_K: w = d * scale * (q - 32).  The 6-bit codes are assembled bytewise (nibble | two high bits << 4), become the
// f16 pair (1024 + q0, 1024 + q1) with one permute, 1056 is subtracted exactly, and the product with d * scale
// (computed in f32, rounded to f16) is rounded once more: two roundings of 2^-11 per weight.
__device__ __forceinline__ void emit_q6_k(const RawA& r, uint32_t (&out)[8]) {
  const uint32_t shl = r.ext.w & 31u, shh = (r.ext.w >> 8) & 31u;   // 0 or 16
  const uint32_t j = r.aux;
  const uint32_t lo[5] = {r.q.x, r.q.y, r.q.z, r.q.w, r.ext.x};
  const uint32_t hi[5] = {r.hdr.x, r.hdr.y, r.hdr.z, r.hdr.w, r.ext.y};
  const float ds = half_bits_to_float(r.ext.z & 0xFFFFu) * (float)(int)(int8_t)((r.ext.z >> 16) & 0xFFu);
  const __half2 ds2 = __float2half2_rn(ds);
  const uint32_t off = 0x64206420u;                  // f16 1056 twice
  const __half2 o2 = *reinterpret_cast<const __half2*>(&off);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t lw = __funnelshift_r(lo[i], lo[i + 1], shl);
    const uint32_t hw = __funnelshift_r(hi[i], hi[i + 1], shh);
    const uint32_t nib = (lw >> (2 * (j & 2))) & 0x0F0F0F0Fu;
    const uint32_t w6 = nib | (((hw >> (2 * j)) & 0x03030303u) << 4);
    uint32_t p01 = __byte_perm(w6, 0x64646464u, 0x4140);
    uint32_t p23 = __byte_perm(w6, 0x64646464u, 0x4342);
    __half2 w01 = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&p01), o2), ds2);
    __half2 w23 = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&p23), o2), ds2);
    out[2 * i] = *reinterpret_cast<uint32_t*>(&w01);
    out[2 * i + 1] = *reinterpret_cast<uint32_t*>(&w23);
  }
}

// Q4_0: w = d * (q - 8); Q5_0: w = d * (q - 16); Q4_1 / Q5_1: w = d * q + m; q = nibble [| fifth bit << 4].  The
// codes become the f16 pair (1024 + q0, 1024 + q1) with one permute, 1024 + zero point is subtracted exactly, and the
// product with the block's f16 d (plus m, in one fused multiply-add) is rounded once to f16.
template <int FMT>
__device__ __forceinline__ void emit_q4_0_q5_0(const RawA& r, uint32_t (&out)[8]) {
  constexpr bool FIVE = FMT == HQ_FMT_Q5_0 || FMT == HQ_FMT_Q5_1;
  constexpr bool MIN = FMT == HQ_FMT_Q4_1 || FMT == HQ_FMT_Q5_1;
  const uint32_t sh = (r.aux >> 16) & 31u;           // 0 or 16
  const uint32_t half = (r.aux >> 24) & 1u;
  const uint32_t raw[5] = {r.q.x, r.q.y, r.q.z, r.q.w, r.hdr.x};
  const uint32_t d16 = r.aux & 0xFFFFu;
  const uint32_t dd = d16 | (d16 << 16);
  const __half2 d2 = *reinterpret_cast<const __half2*>(&dd);
  const uint32_t m16 = MIN ? (r.hdr.y & 0xFFFFu) : 0u;
  const uint32_t mm = m16 | (m16 << 16);
  const __half2 m2 = *reinterpret_cast<const __half2*>(&mm);
  const uint32_t off = MIN ? 0x64006400u : (FMT == HQ_FMT_Q4_0 ? 0x64086408u : 0x64106410u);   // f16 1024 + zero, twice
  const __half2 o2 = *reinterpret_cast<const __half2*>(&off);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w = __funnelshift_r(raw[i], raw[i + 1], sh);
    uint32_t vm = (half ? (w >> 4) : w) & 0x0F0F0F0Fu;
    if (FIVE)   // four bits -> bit 4 of four bytes: x * 0x00204081 puts bit c of x at bit 8 c
      vm |= ((((r.ext.x >> (4 * i)) & 0xFu) * 0x00204081u) & 0x01010101u) << 4;
    uint32_t p01 = __byte_perm(vm, 0x64646464u, 0x4140);
    uint32_t p23 = __byte_perm(vm, 0x64646464u, 0x4342);
    const __half2 q01 = __hsub2(*reinterpret_cast<__half2*>(&p01), o2), q23 = __hsub2(*reinterpret_cast<__half2*>(&p23), o2);
    __half2 w01 = MIN ? __hfma2(q01, d2, m2) : __hmul2(q01, d2);
    __half2 w23 = MIN ? __hfma2(q23, d2, m2) : __hmul2(q23, d2);
    out[2 * i] = *reinterpret_cast<uint32_t*>(&w01);
    out[2 * i + 1] = *reinterpret_cast<uint32_t*>(&w23);
  }
}

// Q3_K: w = d * (scale - 32) * (q - 4), q = two code bits | hmask bit << 2: as emit_q6_k with 1028 subtracted.
__device__ __forceinline__ void emit_q3_k(const RawA& r, uint32_t (&out)[8]) {
  const uint32_t shl = r.ext.w & 31u, shh = (r.ext.w >> 8) & 31u;   // 0 or 16
  const uint32_t j = r.aux & 3u, hbit = (r.aux >> 8) & 7u;
  const uint32_t lo[5] = {r.q.x, r.q.y, r.q.z, r.q.w, r.ext.x};
  const uint32_t hi[5] = {r.hdr.x, r.hdr.y, r.hdr.z, r.hdr.w, r.ext.y};
  const float ds = half_bits_to_float(r.ext.z & 0xFFFFu) * (float)((int)((r.ext.z >> 16) & 0xFFu) - 32);
  const __half2 ds2 = __float2half2_rn(ds);
  const uint32_t off = 0x64046404u;                  // f16 1028 twice
  const __half2 o2 = *reinterpret_cast<const __half2*>(&off);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t lw = __funnelshift_r(lo[i], lo[i + 1], shl);
    const uint32_t hw = __funnelshift_r(hi[i], hi[i + 1], shh);
    const uint32_t w3 = ((lw >> (2 * j)) & 0x03030303u) | (((hw >> hbit) & 0x01010101u) << 2);
    uint32_t p01 = __byte_perm(w3, 0x64646464u, 0x4140);
    uint32_t p23 = __byte_perm(w3, 0x64646464u, 0x4342);
    __half2 w01 = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&p01), o2), ds2);
    __half2 w23 = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&p23), o2), ds2);
    out[2 * i] = *reinterpret_cast<uint32_t*>(&w01);
    out[2 * i + 1] = *reinterpret_cast<uint32_t*>(&w23);
  }
}

// e4m3 -> f16 is exact; the block's scale relative to the largest scale of its 128-row block (<= 1) is folded
// in here, the largest scale itself multiplies the accumulator in the epilogue.
__device__ __forceinline__ void emit_fp8(const RawA& r, uint32_t (&out)[8]) {
  const uint32_t w[4] = {r.q.x, r.q.y, r.q.z, r.q.w};
  const __half2 r2 = __float2half2_rn(__uint_as_float(r.aux));
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t lo, hi;
    asm("{\n"
        ".reg .b16 l, h;\n"
        "mov.b32 {l, h}, %2;\n"
        "cvt.rn.f16x2.e4m3x2 %0, l;\n"
        "cvt.rn.f16x2.e4m3x2 %1, h;\n"
        "}\n"
        : "=r"(lo), "=r"(hi)
        : "r"(w[i]));
    __half2 l2 = __hmul2(*reinterpret_cast<__half2*>(&lo), r2);
    __half2 h2 = __hmul2(*reinterpret_cast<__half2*>(&hi), r2);
    out[2 * i] = *reinterpret_cast<uint32_t*>(&l2);
    out[2 * i + 1] = *reinterpret_cast<uint32_t*>(&h2);
  }
}

// MXFP4: e2m1 pairs -> f16x2 (hardware conversion, low nibble = even element = low half), times 2^(e-127) as
// an exact f16 power of two.  e = 0 decodes to a zero scale (the reference's table builds the scale from the
// bits e << 23).  The f16 operand covers block scales 2^-14 .. 2^13 (e = 113 .. 140); a block outside that
// range is expanded as zero and the caller raises HQ_DEV_SCALE_RANGE, so a bank with such blocks has to stay on
// the decode kernel, which applies the scale in f32.
__device__ __forceinline__ bool emit_mxfp4(const RawA& r, uint32_t (&out)[8]) {
  const uint32_t e = r.aux;
  const bool in_range = (e == 0) || (e >= 113 && e <= 140);   // 2^-14 .. 2^13: products stay finite in f16
  const uint32_t ef = (e >= 113 && e <= 140) ? (e - 112) : 0u;  // f16 exponent field of 2^(e-127)
  const uint32_t sc16 = ef << 10;
  const uint32_t sc2 = sc16 | (sc16 << 16);
  const __half2 s2 = *reinterpret_cast<const __half2*>(&sc2);
  const uint32_t w[2] = {r.q.x, r.q.y};
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    uint32_t h[4];
    asm("{\n"
        ".reg .b8 b0, b1, b2, b3;\n"
        "mov.b32 {b0, b1, b2, b3}, %4;\n"
        "cvt.rn.f16x2.e2m1x2 %0, b0;\n"
        "cvt.rn.f16x2.e2m1x2 %1, b1;\n"
        "cvt.rn.f16x2.e2m1x2 %2, b2;\n"
        "cvt.rn.f16x2.e2m1x2 %3, b3;\n"
        "}\n"
        : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
        : "r"(w[i]));
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      __half2 v = __hmul2(*reinterpret_cast<__half2*>(&h[b]), s2);
      out[4 * i + b] = *reinterpret_cast<uint32_t*>(&v);
    }
  }
  return in_range;
}
__device__ __forceinline__ float gg_gated(float g, float u, const hq_act_args& a) {
  if (a.act == HQ_ACT_GPTOSS) {
    g = fminf(g, a.limit);
    u = fminf(fmaxf(u, -a.limit), a.limit);
    return (u + 1.f) * __fdividef(g, 1.f + __expf(-a.alpha * g));
  }
  if (a.has_limit) {
    g = fminf(g, a.limit);
    u = fminf(fmaxf(u, -a.limit), a.limit);
  }
  return __fdividef(g, 1.f + __expf(-g)) * u;
}

}  // namespace hq
