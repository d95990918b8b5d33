// Dequantizing GEMM on the 5th-generation tensor cores, for more activation rows than a decode work item holds and for
// expert banks: out[rows of expert e] = act( x_rows . dequant(W[e])^T ).
//
// Orientation: tensor-memory lanes = 128 weight rows (MMA M), columns = tokens (MMA N, 16 .. 256).  A tile with few
// tokens then costs columns, which are cheap, and the token count of a tile is a run-time number: the last tile of an
// expert is as narrow as its rows need.  With a gate and an up bank a tile holds 64 features: lanes 16q .. 16q+15 of
// every 32-lane quarter q carry the gate rows, the next 16 lanes the up rows of the same features, so one MMA serves
// both banks and the gated activation pairs lanes 16 apart of one epilogue warp.
//
// One persistent CTA per SM, 28 or 32 warps:
//   warp 0       issues tcgen05.mma (A = expanded weights in tensor memory, B = tokens in shared memory)
//   warps 1-8    epilogue, two per lane quarter: tcgen05.ld, bias, gated activation, store
//   warp 9       raw weight bytes of 256 k x 128 rows into a second ring, as boxes
//   warps 10-11  the f16 activation rows into a ring of operand stages of two or four 64-k tiles: boxes when the rows are
//                in order (warp 10; warp 11 then takes every second raw stage), else gathered with cp.async
//   warps 12-15  (types whose rows are no multiple of 16 bytes apart only) raw bytes in 4-byte pieces with cp.async
//   last 16      expand: four groups of four warps; group c owns the 64 weights 64c .. of every 256-k stage, so where
//                its codes, scales and bits lie inside the block is a compile-time constant.  A thread owns one weight
//                row: it picks the bytes out of shared memory (row pitch = an odd number of 16-byte units: no bank
//                conflicts), expands 64 weights in registers and writes them to a ring of A stages in tensor memory
//                (tcgen05.st), so the expanded weights never pass through shared memory.
// What bounds it: narrow tiles, the expanding warps' issue slots (410-740 cycles per 128 x 64 weights) and, for FP8 and
// MXFP4, HBM (65,536 x 4,096 at 16 rows: FP8 55 us, 4.9 TB/s); wide tiles, the MMA (14,336 x 4,096 Q4_K at 2,048 rows:
// 212 us, 1.13 PFLOP/s).  The MMA, commit, arrival and copy instructions are issued by whole warps under an elected
// predicate: from a branch for one lane a tcgen05.mma costs 75 cycles and a commit 125, whatever the width.
//
// Split K: a problem with fewer tiles than SMs gives each tile to a cluster of CTAs, one K slice each; the slices'
// partial sums are exchanged through distributed shared memory (each CTA finishes a share of the tile's tokens) and
// added in rank order, so the result does not depend on timing and no scratch is needed.
//
// Every wait is bounded; after a time-out the status word is set, the copy warps issue nothing more and wait (bounded) for what
// they have issued, and the kernel reaches its normal exit.  The epilogue stores nothing behind a wait of its own or of the issuing
// warp that ran out; an expanding warp hands over what it has, so with the status word set no output is to be used.  No
// multicast, no peer memory.
#pragma once
#include <cuda.h>

#include "hq_dequant.cuh"
#include "hq_warp_issue.cuh"

namespace hq {

constexpr uint32_t kDqSpin = 1u << 16;       // polls of a wait, each suspended for a while
constexpr int kDqMaxTokens = 256;
constexpr int kDqExpandWarps = 16;
constexpr int kDqTokenWarps = 2;
constexpr int kDqEpilogueWarps = 8;     // two per lane quarter of tensor memory
constexpr int kDqSmem = 227 * 1024;

// Geometry of a 256-k stage of one weight row.  SB = bytes of 256 weights.  WIDE types start every stage of every row on
// a 16-byte boundary.  The others (Q6_K, Q3_K, Q2_K) do not: where the row pitch is a multiple of 16 bytes the copy
// starts at the 16-byte boundary at or below the block, the same distance in front of it in every row; else the rows are
// copied in 4-byte pieces from the 4-byte boundary at or below it, so only a misalignment of 0 or 2 bytes is left.
// PITCH = bytes of a row in shared memory (the width of the copied box), an odd number of 16-byte units, or 128 with the
// 128-byte swizzle (SWZ): either way a warp's 16-byte loads of one column of 32 rows meet no bank conflicts.
template <int FMT>
struct DqTraits;
#define HQ_DQ_TRAITS(F, SBV, WIDEV, PITCHV, SWZV)                                                    \
  template <>                                                                                        \
  struct DqTraits<F> {                                                                               \
    static constexpr int SB = SBV, PITCH = PITCHV;                                                   \
    static constexpr bool WIDE = WIDEV, SWZ = SWZV;                                                  \
    static constexpr int BOXES = SWZV ? SBV / 128 : 1;         /* copies per bank and stage */       \
    static constexpr int STAGE = 128 * PITCHV * BOXES;         /* bytes of a raw stage */            \
    static constexpr int CH = (SBV + 2 + 3) / 4;               /* 4-byte pieces per row */           \
    static constexpr int COPY_WARPS = WIDEV ? 0 : 4;                                                 \
    static constexpr int FIRST_EXPAND = 2 + kDqEpilogueWarps + kDqTokenWarps + COPY_WARPS;                              \
    static constexpr int THREADS = 32 * (FIRST_EXPAND + kDqExpandWarps);                             \
  };
HQ_DQ_TRAITS(HQ_FMT_Q8_0, 272, true, 272, false)
HQ_DQ_TRAITS(HQ_FMT_Q4_K, 144, true, 144, false)
HQ_DQ_TRAITS(HQ_FMT_FP8_BLOCK, 256, true, 128, true)
HQ_DQ_TRAITS(HQ_FMT_MXFP4, 128, true, 128, true)
HQ_DQ_TRAITS(HQ_FMT_Q6_K, 210, false, 240, false)
HQ_DQ_TRAITS(HQ_FMT_Q5_K, 176, true, 176, false)
HQ_DQ_TRAITS(HQ_FMT_Q4_0, 144, true, 144, false)
HQ_DQ_TRAITS(HQ_FMT_Q5_0, 176, true, 176, false)
HQ_DQ_TRAITS(HQ_FMT_Q4_1, 160, true, 176, false)
HQ_DQ_TRAITS(HQ_FMT_Q5_1, 192, true, 208, false)
HQ_DQ_TRAITS(HQ_FMT_Q2_K, 84, false, 112, false)
HQ_DQ_TRAITS(HQ_FMT_Q3_K, 110, false, 144, false)
#undef HQ_DQ_TRAITS

// run-time plan of one launch (host side: dq_plan)
struct DqPlan {
  int tn;             // most tokens a tile may hold (multiple of 16)
  int rows_per_tile;  // dense: activation rows per token tile
  int n_tt;           // dense: token tiles
  int nbuf;           // accumulator buffers in tensor memory (2 up to 192 tokens, else 1)
  int subs;           // 64-k steps per operand stage: 2 or 4 (one barrier wait and one commit per stage)
  int ns;             // operand stages: A in tensor memory, tokens in shared memory
  uint32_t ns_magic;  // umulhi(i, ns_magic) = i / ns
  int nr;             // raw stages in shared memory
  int kslices;        // CTAs (cluster size) per tile
  int cpc;            // split K: most token columns a CTA of the cluster finishes
  int x_tma;          // token rows lie in tile order: one box per operand stage
  int raw_tma;        // raw rows copied as boxes (else in 4-byte pieces)
  int off_raw, off_recv, off_rows, off_pref, off_bar, smem;
};

__device__ __forceinline__ uint4 dq_lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
// NW words from `shift` words (0..3, the same in every lane) behind a 16-byte boundary: whole 16-byte loads, which meet no
// bank conflicts at the raw stages' row pitch, and a renaming of registers
template <int NW, int S>
__device__ __forceinline__ void dq_lds_shifted(uint32_t* w, uint32_t addr) {
  constexpr int NC = (NW + S + 3) / 4;
  uint32_t t[4 * NC];
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const uint4 v = dq_lds128(addr + 16 * i);
    t[4 * i] = v.x; t[4 * i + 1] = v.y; t[4 * i + 2] = v.z; t[4 * i + 3] = v.w;
  }
#pragma unroll
  for (int i = 0; i < NW; ++i) w[i] = t[S + i];
}
template <int NW>
__device__ __forceinline__ void dq_lds_words(uint32_t* w, uint32_t addr, int shift) {
  switch (shift) {
    case 0: dq_lds_shifted<NW, 0>(w, addr); break;
    case 1: dq_lds_shifted<NW, 1>(w, addr); break;
    case 2: dq_lds_shifted<NW, 2>(w, addr); break;
    default: dq_lds_shifted<NW, 3>(w, addr); break;
  }
}

// The 64 weights 64 c .. of one row's 256-k stage, in two halves of 32.  load() reads what both halves share or what is
// too oddly aligned to be read twice, half<>() expands one half.  c, half and the alignments are run-time numbers (the
// same in a whole warp) on purpose: one short loop body for all sixteen warps stays in the instruction caches -- with a
// body per c, unrolled over the halves, the warps spent a quarter of their time waiting for instructions.
//   addr: shared address of the row's stage (16-byte aligned); ws, mis: narrow types, the block starts ws words and
//   mis (0 or 2) bytes behind it; sw: swizzle term (row & 7) of the 128-byte-swizzled stages; sc: FP8 relative block
//   scale (f32 bits), MXFP4 the two e8m0 bytes of the 64 weights
template <int FMT>
struct DqRow {
  static constexpr int NW = FMT == HQ_FMT_Q8_0 ? 17 : FMT == HQ_FMT_Q5_K ? 20 : FMT == HQ_FMT_Q6_K ? 28
                            : FMT == HQ_FMT_Q3_K ? 20 : FMT == HQ_FMT_Q4_K ? 12 : FMT == HQ_FMT_Q2_K ? 10
                            : FMT == HQ_FMT_Q4_0 ? 9 : FMT == HQ_FMT_Q5_0 ? 11 : FMT == HQ_FMT_Q4_1 ? 10 : 1;
  uint32_t w[NW];
  uint32_t d, sh, addr, sw, sc, mis;

  __device__ __forceinline__ void load(uint32_t addr_, int c, int ws, uint32_t mis_, uint32_t sw_, uint32_t sc_) {
    addr = addr_; sw = sw_; sc = sc_; mis = mis_;
    if constexpr (FMT == HQ_FMT_Q4_K || FMT == HQ_FMT_Q5_K) {
      dq_lds_shifted<4, 0>(w, addr);
      dq_lds_shifted<8, 0>(w + 4, addr + (FMT == HQ_FMT_Q4_K ? 16 : 48) + 32 * c);
      if constexpr (FMT == HQ_FMT_Q5_K) dq_lds_shifted<8, 0>(w + 12, addr + 16);
      uint32_t s4, m4;
      k_scales(w[1], w[2], w[3], c >= 2, s4, m4);
      affine_pair<FMT == HQ_FMT_Q4_K>(w, s4, m4, (c & 1) ? 0x4342u : 0x4140u);
    } else if constexpr (FMT == HQ_FMT_Q8_0) {
      // two 34-byte blocks {f16 d, int8 q[32]} from byte 68 c on
      dq_lds_words<17>(w, addr + ((68 * c) & ~15), c);
      d = w[0] & 0xFFFFu;
      sh = 16;
    } else if constexpr (FMT == HQ_FMT_Q6_K) {
      // {ql[128], qh[64], scales[16], d}: weights 32 i + 16 s + t of the 64 (c = 2 h + (c & 1)) take nibble c & 1 of
      // ql[64 h + 32 i + 16 s + t], bits 2 j, 2 j + 1 (j = 2 (c & 1) + i) of qh[32 h + 16 s + t], scale 8 h + 2 j + s
      const int h = c >> 1;
      dq_lds_words<17>(w, addr + 64 * h, ws);
      dq_lds_words<9>(w + 17, addr + 128 + 32 * h, ws);
      const uint32_t at = addr + 192 + 4 * c + 4 * ws;
      w[26] = __funnelshift_r(lds32(at), lds32<4>(at), mis * 8);
      d = lds16<208>(addr + 4 * ws + mis);
    } else if constexpr (FMT == HQ_FMT_Q3_K) {
      // {hmask[32], qs[64], scales[12], d}: weights as for Q6_K with bits 2 j of qs[32 h + 16 s + t] and bit 4 h + j of
      // hmask[16 s + t]; the 6-bit scale of group 4 c + b is a nibble of byte 4 (c % 2) + b (low for c < 2) with bits
      // 2 c, 2 c + 1 of byte 8 + b on top
      const int h = c >> 1;
      dq_lds_words<9>(w, addr + 32 + 32 * h, ws);
      dq_lds_words<9>(w + 9, addr, ws);
      const uint32_t at = addr + 96 + 4 * ws;
      const uint32_t nib = __funnelshift_r(lds32(at + 4 * (c & 1)), lds32<4>(at + 4 * (c & 1)), mis * 8) >> (c < 2 ? 0 : 4);
      const uint32_t top = __funnelshift_r(lds32<8>(at), lds32<12>(at), mis * 8) >> (2 * c);
      w[18] = (nib & 0x0F0F0F0Fu) | ((top & 0x03030303u) << 4);
      d = lds16<108>(addr + 4 * ws + mis);
    } else if constexpr (FMT == HQ_FMT_Q2_K) {
      // {scales[16], qs[64], d, dmin}: weights as for Q3_K
      dq_lds_words<8>(w, addr + 16 + 32 * (c >> 1), ws);
      w[8] = lds32(addr + 4 * c + 4 * ws);
      w[9] = lds32<80>(addr + 4 * ws);
    } else if constexpr (FMT == HQ_FMT_Q4_0 || FMT == HQ_FMT_Q5_0 || FMT == HQ_FMT_Q4_1) {
      // two blocks of 18, 22 or 20 bytes {f16 d, [f16 m,] [u32 qh,] qs[16]} from byte 2 BB c on
      constexpr int BB = FMT == HQ_FMT_Q4_0 ? 18 : FMT == HQ_FMT_Q5_0 ? 22 : 20;
      const int at = 2 * BB * c;
      dq_lds_words<NW>(w, addr + (at & ~15), (at & 15) >> 2);
      sh = FMT == HQ_FMT_Q4_1 ? 0 : 16;
    }
  }

  // 32 weights -> sixteen f16 pairs in natural k order, handed to put(pair index, eight pairs) as they are ready;
  // false: an MXFP4 block scale the f16 operand cannot hold
  template <typename Put>
  __device__ __forceinline__ bool half(int c, int i, Put put) {
    RawA a;
    uint32_t o[8];
    bool ok = true;
    if constexpr (FMT == HQ_FMT_Q4_K || FMT == HQ_FMT_Q5_K) {
      const AffineH2 f = affine_of(w, i);
      const uint32_t nibbles = 0x0F0F0F0Fu << (4 * i);      // Q4_K: the second half's codes stay 16 times too large
#pragma unroll
      for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t codes;
          if constexpr (FMT == HQ_FMT_Q4_K) codes = w[4 + 4 * u + j] & nibbles;
          else codes = ((w[4 + 4 * u + j] >> (4 * i)) & 0x0F0F0F0Fu) | (((w[12 + 4 * u + j] >> (2 * c + i)) & 0x01010101u) << 4);
          affine4(f, codes, o[2 * j], o[2 * j + 1]);
        }
        put(8 * u, o);
      }
    } else if constexpr (FMT == HQ_FMT_Q8_0) {
      a.aux = d | (sh << 16);
      a.q = make_uint4(w[0], w[1], w[2], w[3]);
      a.hdr.x = w[4];
      emit_q8_0(a, o);
      put(0, o);
      a.q = make_uint4(w[4], w[5], w[6], w[7]);
      a.hdr.x = w[8];
      emit_q8_0(a, o);
      put(8, o);
      // the second block's d shares a word with the first block's end, its payload starts on a word
      d = w[8] >> 16;
      sh = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = w[9 + j];
    } else if constexpr (FMT == HQ_FMT_FP8_BLOCK) {
      a.aux = sc;
      const uint32_t at = addr + mis * (c >> 1);      // the second 128 columns of the rows lie behind the first
      const int ch = 4 * (c & 1) + 2 * i;
      a.q = dq_lds128(at + ((ch ^ sw) << 4));
      emit_fp8(a, o);
      put(0, o);
      a.q = dq_lds128(at + (((ch + 1) ^ sw) << 4));
      emit_fp8(a, o);
      put(8, o);
    } else if constexpr (FMT == HQ_FMT_MXFP4) {
      const uint4 v = dq_lds128(addr + (((2 * c + i) ^ sw) << 4));
      a.aux = (sc >> (8 * i)) & 0xFFu;
      a.q.x = v.x; a.q.y = v.y;
      ok = emit_mxfp4(a, o);
      put(0, o);
      a.q.x = v.z; a.q.y = v.w;
      ok = emit_mxfp4(a, o) && ok;
      put(8, o);
    } else if constexpr (FMT == HQ_FMT_Q6_K) {
      a.aux = 2 * (c & 1) + i;
      const uint32_t sc2 = w[26] >> (16 * i);
      a.q = make_uint4(w[0], w[1], w[2], w[3]);
      a.hdr = make_uint4(w[17], w[18], w[19], w[20]);
      a.ext = make_uint4(w[4], w[21], d | ((sc2 & 0xFFu) << 16), (mis << 3) | (mis << 11));
      emit_q6_k(a, o);
      put(0, o);
      a.q = make_uint4(w[4], w[5], w[6], w[7]);
      a.hdr = make_uint4(w[21], w[22], w[23], w[24]);
      a.ext = make_uint4(w[8], w[25], d | (((sc2 >> 8) & 0xFFu) << 16), (mis << 3) | (mis << 11));
      emit_q6_k(a, o);
      put(8, o);
#pragma unroll
      for (int j = 0; j < 9; ++j) w[j] = w[8 + j];
    } else if constexpr (FMT == HQ_FMT_Q3_K) {
      const uint32_t j = 2 * (c & 1) + i, sc2 = w[18] >> (16 * i);
      a.aux = j | ((4 * (c >> 1) + j) << 8);
      a.q = make_uint4(w[0], w[1], w[2], w[3]);
      a.hdr = make_uint4(w[9], w[10], w[11], w[12]);
      a.ext = make_uint4(w[4], w[13], d | ((sc2 & 0xFFu) << 16), (mis << 3) | (mis << 11));
      emit_q3_k(a, o);
      put(0, o);
      a.q = make_uint4(w[4], w[5], w[6], w[7]);
      a.hdr = make_uint4(w[13], w[14], w[15], w[16]);
      a.ext = make_uint4(w[8], w[17], d | (((sc2 >> 8) & 0xFFu) << 16), (mis << 3) | (mis << 11));
      emit_q3_k(a, o);
      put(8, o);
    } else if constexpr (FMT == HQ_FMT_Q2_K) {
      const uint32_t j = 2 * (c & 1) + i, sc2 = w[8] >> (16 * i);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint32_t sb = sc2 >> (8 * u);
        const AffineH2 f = make_affine(w[9], sb & 15u, (sb >> 4) & 15u);
#pragma unroll
        for (int t = 0; t < 4; ++t) affine4(f, (w[4 * u + t] >> (2 * j)) & 0x03030303u, o[2 * t], o[2 * t + 1]);
        put(8 * u, o);
      }
    } else {
      // one 32-weight block: weight t is the low, 16 + t the high nibble of qs[t]
      uint32_t q[5], qh = 0u, dd, mm = 0u;
      if constexpr (FMT == HQ_FMT_Q4_0) {
        // block 0: d in the low half of w[0], qs across the words from there; block 1: d in the high half of w[4]
        dd = sh ? w[0] & 0xFFFFu : d;
#pragma unroll
        for (int j = 0; j < 5; ++j) q[j] = w[j];
        d = w[4] >> 16;
      } else if constexpr (FMT == HQ_FMT_Q5_0) {
        // block 0: d low half of w[0], qh across w[0], w[1], qs from the middle of w[1]; block 1: d high half of w[5]
        dd = sh ? w[0] & 0xFFFFu : d;
        qh = __funnelshift_r(w[0], w[1], sh);
#pragma unroll
        for (int j = 0; j < 5; ++j) q[j] = w[1 + j];
        d = w[5] >> 16;
      } else if constexpr (FMT == HQ_FMT_Q4_1) {
        dd = w[0] & 0xFFFFu;
        mm = w[0] >> 16;
#pragma unroll
        for (int j = 0; j < 4; ++j) q[j] = w[1 + j];
        q[4] = 0u;
      } else {
        static_assert(FMT == HQ_FMT_Q5_1, "format");
        const uint32_t at = addr + 48 * c + 24 * i;
        const uint2 h0 = lds64<0>(at), h1 = lds64<8>(at), h2 = lds64<16>(at);
        dd = h0.x & 0xFFFFu;
        mm = h0.x >> 16;
        qh = h0.y;
        q[0] = h1.x; q[1] = h1.y; q[2] = h2.x; q[3] = h2.y; q[4] = 0u;
        sh = 0;
      }
      a.q = make_uint4(q[0], q[1], q[2], q[3]);
      a.hdr = make_uint4(q[4], mm, 0u, 0u);
      a.aux = dd | (sh << 16);
      a.ext.x = qh & 0xFFFFu;
      emit_q4_0_q5_0<FMT>(a, o);
      put(0, o);
      a.aux |= 1u << 24;
      a.ext.x = qh >> 16;
      emit_q4_0_q5_0<FMT>(a, o);
      put(8, o);
      constexpr int ADV = FMT == HQ_FMT_Q5_0 ? 6 : 5, KEEP = FMT == HQ_FMT_Q4_0 ? 4 : 5;
      if constexpr (FMT != HQ_FMT_Q5_1) {
#pragma unroll
        for (int j = 0; j < KEEP; ++j) w[j] = w[ADV + j];
      }
      sh = 0;
    }
    return ok;
  }
};

// Token boxes: a stage's 64-k steps of 16, 32, .. rows, so that an expert's tile of whatever size is one copy (dense calls: the
// first map, rows of the plan's tile).  A copy instruction costs its warp some 250 cycles: with boxes of 64 and 16 rows and one
// step each a stage of 128 tokens took six, 1,500 cycles for 1,000 cycles of products (128 experts of 768 x 2,048 Q4_K, 4,096
// tokens: gated launch 365 us so, 265 with one box; down launch 237, 172).
struct DqTokenMaps {
  CUtensorMap m[kDqMaxTokens / 16];
};

// ---- work items --------------------------------------------------------------------------------------------------
struct DqTile {
  int expert, row_start, count, n0;
};
__device__ __forceinline__ DqTile dq_tile(const GroupedParams& p, const DqPlan& pl, const int32_t* pref, int w, int n_nt,
                                          int fw) {
  DqTile t;
  const int tt = w / n_nt;
  t.n0 = (w - tt * n_nt) * fw;
  if (p.expert_bounds == nullptr) {
    t.expert = 0;
    t.row_start = pl.rows_per_tile * tt;
    t.count = min(pl.rows_per_tile, p.m - t.row_start);
    return t;
  }
  int lo = 0, hi = p.n_experts - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pref[mid] <= tt) lo = mid; else hi = mid - 1;
  }
  const int32_t* rows = pref + p.n_experts + 1;
  const int base = rows[lo], cnt = rows[lo + 1] - base;
  // an expert's rows are cut into equal tiles (multiples of 16 rows)
  const int nt = pref[lo + 1] - pref[lo], j = tt - pref[lo];
  const int per = ((cnt + nt - 1) / nt + 15) & ~15;
  t.expert = lo;
  t.row_start = base + j * per;
  t.count = max(0, min(per, cnt - j * per));
  return t;
}

// rows of a tile's tokens in shared memory: the distance between the 64-k steps of a stage
__device__ __forceinline__ int dq_box_rows(const GroupedParams& p, const DqPlan& pl, const DqTile& t) {
  return p.expert_bounds != nullptr ? max(16, (t.count + 15) & ~15) : pl.tn;
}

__device__ __forceinline__ void dq_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ uint32_t dq_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t dq_mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void dq_arrive_remote(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool dq_wait_cluster(uint64_t* bar, uint32_t parity, uint32_t spin_limit) {
  for (uint32_t i = 0; i < spin_limit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(kWaitSuspendNs)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// 64 k of one stage: four MMAs of K = 16 (8 columns of A in tensor memory, 32 bytes along the swizzled rows of B).  Called
// by a whole warp; the elected lane issues.
__device__ __forceinline__ void dq_mma64(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p, e;\n"
      ".reg .b32 a1;\n"
      ".reg .b64 b1;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "add.s32 a1, %1, 8;\n"
      "add.s64 b1, %2, 2;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, 1;\n"
      "add.s32 a1, %1, 16;\n"
      "add.s64 b1, %2, 4;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, 1;\n"
      "add.s32 a1, %1, 24;\n"
      "add.s64 b1, %2, 6;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, 1;\n"
      "}\n" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
constexpr int kDqMaxStages = 8, kDqMaxRaw = 12;
constexpr int kDqNumBars = 2 * kDqMaxStages + 2 * kDqMaxRaw + 4 + 2;   // operand ring, raw ring, accumulators, exchange
struct DqBars {
  uint64_t *full, *empty, *full_r, *empty_r, *acc_full, *acc_empty, *red_full, *red_empty;
  __device__ __forceinline__ explicit DqBars(uint8_t* base) {
    full = reinterpret_cast<uint64_t*>(base);
    empty = full + kDqMaxStages;
    full_r = empty + kDqMaxStages;
    empty_r = full_r + kDqMaxRaw;
    acc_full = empty_r + kDqMaxRaw;
    acc_empty = acc_full + 2;
    red_full = acc_empty + 2;
    red_empty = red_full + 1;
  }
};
// position of operand stage `i` of the CTA's sequence in the ring
struct DqSlot {
  int s;
  uint32_t use;      // how often the slot was used before
};
__device__ __forceinline__ DqSlot dq_slot(const DqPlan& pl, int i) {
  DqSlot r;
  r.use = __umulhi((uint32_t)i, pl.ns_magic);
  r.s = i - (int)r.use * pl.ns;
  return r;
}

template <int FMT, bool ODD>
__device__ __forceinline__ void dq_expand_warps(const GroupedParams& p, const DqPlan& pl, uint8_t* smem, int n_tiles,
                                                int n_nt, int rs_lo, int rs_hi, int first, int step, uint32_t tmem_base,
                                                int C, int q, int lane) {
  using T = DqTraits<FMT>;
  const DqBars bar(smem + pl.off_bar);
  const int32_t* pref = reinterpret_cast<const int32_t*>(smem + pl.off_pref);
  const bool two = p.w_up != nullptr;
  const int fw = two ? 64 : 128;
  const int bank = two ? lane >> 4 : 0;
  const int frow = two ? 16 * q + (lane & 15) : 32 * q + lane;      // feature within the tile
  const int srow = two ? 64 * bank + frow : frow;                   // row of the raw stage
  // block-FP8: two 128-byte column halves per bank, one behind the other
  const uint32_t raw0 = smem_u32(smem + pl.off_raw) +
                        (T::BOXES == 2 && two ? (uint32_t)(16384 * bank + 128 * frow) : (uint32_t)srow * T::PITCH);
  const uint32_t half_stride = two ? 8192u : 16384u;
  const uint32_t sw = (uint32_t)srow & 7u;
  const int kb64 = p.k >> 6;                                        // 64-k steps of the whole K
  const int subs = pl.subs, sub_shift = subs == 4 ? 2 : 1;
  const int my_stage = C >> sub_shift, my_sub = C & (subs - 1);     // stage within the raw stage, step within the stage
  const int stages_per_raw = 4 >> sub_shift;
  const int slice_stages = (dq_walk_steps(ODD, min(kb64, 4 * rs_hi) - 4 * rs_lo) + subs - 1) >> sub_shift;
  const uint32_t tcol = tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(512 - 32 * subs * pl.ns + 32 * my_sub);
  // What binds these warps is the number of their instructions, so a wait should leave no branch behind (warp_wait_uni: `spin`
  // becomes 0 when one runs out, which is reported at the end).  65,536 x 4,096 at 16 rows, us, with the branches and without:
  // FP8 51.0 : 49.8, MXFP4 54.8 : 52.8, Q5_K 75.0 : 72.8; Q4_K 61.6 : 64.9 and Q6_K 94.6 : 94.8, which leave no register free.
  // (The first use of a slot waits for the phase before its first, which counts as complete.)
  constexpr bool BRANCH = FMT == HQ_FMT_Q4_K || !T::WIDE;
  uint32_t spin = kDqSpin;
  auto await = [&](uint64_t* b, uint32_t parity, int tag) {
    if constexpr (BRANCH) {
      if (!warp_wait(b, parity, spin)) {
        if (lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, tag);
        spin = 1;
      }
    } else {
      spin = warp_wait_uni(smem_u32(b), parity, spin) ? spin : 0u;
    }
  };
  int slot = 0, ph = 0, it0 = 0;
  // scales that do not travel with the raw bytes: MXFP4 e8m0 pairs, FP8 relative block scales; fetched a stage ahead
  constexpr bool SIDE = FMT == HQ_FMT_MXFP4 || FMT == HQ_FMT_FP8_BLOCK;
  for (int w = first; w < n_tiles; w += step) {
    const DqTile t = dq_tile(p, pl, pref, w, n_nt, fw);
    const bool n_ok = t.n0 + frow < p.n;
    const int64_t wrow = (int64_t)t.expert * p.n + (n_ok ? t.n0 + frow : 0);
    uint32_t mis = 0;            // narrow types: bytes between the start of the copied row and the block
    if (!T::WIDE)
      mis = (uint32_t)((reinterpret_cast<uintptr_t>(bank == 0 ? p.w : p.w_up) + (uintptr_t)(wrow * p.w_row_bytes) +
                        (uintptr_t)rs_lo * T::SB) & (pl.raw_tma ? 15u : 2u));
    const uint8_t* side = nullptr;
    if constexpr (FMT == HQ_FMT_MXFP4)
      side = reinterpret_cast<const uint8_t*>(bank == 0 ? p.scales : p.scales_up) + wrow * (p.k / 32);
    if constexpr (FMT == HQ_FMT_FP8_BLOCK)
      side = reinterpret_cast<const uint8_t*>((bank == 0 ? p.fp8_rel_scale : p.fp8_rel_scale_up) +
                                              ((int64_t)t.expert * p.fp8_nb + t.n0 / 128) * p.fp8_kb);
    auto fetch_side = [&](int rs) -> uint32_t {
      if (4 * rs + C >= kb64) return 0u;
      if constexpr (FMT == HQ_FMT_MXFP4) return __ldg(reinterpret_cast<const uint16_t*>(side + 8 * rs + 2 * C));
      if constexpr (FMT == HQ_FMT_FP8_BLOCK) return __float_as_uint(__ldg(reinterpret_cast<const float*>(side) + 2 * rs + (C >> 1)));
      return 0u;
    };
    uint32_t sc_next = 0u;
    if (SIDE) sc_next = fetch_side(rs_lo);
    for (int rs = rs_lo; rs < rs_hi; ++rs) {
      const uint32_t sc = sc_next;
      if (SIDE && rs + 1 < rs_hi) sc_next = fetch_side(rs + 1);
      await(&bar.full_r[slot], ph, 500 + slot);
      const int local = (rs - rs_lo) * stages_per_raw + my_stage;        // operand stage within this tile
      const DqSlot at = dq_slot(pl, it0 + local);
      if (4 * rs + C < kb64) {
        const uint32_t taddr = tcol + (uint32_t)(32 * subs * at.s);
        DqRow<FMT> row;
        row.load(raw0 + (uint32_t)slot * T::STAGE, C, T::WIDE ? 0 : (int)(mis >> 2),
                 T::BOXES == 2 ? half_stride : T::WIDE ? 0u : mis & 2u, sw, sc);
        bool ok = true;
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          ok = row.half(C, i, [&](int at_pair, const uint32_t (&v)[8]) {
            if (i == 0 && at_pair == 0) await(&bar.empty[at.s], (at.use - 1) & 1, 520 + at.s);
            tmem_st8(taddr + 16 * i + at_pair, v);
          }) && ok;
        }
        // every byte of the raw stage this warp needs has been read
        __syncwarp();
        warp_arrive(&bar.empty_r[slot]);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        warp_arrive(&bar.full[at.s]);
        if (FMT == HQ_FMT_MXFP4 && !ok && n_ok) report_status(p.status, HQ_DEV_SCALE_RANGE, 600);
      } else {
        __syncwarp();
        warp_arrive(&bar.empty_r[slot]);
        // the K tail ends inside or in front of this group's stage: nothing to add, but the stage counts its arrivals
        if (local < slice_stages) {
          await(&bar.empty[at.s], (at.use - 1) & 1, 521);
          __syncwarp();
          warp_arrive(&bar.full[at.s]);
        }
      }
      if (!T::WIDE) mis = (mis + T::SB) & (pl.raw_tma ? 15u : 2u);
      if (++slot == pl.nr) { slot = 0; ph ^= 1; }
    }
    it0 += slice_stages;
  }
  if (!BRANCH && spin == 0u && lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, 500 + C);
}

// ODD: some tiles have an odd number of operand stages and there are two slots for them (dq_walk_steps).  An instance of its own,
// because the kernel is sensitive to its code: with the walk decided at run time other shapes ran 0.3 to 1.3 % slower.
template <int FMT, bool ODD>
__global__ void __launch_bounds__(DqTraits<FMT>::THREADS, 1)
dq_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_wu,
               const __grid_constant__ DqTokenMaps tm_x, const GroupedParams p, const DqPlan pl) {
  using T = DqTraits<FMT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const DqBars bar(smem + pl.off_bar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + pl.off_bar + kDqNumBars * 8);
  int32_t* pref = reinterpret_cast<int32_t*>(smem + pl.off_pref);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool two = p.w_up != nullptr;
  const int fw = two ? 64 : 128;
  const int n_nt = (p.n + fw - 1) / fw;
  const int S = pl.kslices;
  const int rank = S > 1 ? (int)dq_cluster_rank() : 0;
  const int first = blockIdx.x / S, step = gridDim.x / S;
  const int kb64 = p.k >> 6;
  const int nrs = (kb64 + 3) >> 2;
  const int per = (nrs + S - 1) / S;
  const int rs_lo = min(nrs, rank * per), rs_hi = min(nrs, rs_lo + per);

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == 0) {
    // a stage is complete when its expanding warps and its tokens (the copies of one thread, or two warps) have arrived
    for (int s = 0; s < pl.ns; ++s) {
      mbar_init(&bar.full[s], 4 * pl.subs + (pl.x_tma ? 1 : kDqTokenWarps));
      mbar_init(&bar.empty[s], 1);
    }
    for (int s = 0; s < pl.nr; ++s) {
      mbar_init(&bar.full_r[s], pl.raw_tma ? 1 : 32 * T::COPY_WARPS);
      mbar_init(&bar.empty_r[s], kDqExpandWarps);
    }
    for (int b = 0; b < 2; ++b) { mbar_init(&bar.acc_full[b], 1); mbar_init(&bar.acc_empty[b], kDqEpilogueWarps); }
    mbar_init(bar.red_full, kDqEpilogueWarps * S);
    mbar_init(bar.red_empty, kDqEpilogueWarps * S);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  if (p.expert_bounds != nullptr) {
    dq_pdl_wait();                 // the routing tables come from the previous kernels
    for (int e = tid; e < p.n_experts; e += T::THREADS) {
      const int lo = __ldg(p.expert_bounds + e), hi = __ldg(p.expert_bounds + e + 1);
      pref[e + 1] = (hi - lo + pl.tn - 1) / pl.tn;
      int32_t* rows = pref + p.n_experts + 1;      // the experts' first rows behind their first tiles
      rows[e] = lo;
      if (e == p.n_experts - 1) rows[e + 1] = hi;
    }
    if (tid == 0) pref[0] = 0;
    __syncthreads();
    if (warp == 1) {
      int carry = 0;
      for (int base = 0; base < p.n_experts; base += 32) {
        const int e = base + lane;
        int v = e < p.n_experts ? pref[e + 1] : 0;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int o = __shfl_up_sync(0xffffffffu, v, d);
          if (lane >= d) v += o;
        }
        if (e < p.n_experts) pref[e + 1] = carry + v;
        carry += __shfl_sync(0xffffffffu, v, 31);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (S > 1) {      // every CTA's barriers exist before a peer arrives on them
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  const uint32_t tmem_base = *tmem_slot;
  const int n_tiles = (p.expert_bounds != nullptr ? pref[p.n_experts] : pl.n_tt) * n_nt;

  if (warp == 0) {
    // =========================== MMA issuer ===========================================================
    // The whole warp walks the loop and one elected lane issues: operands stay in uniform registers.  (Issued from a
    // single-lane branch a stage of four MMAs and two commits took 870 cycles whatever its width, against 256 the
    // tensor core needs for 128 columns.)
    uint32_t spin = kDqSpin;
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint32_t step_bytes = (uint32_t)pl.tn * 128u, b0 = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
    const int a_col = 512 - 32 * pl.subs * pl.ns;
    const int slice_subs = min(kb64, 4 * rs_hi) - 4 * rs_lo, walk_subs = dq_walk_steps(ODD, slice_subs);
    int it = 0, tcount = 0;
    for (int w = first; w < n_tiles; w += step, ++tcount) {
      const DqTile t = dq_tile(p, pl, pref, w, n_nt, fw);
      const uint32_t idesc = make_idesc_f16(__shfl_sync(0xffffffffu, max(16, (t.count + 15) & ~15), 0));
      const uint32_t sub_bytes = __shfl_sync(0xffffffffu, (uint32_t)dq_box_rows(p, pl, t) * 128u, 0);
      const int buf = pl.nbuf == 2 ? tcount & 1 : 0;
      const int use = pl.nbuf == 2 ? tcount >> 1 : tcount;
      if (use > 0 && !warp_wait(&bar.acc_empty[buf], (use - 1) & 1, spin)) {
        if (lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, 300 + buf);
        spin = 1;
      }
      tc_fence_after();
      const uint32_t d0 = tmem_u + (uint32_t)(buf * pl.tn);
      for (int j = 0; j < walk_subs; j += pl.subs, ++it) {
        const DqSlot at = dq_slot(pl, it);
        if (!warp_wait(&bar.full[at.s], at.use & 1, spin)) {
          if (lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, 310 + at.s);
          spin = 1;
        }
        tc_fence_after();
        uint64_t bdesc = make_smem_desc(b0 + (uint32_t)(at.s * pl.subs) * step_bytes);
        uint32_t a0 = tmem_u + (uint32_t)(a_col + 32 * pl.subs * at.s);
        const int n_sub = min(pl.subs, slice_subs - j);
        for (int c = 0; c < n_sub; ++c) {
          dq_mma64(d0, a0, bdesc, idesc, (j + c) > 0 ? 1u : 0u);
          bdesc += sub_bytes >> 4;
          a0 += 32;
        }
        warp_commit(&bar.empty[at.s]);
      }
      warp_commit(&bar.acc_full[buf]);
    }
    __syncwarp();
  } else if (warp <= kDqEpilogueWarps) {
    // =========================== epilogue =============================================================
    dq_pdl_wait();                          // the previous kernel may still be reading what y's memory held
    const int q = warp & 3;                 // tensor-memory lane quarter this warp may read
    const int hw = (warp - 1) >> 2;         // the two warps of a quarter take column groups in turn
    uint32_t spin = kDqSpin;
    bool failed = false;
    int tcount = 0;
    const bool interleaved = !two && p.act.act != HQ_ACT_NONE;
    const int bank = two ? lane >> 4 : 0;
    const int frow = two ? 16 * q + (lane & 15) : 32 * q + lane;
    const int esz = dtype_size(p.y_dtype);
    const int64_t ystride_b = (int64_t)p.y_stride * esz;
    float* recv = reinterpret_cast<float*>(smem + pl.off_recv);
    const uint32_t recv_u = smem_u32(recv), redf_u = smem_u32(bar.red_full), rede_u = smem_u32(bar.red_empty);
    for (int w = first; w < n_tiles; w += step, ++tcount) {
      const DqTile t = dq_tile(p, pl, pref, w, n_nt, fw);
      const int buf = pl.nbuf == 2 ? tcount & 1 : 0;
      const int use = pl.nbuf == 2 ? tcount >> 1 : tcount;
      const int n = t.n0 + frow;
      const bool n_ok = n < p.n;
      float bias = 0.f;
      const void* bptr = bank == 0 ? p.bias : p.bias_up;
      if (n_ok && bptr != nullptr) bias = load_as_float(bptr, p.bias_dtype, (int64_t)t.expert * p.n + n);
      float sc = 1.f;
      if (FMT == HQ_FMT_FP8_BLOCK)
        sc = __ldg((bank == 0 ? p.fp8_tile_scale : p.fp8_tile_scale_up) + (int64_t)t.expert * p.fp8_nb + t.n0 / 128);
      if (!warp_wait(&bar.acc_full[buf], use & 1, spin)) {
        if (lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, 400 + buf);
        spin = 1;
        failed = true;                 // nothing is stored once a wait has run out
      }
      tc_fence_after();
      const int64_t out_n = interleaved ? (n >> 1) : n;
      const bool writer = n_ok && (two ? lane < 16 : (!interleaved || (n & 1) == 0));
      const uint32_t taddr = tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(buf * pl.tn);
      char* const ybase = reinterpret_cast<char*>(p.y) + out_n * esz;
      const int* __restrict__ yrows = p.y_rows;
      auto finish = [&](float acc) -> float {
        float r = fmaf(acc, sc, bias);
        if (two) r = gg_gated(r, __shfl_xor_sync(0xffffffffu, r, 16), p.act);          // the up row of this gate row
        else if (interleaved) r = gg_gated(r, __shfl_xor_sync(0xffffffffu, r, 1), p.act);
        return r;
      };
      if (S == 1) {
        // Sixteen columns at a time in a rolled loop (short code: it keeps out of the way of the expanding warps').  With
        // two banks lanes 0..15 finish the even columns and lanes 16..31 the odd ones: one exchange of partners per pair
        // of columns, no activation computed twice.
        const int groups = (t.count + 15) >> 4;
        auto columns = [&](auto cvt) {
          using TY = decltype(cvt(0.f));
#pragma unroll 1
          for (int g = hw; g < groups; g += 2) {
            const int c0 = 16 * g;
            uint32_t v[16];
            tmem_ld16(taddr + c0, v);
            int orow = 0;
            if (yrows != nullptr) orow = __ldg(yrows + min(t.row_start + c0 + (lane & 15), t.row_start + t.count - 1));
            tmem_ld_wait();
            char* dst = ybase + (int64_t)(t.row_start + c0 + (two ? bank : 0)) * ystride_b;
            const int left = t.count - c0;
            if (two) {
#pragma unroll
              for (int j = 0; j < 16; j += 2) {
                const float a0 = fmaf(__uint_as_float(v[j]), sc, bias), a1 = fmaf(__uint_as_float(v[j + 1]), sc, bias);
                const float other = __shfl_xor_sync(0xffffffffu, bank == 0 ? a1 : a0, 16);
                const float r = gg_gated(bank == 0 ? a0 : other, bank == 0 ? other : a1, p.act);
                if (yrows != nullptr) dst = ybase + (int64_t)__shfl_sync(0xffffffffu, orow, j + bank) * ystride_b;
                if (n_ok && !failed && j + bank < left) *reinterpret_cast<TY*>(dst) = cvt(r);
                dst += 2 * ystride_b;
              }
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const float r = finish(__uint_as_float(v[j]));
                if (yrows != nullptr) dst = ybase + (int64_t)__shfl_sync(0xffffffffu, orow, j) * ystride_b;
                if (writer && !failed && j < left) *reinterpret_cast<TY*>(dst) = cvt(r);
                dst += ystride_b;
              }
            }
          }
        };
        if (p.y_dtype == HQ_DT_BF16) columns([](float f) { return __float2bfloat16_rn(f); });
        else if (p.y_dtype == HQ_DT_F16) columns([](float f) { return __float2half_rn(f); });
        else columns([](float f) { return f; });
        tc_fence_before();               // the buffer is read out: the next tile may accumulate into it
        __syncwarp();
        warp_arrive(&bar.acc_empty[buf]);
      } else {
        // ---- split K: token column c is finished by CTA c / cpc of the cluster ------------------------
        const int cpc = (t.count + S - 1) / S;
        if (tcount > 0 && !dq_wait_cluster(bar.red_empty, (tcount - 1) & 1, spin)) {
          if (lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, 410);
          spin = 1;
          failed = true;
        }
        const uint32_t mine = recv_u + (uint32_t)(rank * pl.cpc * 128 + 32 * q + lane) * 4u;
#pragma unroll 1
        for (int c0 = 8 * hw; c0 < t.count; c0 += 16) {
          uint32_t v[8];
          tmem_ld8(taddr + c0, v);
          int dst = c0 / cpc, within = c0 - dst * cpc;
          uint32_t dst_addr = dq_mapa(mine, (uint32_t)dst);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (c0 + j < t.count) {
              asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(dst_addr + (uint32_t)within * 512u), "r"(v[j]) : "memory");
              if (++within == cpc) {
                within = 0;
                if (++dst < S) dst_addr = dq_mapa(mine, (uint32_t)dst);
              }
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        warp_arrive(&bar.acc_empty[buf]);
        if (lane < S) dq_arrive_remote(dq_mapa(redf_u, (uint32_t)lane));
        if (!dq_wait_cluster(bar.red_full, tcount & 1, spin)) {
          if (lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, 420);
          spin = 1;
          failed = true;
        }
        const int my0 = rank * cpc, my1 = min(t.count, my0 + cpc);
        for (int c = my0 + hw; c < my1; c += 2) {
          const float* src = recv + (c - my0) * 128 + 32 * q + lane;
          float a = 0.f;
          for (int s = 0; s < S; ++s) a += src[s * pl.cpc * 128];       // rank order
          const float r = finish(a);
          const int sp = t.row_start + c;
          const int64_t orow = yrows != nullptr ? __ldg(yrows + sp) : sp;
          if (writer && !failed) store_from_float(ybase + orow * ystride_b, p.y_dtype, 0, r);
        }
        __syncwarp();
        if (lane < S) dq_arrive_remote(dq_mapa(rede_u, (uint32_t)lane));
      }
    }
  } else if (warp == 1 + kDqEpilogueWarps || (pl.x_tma && warp == 3 + kDqEpilogueWarps)) {
    // =========================== raw weight bytes, as boxes =============================================
    if (pl.raw_tma) {
      uint32_t spin = kDqSpin;
      int slot = 0, ph = 0;
      bool wrapped = false, stop = false;
      const int banks = two ? 2 : 1;
      // One round {wait, arrive, copy} is a chain of some five hundred cycles whatever it copies: two warps take the
      // stages in turn (the second token warp has nothing to do when one box holds a stage's tokens)
      // (65,536 x 4,096 at 16 rows, one warp and a box per 64 k before: MXFP4 68 -> 57 us, FP8 64 -> 55).  A slot's
      // parity stays unambiguous: stages are consumed in order, so a warp that has issued stage i - 2 knows that the
      // use of its slot before the last one (stage i - 2 nr) is long over.
      const int helpers = pl.x_tma ? 2 : 1, me = warp == 1 + kDqEpilogueWarps ? 0 : 1;
      int turn = 0;
      for (int w = first; w < n_tiles && !stop; w += step) {
        const DqTile t = dq_tile(p, pl, pref, w, n_nt, fw);
        const int row = t.expert * p.n + t.n0;
        for (int rs = rs_lo; rs < rs_hi; ++rs) {
          const bool mine = helpers == 1 || (turn & 1) == me;
          ++turn;
          if (!mine) {
            if (++slot == pl.nr) { slot = 0; ph ^= 1; wrapped = true; }
            continue;
          }
          if (wrapped && !warp_wait(&bar.empty_r[slot], ph ^ 1, spin)) {
            if (lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, 560 + slot);
            stop = true;               // nothing more is issued: the target may still be in use
            break;
          }
          warp_arrive_expect(&bar.full_r[slot], (uint32_t)T::STAGE);
          const uint32_t dst = smem_u32(smem + pl.off_raw) + (uint32_t)slot * T::STAGE;
          const int x = ((rs * T::SB) & ~15) / 2;            // 16-bit elements
          for (int b = 0; b < banks; ++b) {
            if constexpr (T::BOXES == 2)
              warp_tma_3d(dst + b * 16384u, b ? &tm_wu : &tm_w, 0, row, 2 * rs, &bar.full_r[slot]);
            else
              warp_tma_2d(dst + b * (64u * T::PITCH), b ? &tm_wu : &tm_w, x, row, &bar.full_r[slot]);
          }
          if (++slot == pl.nr) { slot = 0; ph ^= 1; wrapped = true; }
        }
      }
      // No copy may still be writing the CTA's shared memory when it exits: the stages ring_drain names, walked as it does (written
      // out here and for the tokens: of the forms tried the one that left other code as fast as it was).
      const int next = stop ? turn - 1 : turn;
#pragma unroll 1
      for (int i = next - pl.nr; i < next; ++i) {
        if (i >= 0 && (i & (helpers - 1)) == me && !warp_wait(&bar.full_r[slot], ph ^ 1, spin)) {
          if (lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, 580 + me);
          spin = 1;
        }
        if (++slot == pl.nr) { slot = 0; ph ^= 1; }
      }
    }
  } else if (warp < 2 + kDqEpilogueWarps + kDqTokenWarps) {
    // =========================== activation rows ========================================================
    dq_pdl_wait();
    const uint32_t step_bytes = (uint32_t)pl.tn * 128u;
    const int slice_subs = min(kb64, 4 * rs_hi) - 4 * rs_lo, walk_subs = dq_walk_steps(ODD, slice_subs);
    uint32_t spin = kDqSpin;
    int it = 0;
    if (pl.x_tma) {
      if (warp == 2 + kDqEpilogueWarps) {
        bool stop = false;
        for (int w = first; w < n_tiles && !stop; w += step) {
          const DqTile t = dq_tile(p, pl, pref, w, n_nt, fw);
          // (rows behind the tile's last are copied along: other experts' or zeros, in accumulator columns nobody reads)
          const int box = dq_box_rows(p, pl, t);
          const uint32_t bytes = (uint32_t)(pl.subs * box) * 128u;
          const CUtensorMap* map = &tm_x.m[p.expert_bounds != nullptr ? (box >> 4) - 1 : 0];
          for (int j = 0; j < walk_subs; j += pl.subs, ++it) {
            const DqSlot at = dq_slot(pl, it);
            if (at.use > 0 && !warp_wait(&bar.empty[at.s], (at.use - 1) & 1, spin)) {
              if (lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, 540 + at.s);
              stop = true;
              break;
            }
            if (ODD && j >= slice_subs) {      // a stage without products
              warp_arrive(&bar.full[at.s]);
              continue;
            }
            warp_arrive_expect(&bar.full[at.s], bytes);
            warp_tma_3d(smem_u32(smem) + (uint32_t)(at.s * pl.subs) * step_bytes, map, 0, t.row_start, 4 * rs_lo + j,
                        &bar.full[at.s]);
          }
        }
#pragma unroll 1
        for (int i = max(0, it - pl.ns); i < it; ++i) {      // ... and the last stages of tokens
          const DqSlot at = dq_slot(pl, i);
          if (!warp_wait(&bar.full[at.s], at.use & 1, spin)) {
            if (lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, 590 + at.s);
            spin = 1;
          }
        }
      }
    } else {
      // rows in token order: gathered in 16-byte pieces
      const int bt = (warp - 2 - kDqEpilogueWarps) * 32 + lane;
      const int chunk = bt & 7, row0 = bt >> 3;              // rows row0 + 8 j, 16-byte chunk `chunk` of each
      const uint32_t x_stride16 = (uint32_t)(p.x_stride >> 3);
      const uint32_t dst_thread = smem_u32(smem) + swz(row0, chunk);
      uint32_t* const row_tab = reinterpret_cast<uint32_t*>(smem + pl.off_rows);
      int done = 0, tcount = 0;                              // one stage in flight behind the one being issued
      auto hand_over = [&]() {
        fence_proxy_async_smem();     // the copies are visible to the tensor core (async proxy)
        __syncwarp();
        warp_arrive(&bar.full[dq_slot(pl, done).s]);
        ++done;
      };
      for (int w = first; w < n_tiles; w += step, ++tcount) {
        const DqTile t = dq_tile(p, pl, pref, w, n_nt, fw);
        // offsets of the tile's rows (16-byte units) in a table of the two token warps; the tables of two tiles
        // alternate, and a warp refills one only after both have left the tile before
        uint32_t* const rows = row_tab + (tcount & 1) * kDqMaxTokens;
        for (int r = bt; r < t.count; r += 32 * kDqTokenWarps) {
          const int sp = t.row_start + r;
          rows[r] = (uint32_t)(p.x_rows ? __ldg(p.x_rows + sp) : sp) * x_stride16;
        }
        named_bar_sync(1, 32 * kDqTokenWarps);
        const uint32_t sub_bytes = (uint32_t)dq_box_rows(p, pl, t) * 128u;
        for (int j = 0; j < walk_subs; j += pl.subs, ++it) {
          const DqSlot at = dq_slot(pl, it);
          if (at.use > 0 && !warp_wait(&bar.empty[at.s], (at.use - 1) & 1, spin)) {
            if (lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, 540 + at.s);
            spin = 1;
          }
          const int n_sub = min(pl.subs, slice_subs - j);
          for (int c = 0; c < n_sub; ++c) {
            uint32_t dst = dst_thread + (uint32_t)(at.s * pl.subs) * step_bytes + (uint32_t)c * sub_bytes;
            const uint4* src = reinterpret_cast<const uint4*>(p.x) + ((uint32_t)(4 * rs_lo + j + c) * 8u + (uint32_t)chunk);
#pragma unroll 8
            for (int r = row0; r < t.count; r += 8, dst += 1024u)
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + rows[r]) : "memory");
          }
          asm volatile("cp.async.commit_group;" ::: "memory");
          if (it > done) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            hand_over();
          }
        }
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      while (done < it) hand_over();
    }
  } else if (warp < T::FIRST_EXPAND) {
    // =========================== raw weight bytes, in 4-byte pieces (narrow types only) =====================
    if (!pl.raw_tma) {
      constexpr int LT = T::COPY_WARPS > 0 ? 32 * T::COPY_WARPS : 32;
      const int lt = (warp - 2 - kDqEpilogueWarps - kDqTokenWarps) * 32 + lane;
      uint32_t spin = kDqSpin;
      int slot = 0, ph = 0;
      bool wrapped = false;
      const int64_t tensor_bytes = (int64_t)p.n_experts * p.n * p.w_row_bytes;
      for (int w = first; w < n_tiles; w += step) {
        const DqTile t = dq_tile(p, pl, pref, w, n_nt, fw);
        const int rows_valid = min(fw, p.n - t.n0);
        const int64_t tile_off = ((int64_t)t.expert * p.n + t.n0) * p.w_row_bytes;
        for (int rs = rs_lo; rs < rs_hi; ++rs) {
          if (wrapped && !warp_wait(&bar.empty_r[slot], ph ^ 1, spin)) {
            if (lane == 0) report_status(p.status, HQ_DEV_WAIT_TIMEOUT, 570 + slot);
            spin = 1;
          }
          const uint32_t dst = smem_u32(smem + pl.off_raw) + (uint32_t)slot * T::STAGE;
#pragma unroll 4
          for (int i = lt; i < 128 * T::CH; i += LT) {
            const int row = i / T::CH, ch = i - row * T::CH;
            const int bank = two ? row >> 6 : 0;
            const int fr = two ? row & 63 : row;
            const uint8_t* base = reinterpret_cast<const uint8_t*>(bank == 0 ? p.w : p.w_up);
            const int64_t off = tile_off + (int64_t)fr * p.w_row_bytes + rs * T::SB;
            // down to the 4-byte boundary; the last word of the tensor may hold two bytes only
            const int64_t at = (off & ~(int64_t)3) + 4 * ch;
            const int64_t left = tensor_bytes - at;
            const int sz = left >= 4 ? 4 : (int)left;
            if (fr < rows_valid && left > 0)
              asm volatile("cp.async.ca.shared.global.L2::128B [%0], [%1], 4, %2;" ::"r"(dst + (uint32_t)row * T::PITCH +
                                                                                         (uint32_t)ch * 4u),
                           "l"(base + at), "r"(sz)
                           : "memory");
          }
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&bar.full_r[slot])) : "memory");
          if (++slot == pl.nr) { slot = 0; ph ^= 1; wrapped = true; }
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  } else {
    // =========================== expansion ==============================================================
    const int ew = warp - T::FIRST_EXPAND;
    const int quarter = warp & 3;      // the tensor-memory lane quarter a warp may write
    dq_expand_warps<FMT, ODD>(p, pl, smem, n_tiles, n_nt, rs_lo, rs_hi, first, step, tmem_base, ew >> 2, quarter, lane);
  }

  tc_fence_before();
  __syncthreads();
  if (S > 1) {      // no CTA leaves while a peer may still write into its shared memory
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace hq
