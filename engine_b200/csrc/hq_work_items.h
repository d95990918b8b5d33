// Work items of the expert-indexed decode kernels, and where the dispatch tables keep them in a call's workspace.  Plain
// arithmetic on 32-bit words, the same on the host (tests/test_work_items.py) and in the kernels: a workspace may start at any
// word, and the lists can be read without the sizes they were built with (a projection that takes one row per slot may call itself
// n_tokens * top_k tokens of one slot).
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define HQ_ITEM_FN __host__ __device__ __forceinline__
#else
#define HQ_ITEM_FN inline
#endif

namespace hq {

// Rows of a work item: 4 when every expert can have at most 4 rows (no token picks an expert twice), 8 otherwise.
constexpr int kDecodeShortTile = 4;

// workspace: 4 header words (items, routed assignments, word at which the items' rows start), two words per item (expert, first
// sorted row), one word per item (its rows: a look at the expert's bounds would wait for the first word)
constexpr int64_t kItemsAt = 4;
constexpr int kHeaderRowsAt = 2;

struct DispatchLayout {
  int tile_rows;         // rows of a work item
  int64_t rows_at, max_items;
  int64_t total_words;
};
HQ_ITEM_FN constexpr DispatchLayout dispatch_layout(int64_t n_tokens, int top_k, int n_experts) {
  const int rows = n_tokens <= kDecodeShortTile ? kDecodeShortTile : 8;
  const int64_t items = (n_tokens * top_k + rows - 1) / rows + n_experts;
  return DispatchLayout{rows, kItemsAt + 2 * items, items, kItemsAt + 3 * items};
}

// Shared memory of the kernels that build the tables: histogram rows and five arrays of one word per expert, sized by the launch,
// beside at most kDispatchStatic bytes the kernel declares.  A launch gets 48 KiB of both together unless it asked for more, and
// 227 KiB at most.
constexpr int64_t kDispatchStatic = 4096;
HQ_ITEM_FN constexpr int dispatch_rows(int n_experts) { return n_experts <= 1024 ? 32 : 8; }      // warps that own a run
HQ_ITEM_FN constexpr int64_t dispatch_smem(int n_experts) { return (int64_t)(dispatch_rows(n_experts) + 5) * n_experts * 4; }
constexpr int64_t kDispatchDynamic = 227 * 1024 - kDispatchStatic;
HQ_ITEM_FN constexpr bool dispatch_asks_for_smem(int64_t dynamic) { return dynamic + kDispatchStatic > 48 * 1024; }

// Largest workspace of up to `assignments` (more than 256, a multiple of 8) over `experts`, however they split into tokens and
// slots (up to 64): what a fixed array has to hold.
HQ_ITEM_FN constexpr int64_t dispatch_words_up_to(int64_t assignments, int experts) {
  return dispatch_layout(assignments, 1, experts).total_words;
}
// The reference-named entry points keep all five tables in one fixed array, each from a multiple of 64 words on.
constexpr int kCompatMaxAssign = 65536;
constexpr int kCompatMaxExperts = 512;
HQ_ITEM_FN constexpr int64_t up64(int64_t words) { return (words + 63) / 64 * 64; }
HQ_ITEM_FN constexpr int64_t compat_words(int64_t assignments, int experts, int64_t ws_words) {
  return up64(experts + 1) + 3 * up64(assignments) + up64(ws_words);
}
constexpr int64_t kCompatWords =
    compat_words(kCompatMaxAssign, kCompatMaxExperts, dispatch_words_up_to(kCompatMaxAssign, kCompatMaxExperts));

struct DecodeItem {
  int32_t expert, row0, rows;      // row0: first sorted row
};
// ws: the workspace; rows_at: its header's word, or the layout's
HQ_ITEM_FN DecodeItem decode_item(const int32_t* ws, int rows_at, int i) {
  const int32_t* w = ws + kItemsAt + 2 * (int64_t)i;
  return DecodeItem{w[0], w[1], ws[rows_at + (int64_t)i]};
}
HQ_ITEM_FN void put_decode_item(int32_t* ws, int rows_at, int i, int32_t expert, int32_t row0, int32_t rows) {
  int32_t* w = ws + kItemsAt + 2 * (int64_t)i;
  w[0] = expert;
  w[1] = row0;
  ws[rows_at + (int64_t)i] = rows;
}

}  // namespace hq
