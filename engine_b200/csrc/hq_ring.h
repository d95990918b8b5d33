// Which slot and which barrier phase a stage of a ring of buffers uses, and which stages a copying warp waits for before its
// CTA exits.  Plain arithmetic, the same on the host (tests/test_ring_protocol.py) and in the kernels.
//
// A slot's barrier tells "use u is complete" from "use u - 1 is" by one parity bit, so a wait for use u is only sound while
// use u - 1 is known to be complete and use u + 1 cannot be: otherwise the bit reads the wrong way round, as complete too
// early or as incomplete for good.
#pragma once

#ifdef __CUDACC__
#define HQ_RING_FN __host__ __device__ __forceinline__
#else
#define HQ_RING_FN inline
#endif

namespace hq {

HQ_RING_FN int ring_slot(int stage, int slots) { return stage % slots; }
HQ_RING_FN int ring_parity(int stage, int slots) { return (stage / slots) & 1; }

// The stages whose copies a warp waits for when it has left its loop in front of stage `next` (the length of the sequence, or
// where a wait ran out): its own -- of `warps` (1 or 2) that take the stages in turn -- among the last `slots`.  They are the last
// uses of their slots, so no later copy moves their barriers on, and the warp issued them, so the use before is known to be
// complete.  A slot's older stages were consumed before its last one was issued.  (A warp that waits for its last two stages
// whatever the ring's length polls, with three slots, one that another warp has used again by then.)
// `slot`, `parity`: the slot stage `next` would take, the parity of its last use.  False: a wait ran out.
template <typename Wait>
HQ_RING_FN bool ring_drain(int next, int slots, int slot, int parity, int warps, int me, Wait wait) {
#ifdef __CUDACC__
#pragma unroll 1
#endif
  for (int i = next - slots; i < next; ++i) {
    if (i >= 0 && (i & (warps - 1)) == me && !wait(slot, parity)) return false;
    if (++slot == slots) { slot = 0; parity ^= 1; }
  }
  return true;
}

// Dequantizing GEMM, tiles of `steps` 64-k steps, `subs` of them per operand stage.  A group of expanding warps serves every
// stage (subs = 4), or every second one of a tile (subs = 2): then the group of the odd ones gets from its last stage of a tile to
// its first of the next three stages on when a tile has an odd number.  Its wait in front of stage j (stage j - slots consumed)
// needs stage j - 2 slots to be known as consumed, and the one in front of stage j - 3 has shown that of stage j - 3 - slots:
// enough with three slots, one short with two.  There a tile is walked for one more stage, without products.
HQ_RING_FN bool dq_odd_on_two_slots(int subs, int slots, int steps) {
  return subs == 2 && slots == 2 && (((steps + 1) >> 1) & 1) != 0;
}
// ... the steps for which the roles walk a tile, `odd`: the above of any of the launch's K slices
HQ_RING_FN int dq_walk_steps(bool odd, int steps) { return odd ? (steps + 3) & ~3 : steps; }

}  // namespace hq
