"""Host model of the barrier protocols of the GEMM kernels' rings: mbarriers with arrival counts, transaction bytes and one
parity bit, the roles as coroutines that a random scheduler advances one step at a time, copies and MMAs that complete
some time after they were issued (MMAs in order).  The index arithmetic under test is the kernels' own
(engine_b200/csrc/hq_ring.h, compiled for the host).  A run is right when every role reaches its end, nothing is written
that has not been read, and no barrier is arrived on more often than its count."""
import ctypes as C
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    out = tmp_path_factory.mktemp("ring")
    src, lib = str(out / "ring.cpp"), str(out / "ring.so")
    with open(src, "w") as f:
        f.write('#include "hq_ring.h"\n'
                'extern "C" int slot(int i, int n) { return hq::ring_slot(i, n); }\n'
                'extern "C" int parity(int i, int n) { return hq::ring_parity(i, n); }\n'
                'extern "C" int drain(int next, int n, int s, int ph, int w, int me, int* out) {\n'
                '  int k = 0;\n'
                '  hq::ring_drain(next, n, s, ph, w, me, [&](int a, int b) { out[k++] = 2 * a + b; return true; });\n'
                '  return k; }\n'
                'extern "C" int walk(int subs, int n, int steps) {\n'
                '  return hq::dq_walk_steps(hq::dq_odd_on_two_slots(subs, n, steps), steps); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "engine_b200", "csrc"), src, "-o", lib],
                   check=True)
    return C.CDLL(lib)


class Wrong(Exception):
    pass


class Bar:
    def __init__(self, count):
        self.count = self.pending = count
        self.done, self.tx = 0, 0             # completed phases; bytes still expected in this one

    def arrive(self, expect=0):
        if self.pending == 0:
            raise Wrong("arrival beyond the count")
        self.pending -= 1
        self.tx += expect
        self._turn()

    def complete(self, n):
        self.tx -= n
        self._turn()

    def _turn(self):
        if self.pending == 0 and self.tx == 0:
            self.done, self.pending = self.done + 1, self.count

    def passed(self, parity):
        """What a wait on the parity bit sees: the phase running now is not of this parity."""
        return (self.done & 1) != parity


class Machine:
    """Roles yield None (a step) or a barrier and the parity they wait for."""

    def __init__(self, seed):
        self.rng, self.roles, self.copies, self.mmas = random.Random(seed), {}, [], []

    def role(self, name, gen):
        self.roles[name] = [gen, None]

    def run(self):
        while True:
            ready = [n for n, (_, w) in self.roles.items() if w is None or w[0].passed(w[1])]
            acts = [("role", n) for n in ready] + [("copy", i) for i in range(len(self.copies))] + \
                   ([("mma", 0)] if self.mmas else [])
            if not acts:
                if self.roles:
                    raise Wrong("stuck: " + ", ".join(sorted(self.roles)))
                return
            kind, which = self.rng.choice(acts)
            if kind == "copy":
                self.copies.pop(which)()
            elif kind == "mma":
                self.mmas.pop(0)()
            else:
                slot = self.roles[which]
                try:
                    slot[1] = next(slot[0])
                except StopIteration:
                    del self.roles[which]


# ---- block-scaled expert GEMM: two copy warps that take the stages in turn --------------------------------------------

def block_scaled(ring, slots, stages, seed, drain):
    m = Machine(seed)
    full, empty = [Bar(1 + 1) for _ in range(slots)], [Bar(1) for _ in range(slots)]
    held = [None] * slots                     # the stage whose bytes lie in the slot and have not been read

    def copy_warp(me):
        for i in range(stages):
            if i % 2 != me:
                continue
            s = ring.slot(i, slots)
            if i >= slots:
                yield empty[s], ring.parity(i - slots, slots)
            if held[s] is not None:
                raise Wrong("copy over an unread stage")
            held[s] = i
            full[s].arrive(1)
            m.copies.append(lambda s=s: full[s].complete(1))
            yield None
        for s, parity in drain(stages, slots, me):
            yield full[s], parity

    def scale_warps(me):
        for i in range(me, stages, 2):
            s = ring.slot(i, slots)
            if i >= slots:
                yield empty[s], ring.parity(i - slots, slots)
            full[s].arrive()
            yield None

    def mma_warp():
        def finish(s, i):
            if held[s] != i:
                raise Wrong("multiplied the wrong stage")
            held[s] = None
            empty[s].arrive()
        for i in range(stages):
            s = ring.slot(i, slots)
            yield full[s], ring.parity(i, slots)
            m.mmas.append(lambda s=s, i=i: finish(s, i))
            yield None

    for me in (0, 1):
        m.role(f"copy {me}", copy_warp(me))
        m.role(f"scale {me}", scale_warps(me))
    m.role("mma", mma_warp())
    m.run()
    if m.copies:
        raise Wrong("copies in flight at the end")


def kernel_drain(ring, copy_warps=2):
    def drain(stages, slots, me):
        out = (C.c_int * slots)()
        n = ring.drain(stages, slots, ring.slot(stages, slots), ring.parity(stages, slots) ^ 1, copy_warps, me, out)
        return [(v // 2, v % 2) for v in out[:n]]
    return drain


@pytest.mark.parametrize("slots", range(2, 13))
def test_the_last_use_of_every_slot_is_drained_once(ring, slots):
    for stages in range(40):
        last = [(i % slots, i // slots % 2) for i in range(max(0, stages - slots), stages)]
        assert kernel_drain(ring, 1)(stages, slots, 0) == last
        halves = [kernel_drain(ring, 2)(stages, slots, me) for me in (0, 1)]
        assert sorted(halves[0] + halves[1]) == sorted(last)


@pytest.mark.parametrize("slots", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("stages", [1, 2, 3, 5, 8, 13, 24, 39])
def test_block_scaled_gemm_ends(ring, slots, stages):
    for seed in range(40):
        block_scaled(ring, slots, stages, seed, kernel_drain(ring))


def test_the_model_finds_a_wait_that_a_later_use_has_overtaken(ring):
    # each warp's own last two stages whatever the ring's length: with two and three slots one of them has been used again
    def own(stages, slots, me):
        last = [i for i in range(stages - 1, -1, -1) if i % 2 == me][:2]
        return [(i % slots, i // slots % 2) for i in last]

    for slots, found in ((2, True), (3, True), (4, False), (6, False)):
        stuck = 0
        for seed in range(100):
            try:
                block_scaled(ring, slots, 24, seed, own)
            except Wrong:
                stuck += 1
        assert (stuck > 0) == found, (slots, stuck)


# ---- dequantizing GEMM: raw ring, four expanding groups, operand ring --------------------------------------------------

def dequantizing(ring, slots, raw_slots, subs, steps, tiles, seed, walk):
    """`steps` 64-k steps per tile; a raw stage holds four, an operand stage `subs`."""
    m = Machine(seed)
    tile_stages, raw_stages = -(-walk(subs, slots, steps) // subs), -(-steps // 4)
    full, empty = [Bar(subs + 1) for _ in range(slots)], [Bar(1) for _ in range(slots)]
    full_r, empty_r = [Bar(1) for _ in range(raw_slots)], [Bar(4) for _ in range(raw_slots)]
    acc_full, acc_empty = [Bar(1) for _ in range(2)], [Bar(1) for _ in range(2)]
    operand = {}                              # (slot, step within the stage) -> stage written and not multiplied yet

    def raw_warp(me):
        for r in range(tiles * raw_stages):
            if r % 2 != me:
                continue
            s = ring.slot(r, raw_slots)
            if r >= raw_slots:
                yield empty_r[s], ring.parity(r - raw_slots, raw_slots)
            full_r[s].arrive(1)
            m.copies.append(lambda s=s: full_r[s].complete(1))
            yield None
        for s, parity in kernel_drain(ring)(tiles * raw_stages, raw_slots, me):
            yield full_r[s], parity

    def group(c):
        stage, sub = c // subs, c % subs
        for t in range(tiles):
            for rs in range(raw_stages):
                r = t * raw_stages + rs
                yield full_r[ring.slot(r, raw_slots)], ring.parity(r, raw_slots)
                local = rs * (4 // subs) + stage
                i = t * tile_stages + local
                s = ring.slot(i, slots)
                live = 4 * rs + c < steps
                if not live:
                    empty_r[ring.slot(r, raw_slots)].arrive()
                    if local >= tile_stages:
                        continue
                if i >= slots:
                    yield empty[s], ring.parity(i - slots, slots)
                if live:
                    if operand.get((s, sub)) is not None:
                        raise Wrong("expanded over an unread operand")
                    operand[s, sub] = i
                    empty_r[ring.slot(r, raw_slots)].arrive()
                    yield None
                full[s].arrive()

    def token_warp():
        for i in range(tiles * tile_stages):
            s = ring.slot(i, slots)
            if i >= slots:
                yield empty[s], ring.parity(i - slots, slots)
            full[s].arrive(1)
            m.copies.append(lambda s=s: full[s].complete(1))
            yield None
        for s, parity in kernel_drain(ring, 1)(tiles * tile_stages, slots, 0):
            yield full[s], parity

    def mma_warp():
        def finish(s, i, n):
            for sub in range(n):
                if operand.pop((s, sub), None) != i:
                    raise Wrong("multiplied the wrong operand")
            empty[s].arrive()
        for t in range(tiles):
            if t >= 2:
                yield acc_empty[t % 2], ring.parity(t - 2, 2)
            for j in range(tile_stages):
                i = t * tile_stages + j
                s = ring.slot(i, slots)
                yield full[s], ring.parity(i, slots)
                m.mmas.append(lambda s=s, i=i, n=min(subs, steps - j * subs): finish(s, i, n))
                yield None
            m.mmas.append(lambda t=t: acc_full[t % 2].arrive())

    def epilogue():
        for t in range(tiles):
            yield acc_full[t % 2], ring.parity(t, 2)
            yield None
            acc_empty[t % 2].arrive()

    for me in (0, 1):
        m.role(f"raw {me}", raw_warp(me))
    for c in range(4):
        m.role(f"group {c}", group(c))
    for name, gen in (("tokens", token_warp()), ("mma", mma_warp()), ("epilogue", epilogue())):
        m.role(name, gen)
    m.run()


@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 22, 45])
@pytest.mark.parametrize("slots,raw_slots,subs", [(2, 2, 2), (2, 5, 2), (3, 3, 2), (4, 2, 2), (2, 2, 4), (4, 4, 4)])
def test_dequantizing_gemm_rings(ring, slots, raw_slots, subs, steps):
    for seed in range(30):
        dequantizing(ring, slots, raw_slots, subs, steps, 5, seed, ring.walk)


def test_the_model_finds_a_slot_two_uses_behind(ring):
    # tiles walked for their own stages only: wrong with two slots and an odd number of them
    for slots, steps, found in ((2, 5, True), (2, 10, True), (2, 45, True), (2, 8, False), (3, 5, False), (3, 45, False)):
        wrong = 0
        for seed in range(300):
            try:
                dequantizing(ring, slots, 5, 2, steps, 5, seed, lambda subs, n, k: k)
            except Wrong:
                wrong += 1
        assert (wrong > 0) == found, (slots, steps, wrong)
