"""Decode paths that run several small launches into one another: dispatch tables built by comparison (up to 256 assignments)
and by sorting above, with the rows that their work items carry; query, key and value projections of one activation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from tests import hq_testlib as T
from tests.test_gpu_dispatch import test_tables_match_a_stable_sort as tables_match

DEV = "cuda:0"


@pytest.mark.parametrize("e", [1, 33, 256, 1024, 4096])
@pytest.mark.parametrize("t,k", [(1, 8), (4, 8), (31, 8), (32, 8), (256, 1), (257, 1), (33, 8)])
def test_tables_around_the_line(t, k, e):
    tables_match(t, k, e)


# the tables' histogram of 318 .. 332 experts fits 48 KiB of shared memory, but not beside what the kernel declares
@pytest.mark.parametrize("e", [317, 318, 320, 332, 333])
@pytest.mark.parametrize("t", [4, 64])
def test_tables_around_48_kib(t, e):
    tables_match(t, 8, e)


@pytest.mark.parametrize("t,k,e", [(3, 8, 128), (32, 8, 16), (40, 8, 16)])
def test_items_carry_their_rows(t, k, e):
    from engine_b200.quant import moe_dispatch_build
    ids = torch.from_numpy(T.rng_for(13, t).integers(0, e // 2, (t, k)).astype(np.int32)).to(DEV)
    tab = moe_dispatch_build(ids, e)
    w = 4 if t <= 4 else 8
    ws, b = tab.workspace.view(torch.int32).tolist(), tab.expert_bounds.tolist()
    want = [min(w, b[x + 1] - r) for x in range(e) for r in range(b[x], b[x + 1], w)]
    at = 4 + 2 * ((t * k + w - 1) // w + e)
    assert ws[at:at + ws[0]] == want


@pytest.mark.parametrize("fmts", [("Q8_0",) * 3, ("Q4_K",) * 3, ("FP8",) * 3])
@pytest.mark.parametrize("m", [1, 2, 3, 8, 9])
def test_a_run_of_projections_is_the_separate_calls(fmts, m):
    import engine_b200 as hq
    rng = T.rng_for(13, 9)
    k = 1024
    layers = [T.make_layer(f, T.make_weight(f, rng, n, k)[0], k, DEV) for f, n in zip(fmts, (1024, 256, 384))]
    for i in range(3):                                    # several in a row: each run's first launch follows the last's last
        x = T.to_dev(rng.standard_normal((m, k)).astype(np.float32), torch.bfloat16, DEV)
        outs = hq.try_fused_quantized_qkv(x, *layers, out_dtype=torch.float32)
        for o, layer in zip(outs, layers):
            assert torch.equal(o, layer.forward_raw(x, torch.float32))


@pytest.mark.parametrize("fmt", ["Q8_0", "Q4_K", "FP8"])
@pytest.mark.parametrize("m", [1, 2])
def test_a_run_reads_what_the_launch_before_it_wrote(fmt, m):
    # one activation buffer, written anew in place before every run: by torch, then by a projection of this library, whose launch
    # the run's first one follows programmatically; no synchronisation in between
    import engine_b200 as hq
    from engine_b200 import _lib as L
    import ctypes as C
    rng = T.rng_for(13, 21)
    k = 2048
    o, q, kk, v = [T.make_layer(fmt, T.make_weight(fmt, rng, n, k)[0], k, DEV) for n in (k, 2048, 256, 384)]
    steps = 40
    inputs = T.to_dev(rng.standard_normal((steps, m, k)).astype(np.float32), torch.float32, DEV)
    want = []
    for i in range(steps):
        x = o.forward_raw(inputs[i], torch.float32)
        torch.cuda.synchronize()
        want.append([layer.forward_raw(x, torch.float32) for layer in (q, kk, v)])
        torch.cuda.synchronize()
    x = torch.empty((m, k), dtype=torch.float32, device=DEV)
    w, stream = o._weight_struct(), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    got = []
    for i in range(steps):
        L.check(L.lib().hq_linear_forward(C.byref(w), C.c_void_p(inputs[i].data_ptr()), L.DT_F32, k, C.c_void_p(x.data_ptr()), L.DT_F32,
                                          k, m, None, stream), "hq_linear_forward")
        got.append(hq.try_fused_quantized_qkv(x, q, kk, v, out_dtype=torch.float32))
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        for s, t in zip(a, b):
            assert torch.equal(s, t)
    for i in range(steps):
        x.copy_(inputs[i])
        got[i] = hq.try_fused_quantized_qkv(x, q, kk, v, out_dtype=torch.float32)
    for i in range(steps):
        for s, layer in zip(got[i], (q, kk, v)):
            assert torch.equal(s, layer.forward_raw(inputs[i], torch.float32))
