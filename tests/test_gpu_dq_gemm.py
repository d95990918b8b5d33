"""The dequantizing GEMM at the edges of its plans: token tiles of 16 .. 256 columns (one or two accumulator buffers, two
or four 64-k steps per stage), K slices over clusters, K tails, and weight rows whose pitch is not a multiple of 16 bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from oracle import moe as M
from tests import hq_testlib as T
from tests.test_gpu_linear import TOL, run_case

DEV = "cuda:0"


@pytest.mark.parametrize("m", [9, 16, 17, 64, 65, 128, 129, 192, 193, 256, 257, 521])
@pytest.mark.parametrize("fmt,n,k", [("Q4_K", 200, 1280), ("FP8", 576, 640), ("MXFP4", 130, 320)])
def test_token_tile_edges(fmt, n, k, m):
    # MXFP4: K = 320 ends in a stage with one 64-k step; FP8: N = 576 ends in half a 128-row scale block, K = 640 in half
    # a 256-k stage; few features: K is cut into slices, no CTA meets a second tile
    got, want = run_case(fmt, n, k, m, torch.float16, torch.float32, 700 + m, bias=True)
    assert T.rel_l2(got, want) <= TOL[fmt]


@pytest.mark.parametrize("k", [256, 768, 2048, 4096])
@pytest.mark.parametrize("fmt", ["Q6_K", "Q3_K", "Q2_K"])
def test_narrow_rows_copied_as_boxes_and_in_words(fmt, k):
    # K = 2048 and 4096: row pitch a multiple of 16 bytes, blocks at every even offset of a 16-byte unit; else words
    got, want = run_case(fmt, 300, k, 40, torch.bfloat16, torch.float32, 720)
    assert T.rel_l2(got, want) <= TOL[fmt]


@pytest.mark.parametrize("m", [20, 300])
@pytest.mark.parametrize("fmt", ["Q4_K", "Q5_1", "FP8"])
def test_gate_and_up_bank(fmt, m):
    import engine_b200 as hq
    rng = T.rng_for(7, m)
    n, k = 320, 1024
    (ga, gd), (ua, ud) = T.make_weight(fmt, rng, n, k), T.make_weight(fmt, rng, n, k)
    x = T.to_dev(rng.standard_normal((m, k)).astype(np.float32), torch.float16, DEV)
    gate, up = T.make_layer(fmt, ga, k, DEV), T.make_layer(fmt, ua, k, DEV)
    got = hq.try_fused_quantized_gate_up(x, gate, up, out_dtype=torch.float32).cpu().numpy()
    xf = x.float().cpu().numpy()
    want = M.swiglu(M.dense_forward(xf, gd), M.dense_forward(xf, ud))
    assert gate.device_status()[0] == 0
    assert T.rel_l2(got, want) <= 2e-3


@pytest.mark.parametrize("per_expert", [9, 40, 150, 300])
def test_expert_rows_cut_into_equal_tiles(per_expert):
    # skewed counts: experts without rows, with a few, and with more than one tile
    import engine_b200 as hq
    rng = T.rng_for(8, per_expert)
    e, n, k, topk = 4, 192, 512, 2
    arrays, deq = T.make_weight("Q4_K", rng, n, k, experts=e)
    t = per_expert * e // topk
    ids = np.stack([rng.choice(e - 1, size=topk, replace=False, p=[0.7, 0.25, 0.05]) for _ in range(t)]).astype(np.int32)
    x = T.to_dev(rng.standard_normal((t, k)).astype(np.float32), torch.bfloat16, DEV)
    layer = T.make_layer("Q4_K", arrays, k, DEV)
    got = layer.gather_forward_raw(x, T.to_dev(ids, torch.int32, DEV), torch.float32).cpu().numpy()
    want = np.einsum("tk,tsnk->tsn", x.float().cpu().numpy(), deq[ids])
    assert layer.device_status()[0] == 0
    assert T.rel_l2(got, want) <= 1e-3


@pytest.mark.parametrize("m", [1, 8])
@pytest.mark.parametrize("byte", [112, 113, 140, 141])
def test_mxfp4_rows_by_scale_range(byte, m):
    # e8m0 bytes 113 .. 140 are exact f16 operands: any row count takes the tensor cores; beyond, few rows do not
    from engine_b200 import _lib as L
    from engine_b200.quant import MXFP4Layer, tensor_path_expected
    n, k = 192, 320
    g = torch.Generator().manual_seed(byte)
    blocks = torch.randint(0, 256, (n, k // 2), generator=g, dtype=torch.uint8)
    scales = torch.randint(113, 141, (n, k // 32), generator=g, dtype=torch.uint8)
    scales[5, 3], scales[7, 1] = byte, 0
    layer = MXFP4Layer(blocks.to(DEV), scales.to(DEV))
    inside = 113 <= byte <= 140
    assert bool(layer._weight_struct().flags & L.WEIGHT_F16_SCALES) == inside
    assert tensor_path_expected(layer, m, dense=True) == inside
    x = torch.randn((m, k), generator=g).to(DEV, torch.bfloat16)
    got = layer.forward_raw(x, torch.float32)
    assert layer.device_status()[0] == 0
    want = x.double() @ layer.dequantize_w().double().t()
    assert float((got.double() - want).norm() / want.norm()) <= 1e-5


def _plan(fmt, n, k, experts, rows):
    import ctypes as C
    from engine_b200 import _lib as L
    out = (C.c_int32 * 8)()
    f = L.lib().hq_dq_gemm_plan
    f.argtypes = [C.c_int32, C.c_int64, C.c_int64, C.c_int32, C.c_int32, C.c_int64, C.c_void_p]
    assert f({"FP8": L.FMT_FP8_BLOCK, "MXFP4": L.FMT_MXFP4}[fmt], n, k, experts, 0, rows, out) == 0
    return dict(zip(("tn", "subs", "ns", "nr", "nbuf", "kslices", "grid"), out))


def _odd_tiles_on_two_slots(fmt, n, k, experts, rows):
    """The case is what its name says: tiles with an odd number of stages, two operand slots, a second tile for every CTA."""
    pl = _plan(fmt, n, k, experts, rows)
    assert (pl["subs"], pl["ns"], pl["kslices"]) == (2, 2, 1) and -(-k // 128) % 2 == 1, pl
    tiles = experts if experts > 1 else -(-rows // pl["tn"])
    assert tiles * (-(-n // 128)) >= 2 * pl["grid"], pl


@pytest.mark.parametrize("fmt,n,k,m", [("FP8", 5120, 1408, 2048), ("MXFP4", 3584, 320, 2432), ("FP8", 3584, 640, 2432)])
def test_odd_stage_counts_over_several_tiles(fmt, n, k, m):
    _odd_tiles_on_two_slots(fmt, n, k, 1, m)
    rng = T.rng_for(8, k)
    arrays, deq = T.make_weight(fmt, rng, n, k)
    layer = T.make_layer(fmt, arrays, k, DEV)
    x = T.to_dev(rng.standard_normal((m, k)).astype(np.float32), torch.float16, DEV)
    y = layer.forward_raw(x, torch.float32)
    for _ in range(20):
        assert torch.equal(layer.forward_raw(x, torch.float32), y)
    assert layer.device_status()[0] == 0
    assert T.rel_l2(y.cpu().numpy(), M.dense_forward(x.float().cpu().numpy(), deq, None)) <= TOL[fmt]


def test_odd_stage_counts_over_several_expert_tiles():
    # rows gathered in token order
    e, n, k, topk, t = 16, 3072, 320, 2, 1200
    _odd_tiles_on_two_slots("MXFP4", n, k, e, t * topk)
    rng = T.rng_for(8, 2)
    arrays, deq = T.make_weight("MXFP4", rng, n, k, experts=e)
    layer = T.make_layer("MXFP4", arrays, k, DEV)
    x = T.to_dev(rng.standard_normal((t, k)).astype(np.float32), torch.float16, DEV)
    ids = np.stack([rng.choice(e, size=topk, replace=False) for _ in range(t)]).astype(np.int32)
    ids_dev = T.to_dev(ids, torch.int32, DEV)
    y = layer.gather_forward_raw(x, ids_dev, torch.float32)
    for _ in range(20):
        assert torch.equal(layer.gather_forward_raw(x, ids_dev, torch.float32), y)
    assert layer.device_status()[0] == 0
    some = rng.choice(t, 100, replace=False)
    want = np.einsum("tk,tsnk->tsn", x.float().cpu().numpy()[some], deq[ids[some]])
    assert T.rel_l2(y.cpu().numpy()[some], want) <= TOL["MXFP4"]
