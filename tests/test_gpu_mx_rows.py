"""MXFP4 expert layers with few rows per expert on the block-scaled MMA (three or four e5m2 terms per activation), against the
oracle's dequantized weights.  The products are exact and the sums f32, so what separates the f32 output from the oracle is the
f16 rounding of the intermediate, which the oracle applies too: a value next to a rounding boundary may fall to either side,
2^-11 of itself, so the tolerance of the MXFP4 layers (2e-3) holds with a wide margin."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from oracle import moe as M
from tests import hq_testlib as T

DEV = "cuda:0"


def _layer(e, h, i, seed):
    import engine_b200 as hq
    from engine_b200 import _lib as L
    rng = T.rng_for(31, seed)
    gu_a, gu = T.make_weight("MXFP4", rng, 2 * i, h, experts=e)
    d_a, d = T.make_weight("MXFP4", rng, h, i, experts=e)
    gub = T.to_dev(rng.normal(0, 0.02, (e, 2 * i)).astype(np.float32), torch.bfloat16, DEV)
    db = T.to_dev(rng.normal(0, 0.02, (e, h)).astype(np.float32), torch.bfloat16, DEV)
    experts = hq.MoEExperts(T.make_layer("MXFP4", d_a, i, DEV, db), gate_up_proj=T.make_layer("MXFP4", gu_a, h, DEV, gub),
                            act=L.ACT_GPTOSS, limit=7.0)

    def want(x, ids, w):
        return M.moe_layer(x, ids, w, None, None, d, L.ACT_GPTOSS, gate_up_bank=gu, gate_up_bias=gub.float().cpu().numpy(),
                           down_bias=db.float().cpu().numpy(), limit=7.0, h_round=lambda a: a.astype(np.float16).astype(np.float32))
    return experts, want, rng


def _run(experts, x, logits, k):
    import engine_b200 as hq
    from engine_b200 import _lib as L
    rcfg = hq.MoeRouterTopKConfig(k, L.SCORE_SOFTMAX, L.WEIGHT_SCORE, True)
    y = experts.forward_layer(x, T.to_dev(logits, torch.float32, DEV), rcfg, out_dtype=torch.float32)
    torch.cuda.synchronize()
    assert experts.gate_up.device_status()[0] == 0
    return y.cpu().numpy()


# K of 128 (one block), 192 and 320 (a last block that overlaps the one before by a half), 2880 (an odd number of blocks); N of
# 192 .. 704, whole tiles of 128 and not; 1 .. 24 rows per expert on average: one column group, 16 and 17 tokens, tiles of 96
# columns, experts without a token
@pytest.mark.parametrize("t,e,k,h,i,dtype", [(1, 4, 2, 128, 128, torch.bfloat16), (5, 4, 4, 192, 320, torch.float16),
                                             (16, 2, 2, 256, 192, torch.float32), (17, 2, 2, 320, 448, torch.bfloat16),
                                             (6, 32, 4, 576, 704, torch.bfloat16), (24, 4, 4, 320, 128, torch.float32),
                                             (23, 4, 3, 2880, 192, torch.bfloat16), (90, 16, 4, 192, 2880, torch.float16)])
def test_layer_matches_the_oracle(t, e, k, h, i, dtype):
    from engine_b200 import _lib as L
    experts, want, rng = _layer(e, h, i, t)
    x = T.to_dev(rng.standard_normal((t, h)).astype(np.float32), dtype, DEV)
    logits = rng.standard_normal((t, e)).astype(np.float32)
    ids, w = M.router_topk(logits, k, L.SCORE_SOFTMAX, L.WEIGHT_SCORE, True)
    got = _run(experts, x, logits, k)
    assert T.rel_l2(got, want(x.float().cpu().numpy(), ids, w)) <= 2e-3
    assert np.array_equal(got, _run(experts, x, logits, k))


def test_wide_ranges_and_values_that_are_not_finite():
    # a block's largest value 2^20 times its others, values no f16 holds, a zero block; then a NaN and an infinity, each of which
    # may reach its own token only (what becomes of them: the test below)
    from engine_b200 import _lib as L
    t, e, k, h, i = 7, 4, 4, 256, 128
    experts, want, rng = _layer(e, h, i, 99)
    x = rng.standard_normal((t, h)).astype(np.float32)
    x[1, 40] = 2.0 ** 20
    x[2] *= 2.0 ** -30
    x[3, 64:128] = 0.0
    x[4, 9] = -1.0e5
    xd = T.to_dev(x, torch.bfloat16, DEV)
    logits = rng.standard_normal((t, e)).astype(np.float32)
    ids, w = M.router_topk(logits, k, L.SCORE_SOFTMAX, L.WEIGHT_SCORE, True)
    got, ref = _run(experts, xd, logits, k), want(xd.float().cpu().numpy(), ids, w)
    for row in range(t):
        assert T.rel_l2(got[row], ref[row]) <= 2e-3, row
    xd[5, 17] = float("nan")
    xd[6, 200] = float("inf")
    bad = _run(experts, xd, logits, k)
    assert np.array_equal(bad[:5], got[:5])


# The clamp of a gated activation takes a NaN for its limit, in every kernel; without a limit a NaN or an infinity passes on.
# Either way a token's result must not depend on how many others are in the call: 7 tokens of 4 experts, top 4, are 7 rows an
# expert (the terms), 64 are 64 (the f16-expanding GEMM, which multiplies the same infinities).
@pytest.mark.parametrize("limit", [True, False])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_values_that_are_not_finite_are_the_same_in_any_batch(dtype, limit):
    import engine_b200 as hq
    from engine_b200 import _lib as L
    t, e, k, h, i = 7, 4, 4, 256, 128
    experts, _, rng = _layer(e, h, i, 99)
    if not limit:
        experts.act.act, experts.act.has_limit = L.ACT_SWIGLU, 0
    x = T.to_dev(rng.standard_normal((64, h)).astype(np.float32), dtype, DEV)
    x[1, 17], x[2, 200], x[3, 3] = float("nan"), float("inf"), -float("inf")
    x[4, 8], x[4, 9] = float("inf"), -float("inf")
    x[5, 32:64] = float("inf")
    logits = T.to_dev(rng.standard_normal((64, e)).astype(np.float32), torch.float32, DEV)
    rcfg = hq.MoeRouterTopKConfig(k, L.SCORE_SOFTMAX, L.WEIGHT_SCORE, True)
    few = experts.forward_layer(x[:t], logits[:t], rcfg, out_dtype=torch.float32).cpu().numpy()
    many = experts.forward_layer(x, logits, rcfg, out_dtype=torch.float32)[:t].cpu().numpy()
    assert experts.gate_up.device_status()[0] == 0
    assert np.isfinite(many[[0, 6]]).all() and np.isfinite(many[1]).all() == limit
    for row in range(t):
        ok = np.isfinite(many[row])
        assert np.array_equal(np.isnan(few[row]), np.isnan(many[row])), row
        assert np.array_equal(few[row][~ok], many[row][~ok], equal_nan=True), row
        if ok.any():
            assert T.rel_l2(few[row][ok], many[row][ok]) <= 2e-3, row


def _layer_with_dead_columns(e, h, i, seed):
    """Every 32-block's first weight of the gate/up bank is zero; the bank's other weights are 2^12 times the usual."""
    import engine_b200 as hq
    from engine_b200 import _lib as L
    from oracle import formats as F
    rng = T.rng_for(31, seed)
    gu_a, _ = T.make_weight("MXFP4", rng, 2 * i, h, experts=e)
    d_a, d = T.make_weight("MXFP4", rng, h, i, experts=e)
    blocks, scales = gu_a["blocks"].copy(), gu_a["scales"] + 12
    blocks.reshape(-1, 16)[:, 0] &= 0xF0
    gu = F.mxfp4_dequant(blocks.reshape(-1, h // 2), scales.reshape(-1, h // 32)).reshape(e, 2 * i, h)
    assert (gu[..., ::32] == 0).all() and scales.min() >= 113 and scales.max() <= 140
    experts = hq.MoEExperts(T.make_layer("MXFP4", d_a, i, DEV), gate_up_proj=T.make_layer("MXFP4", {"blocks": blocks, "scales": scales}, h, DEV),
                            act=L.ACT_GPTOSS, limit=7.0)
    return experts, gu.astype(np.float64), d.astype(np.float64), rng


def _exact(x, ids, w, gu, d):
    """The layer in 64 bits, no value rounded."""
    out = np.zeros((x.shape[0], d.shape[1]))
    for t in range(x.shape[0]):
        for e, weight in zip(ids[t], w[t]):
            both = gu[e] @ x[t].astype(np.float64)
            g, u = np.minimum(both[0::2], 7.0), np.clip(both[1::2], -7.0, 7.0)
            out[t] += float(weight) * (d[e] @ ((u + 1.0) * g / (1.0 + np.exp(-1.702 * g))))
    return out


# a block's largest value meets a zero weight, so its others are all there is, `down` binades below it: with terms that drop bits
# there, the error shows in full.  The f16-expanding GEMM behind the separate calls holds an f16 activation exactly; both round
# the intermediate to f16, which is what their distance from 64 bits then is (2^-12 of each value, 1.5e-4 and more with the
# sums' signs; 1e-3 leaves room for sums that cancel).  `small`: the others are f16 values without a subnormal.
@pytest.mark.parametrize("down", [6, 14, 18, 20])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_small_values_beside_a_large_one_keep_their_bits(down, dtype):
    import engine_b200 as hq
    from engine_b200 import _lib as L
    t, e, k, h, i = 12, 4, 4, 256, 192
    experts, gu, d, rng = _layer_with_dead_columns(e, h, i, 7 + down)
    x = np.sign(rng.standard_normal((t, h))) * rng.uniform(1.0, 2.0, (t, h)) * 2.0 ** (7 - down)
    x[:, ::32] = 200.0
    xd = T.to_dev(x.astype(np.float32), dtype, DEV)
    logits = rng.standard_normal((t, e)).astype(np.float32)
    ids, w = M.router_topk(logits, k, L.SCORE_SOFTMAX, L.WEIGHT_SCORE, True)
    want = _exact(xd.float().cpu().numpy(), ids, w, gu, d)
    got = _run(experts, xd, logits, k)
    top = hq.moe_router_topk(T.to_dev(logits, torch.float32, DEV), hq.MoeRouterTopKConfig(k, L.SCORE_SOFTMAX, L.WEIGHT_SCORE, True))
    split = experts.forward(xd, top.values, top.indices, out_dtype=torch.float32).cpu().numpy()
    err, err_gemm = T.rel_l2(got, want), T.rel_l2(split, want)
    print(f"down {down} {dtype}: {err:.2e}, f16 GEMM {err_gemm:.2e}")
    assert err <= 1e-3 and err <= 1.1 * err_gemm
