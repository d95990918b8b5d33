"""Gated FP8 expert GEMM, the end of an item: gate / (1 + exp(-gate)) * up, its f16 rounding and the 1x128 quantizer, for
every f16 gate value (subnormal ones too).  Weights and inputs are chosen so that every sum is exact; the down projection is
the identity, so the output is code x scale and has to be that of the same steps in torch with IEEE divisions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from oracle import formats as F
from tests import hq_testlib as T

DEV = "cuda:0"
N = 1024                    # a feature per f16 fraction


def _bank(codes):
    s = np.ones((1, codes.shape[0] // 128, codes.shape[1] // 128), np.float32)
    return {"weight": F.e4m3_encode(codes.astype(np.float32))[None], "scale": s}


@pytest.mark.parametrize("limit,alpha", [(None, None), (7.0, None), (7.0, 1.702)])
def test_every_gate_value(limit, alpha):
    import engine_b200 as hq
    from engine_b200 import _lib as L
    # a feature's fraction in 2^-10: 1024 + f = 128 * hi + 8 * mid + lo, each exact in e4m3
    f = np.arange(N) + 1024
    wg = np.zeros((N, 1024), np.float32)
    wg[:, 0], wg[:, 1], wg[:, 2] = f // 128, f // 8 % 16, f % 8
    up = np.array([1.0, -0.875, 0.0625, -1.0, 0.0, 0.5])[np.arange(N) % 6].astype(np.float32)
    wu = np.zeros((N, 1024), np.float32)
    wu[:, 128] = up
    # tokens: +- 2^p.  Column 3 (no weights) fixes the block's scale at 2^(p - 10), so that the codes are those of 128, 8, 1
    p = np.repeat(np.arange(-25, 16), 2)
    sign = np.where(np.arange(p.size) % 2 == 0, 1.0, -1.0)
    x = np.zeros((p.size, 1024), np.float32)
    unit = np.ldexp(1.0, p - 10)
    for col, c in ((0, 128.0), (1, 8.0), (2, 1.0)):
        x[:, col] = sign * c * unit
    x[:, 3] = 448.0 * unit
    x[:, 128], x[:, 129] = 1.0, 448.0
    act = {} if limit is None else {"limit": limit}
    if alpha is not None:
        act.update(act=L.ACT_GPTOSS, alpha=alpha)
    experts = hq.MoEExperts(T.make_layer("FP8", _bank(np.eye(N)), N, DEV), T.make_layer("FP8", _bank(wg), 1024, DEV),
                            T.make_layer("FP8", _bank(wu), 1024, DEV), **act)
    got = experts.forward_fp8_dense(T.to_dev(x, torch.float32, DEV), out_dtype=torch.float32)
    torch.cuda.synchronize()
    assert experts.gate.device_status()[0] == 0
    half = lambda a: a.to(torch.float16).to(torch.float32)
    g = half(torch.from_numpy((sign * np.ldexp(1.0, p - 10))[:, None] * f[None, :]).to(DEV).to(torch.float32))
    u = half(torch.from_numpy(np.broadcast_to(up, g.shape).copy()).to(DEV))
    if limit is not None:
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    h = (u + 1.0) * (g / (1.0 + torch.exp(-float(np.float32(alpha)) * g))) if alpha is not None else g / (1.0 + torch.exp(-g)) * u
    codes, scale = F.fp8_vector_quant(half(h).cpu().numpy(), 128)
    assert np.array_equal(got.cpu().numpy(), F.fp8_vector_dequant(codes, scale, 128))
