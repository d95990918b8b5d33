"""Row quantizers (FP8 1x128, MXFP8 1x32) on both sides of the rule for one or four loads a warp, for each input type, row
lookup, partial last spans and, for MXFP8, rows that cannot be read 16 bytes at a time: every code and scale as the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from oracle import formats as F
from tests import hq_testlib as T

DEV = "cuda:0"
SHAPES = [(1, 128), (9, 384), (66, 2432), (1185, 4224)]          # the last: 18,960 loads of 256, just above the rule's 18,944


def _rows(n, k, dt):
    rng = T.rng_for(12, n)
    x = torch.from_numpy(rng.standard_normal((max(n // 3, 1), k)).astype(np.float32))
    x *= torch.from_numpy(rng.choice([1e-30, 1e-4, 1.0, 500.0], (x.shape[0], 1)).astype(np.float32))
    x[0, :128] = 0.0
    x[-1, ::5] = -0.0
    x = x.to(getattr(torch, dt))
    rows = rng.integers(0, x.shape[0], n).astype(np.int32)
    return x, rows, x.to(torch.float32).numpy()[rows]


@pytest.mark.parametrize("dt", ["float32", "bfloat16", "float16"])
@pytest.mark.parametrize("n,k", SHAPES)
def test_fp8_rows(n, k, dt):
    import engine_b200 as hq
    x, rows, used = _rows(n, k, dt)
    codes, scales = hq.fp8_quantize_rows(x.to(DEV), torch.from_numpy(rows).to(DEV))
    want_c, want_s = F.fp8_vector_quant(used, 128)
    assert np.array_equal(scales.cpu().numpy().reshape(want_s.shape), want_s)
    assert np.array_equal(codes.cpu().numpy().reshape(want_c.shape), want_c)


@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("dt", ["float32", "bfloat16", "float16"])
@pytest.mark.parametrize("n,k", [(n, k + 32 * (n % 3)) for n, k in SHAPES])
def test_mxfp8_rows(n, k, dt, pad):
    import engine_b200 as hq
    x, rows, used = _rows(n, k, dt)
    xd = torch.empty(x.numel() + pad, dtype=x.dtype, device=DEV)[pad:].view(x.shape)      # pad: a base between 16-byte boundaries
    xd.copy_(x)
    codes, scales = hq.mxfp8_quantize_rows(xd, torch.from_numpy(rows).to(DEV))
    want_c, want_s = F.mxfp8_quant(used)
    assert np.array_equal(scales.cpu().numpy(), want_s)
    assert np.array_equal(codes.cpu().numpy(), want_c)
