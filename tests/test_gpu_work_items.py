"""Expert projections out of dispatch tables that a host carved from one scratch block without padding (the workspace then
starts at any 32-bit word), and tables built for [tokens, slots] used by a projection that calls its rows one-slot tokens."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from tests import hq_testlib as T

DEV = "cuda:0"


def _tables(ids, e, shift=0):
    """bounds | sorted_assign | sorted_token | inv_perm | workspace behind one another, `shift` words into a block."""
    from engine_b200 import _lib as L
    from engine_b200.quant import DispatchTables
    t, k = ids.shape
    ws = L.lib().hq_moe_dispatch_workspace_bytes(t, k, e) // 4
    sizes = [e + 1, t * k, t * k, t * k, ws]
    block = torch.full((shift + sum(sizes),), -1, dtype=torch.int32, device=DEV)
    parts, at = [], shift
    for n in sizes:
        parts.append(block[at:at + n])
        at += n
    L.check(L.lib().hq_moe_dispatch_build(C.c_void_p(ids.data_ptr()), t, k, e, *[C.c_void_p(p.data_ptr()) for p in parts], 4 * ws,
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream)), "hq_moe_dispatch_build")
    return DispatchTables(t, k, e, *parts)


def _bank(fmt, n, k, e):
    rng = T.rng_for(17, n)
    return T.make_layer(fmt, T.make_weight(fmt, rng, n, k, experts=e)[0], k, DEV), rng


# 1 x 8 of 128 experts puts the workspace at word 153; 3 x 8 at word 201; shift moves it to the other residues
@pytest.mark.parametrize("fmt", ["Q4_K", "Q8_0", "FP8", "Q6_K"])
@pytest.mark.parametrize("t,shift", [(1, 0), (3, 0), (3, 1), (12, 2), (12, 0), (40, 0)])
def test_a_workspace_at_any_word(fmt, t, shift):
    e, k, width = 128, 8, 512
    layer, rng = _bank(fmt, 256, width, e)
    ids = torch.from_numpy(np.stack([rng.permutation(e)[:k] for _ in range(t)]).astype(np.int32)).to(DEV)
    x = T.to_dev(rng.standard_normal((t, width)).astype(np.float32), torch.bfloat16, DEV)
    want = layer.gather_forward_raw(x, ids, torch.float32)
    got = layer.gather_forward_raw(x, ids, torch.float32, tables=_tables(ids, e, shift))
    assert torch.equal(got, want) and layer.device_status()[0] == 0


@pytest.mark.parametrize("fmt", ["Q4_K", "FP8", "Q6_K"])
@pytest.mark.parametrize("t", [1, 4, 5])
def test_slots_as_tokens(fmt, t):
    from engine_b200 import _lib as L
    e, k, width, n = 64, 8, 512, 256
    layer, rng = _bank(fmt, n, width, e)
    ids = torch.from_numpy(np.stack([rng.permutation(e)[:k] for _ in range(t)]).astype(np.int32)).to(DEV)
    x = T.to_dev(rng.standard_normal((t, k, width)).astype(np.float32), torch.bfloat16, DEV)
    tab = _tables(ids, e)
    want = layer.gather_forward_raw(x, ids, torch.float32, tables=tab).view(t * k, n)
    got = torch.empty((t * k, n), dtype=torch.float32, device=DEV)
    w = layer._weight_struct()
    p = lambda a: C.c_void_p(a.data_ptr())
    L.check(L.lib().hq_moe_gather_forward(C.byref(w), None, None, p(x), L.DT_BF16, L.ROWS_PER_SLOT, t * k, 1, p(tab.expert_bounds),
                                          p(tab.sorted_assign), p(tab.sorted_token), p(tab.workspace), p(got), L.DT_F32,
                                          L.ROWS_PER_SLOT, p(layer._status_buf(got.device)),
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream)), "hq_moe_gather_forward")
    assert layer.device_status()[0] == 0
    # (items of up to four rows and of up to eight may add their f32 sums in another order)
    assert T.rel_l2(got.cpu().numpy(), want.cpu().numpy()) <= 1e-5
