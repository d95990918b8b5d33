"""Dispatch tables against a stable sort: one block and a cluster of eight, runs that end inside a group of 32, expert
counts at the edges of the scan, one crowded expert, skipped ids; and the weighted reduce over them."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

DEV = "cuda:0"


@pytest.mark.parametrize("e", [1, 127, 1024, 1025, 4096])
@pytest.mark.parametrize("t,k", [(1, 1), (5, 7), (512, 8), (4097, 1), (4099, 3)])
def test_tables_match_a_stable_sort(t, k, e):
    from engine_b200.quant import moe_dispatch_build
    g = torch.Generator(device=DEV).manual_seed(t + e)
    ids = torch.randint(0, e, (t, k), generator=g, device=DEV)
    ids[torch.rand((t, k), generator=g, device=DEV) < 0.4] = e // 2
    ids[torch.rand((t, k), generator=g, device=DEV) < 0.1] = -1
    tab = moe_dispatch_build(ids.to(torch.int32), e)
    flat = ids.flatten()
    order = torch.argsort(torch.where(flat < 0, e, flat), stable=True)[:int((flat >= 0).sum())]
    counts = torch.bincount(flat[flat >= 0], minlength=e)
    n = len(order)
    assert torch.equal(tab.expert_bounds.long(), torch.cat([torch.zeros(1, device=DEV, dtype=torch.long), counts.cumsum(0)]))
    assert torch.equal(tab.sorted_assign[:n].long(), order)
    assert torch.equal(tab.sorted_token[:n].long(), order // k)
    inv = torch.full((t * k,), -1, device=DEV, dtype=torch.long)
    inv[order] = torch.arange(n, device=DEV)
    assert torch.equal(tab.inv_perm.long().flatten(), inv)
    # work items of the decode kernels: 4 rows each with at most four tokens, else 8
    w = 4 if t <= 4 else 8
    ws = tab.workspace.view(torch.int32)
    n_items = int(((counts + w - 1) // w).sum())
    assert int(ws[0]) == n_items
    items = ws[4:4 + 2 * n_items].view(-1, 2).tolist()
    b = tab.expert_bounds.tolist()
    assert items == [[x, r] for x in range(e) for r in range(b[x], b[x + 1], w)]


@pytest.mark.parametrize("hidden", [8, 2048, 2056, 2884])
@pytest.mark.parametrize("k", [1, 4, 8, 9])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_weighted_reduce_slots_and_slabs(dt, k, hidden):
    # slots in flight eight (16-bit) or four (f32) at a time; rows in slabs of 2,048; 2,884 f32 is no multiple of eight
    import engine_b200 as hq
    if hidden % 8 and dt != torch.float32:
        pytest.skip("rows of y are whole 16-byte units")
    g = torch.Generator(device=DEV).manual_seed(k + hidden)
    t = 5
    y = torch.randn((t * k, hidden), generator=g, device=DEV).to(dt)
    w = torch.rand((t, k), generator=g, device=DEV)
    inv = torch.randperm(t * k, generator=g, device=DEV).to(torch.int32).reshape(t, k)
    if k > 1:
        inv[2, k - 1] = -1
    add = torch.randn((t, hidden), generator=g, device=DEV)
    got = hq.moe_weighted_reduce(y, w, torch.float32, inv, add)
    rows = torch.where(inv[..., None] >= 0, y.float()[inv.clamp(min=0).long()], 0.0)
    want = (w.double()[..., None] * rows.double()).sum(1) + add.double()
    assert float((got.double() - want).abs().max()) <= 1e-5
