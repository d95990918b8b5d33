"""Dispatch tables against a stable sort: one block and a cluster of eight, runs that end inside a group of 32, expert
counts at the edges of the scan, one crowded expert, skipped ids; and the one-launch router of few tokens."""
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
