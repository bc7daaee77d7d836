"""The order of experts' rows in whole tiles, by one block and by a cluster of eight: every assignment has a row of its own among its expert's, rows between belong to
nobody, tiles follow the experts, at the numbers of assignments and experts where the kernel changes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("E,top", [(1, 1), (8, 2), (33, 3), (63, 1), (64, 8), (300, 4)])
@pytest.mark.parametrize("assignments", [1, 31, 700, 2047, 2064, 4096, 4104, 9000, 40000])
@pytest.mark.parametrize("bn,skewed", [(16, False), (128, True), (256, False)])
def test_order(E, top, assignments, bn, skewed):
    from ithaca_b200.csrc import ops
    T = max(1, assignments // top)
    g = torch.Generator(device=DEV).manual_seed(E + T)
    chosen = torch.randint(0, E, (T, top), generator=g, device=DEV, dtype=torch.int32)
    if skewed:
        chosen = torch.where(torch.rand((T, top), generator=g, device=DEV) < 0.8, torch.full_like(chosen, E // 2), chosen)
    plan = ops.moe_sort_padded(chosen, E, bn)
    row, group, src = plan.row_of.long().view(-1), plan.tile_group.long(), plan.src_token.long()
    flat = chosen.long().view(-1)
    counts = torch.bincount(flat, minlength=E)
    tiles = (counts + bn - 1) // bn
    assert torch.equal(group[:int(tiles.sum())], torch.repeat_interleave(torch.arange(E, device=DEV), tiles)) and bool((group[int(tiles.sum()):] == -1).all())
    first = (tiles.cumsum(0) - tiles) * bn
    assert bool(((row >= first[flat]) & (row < first[flat] + counts[flat])).all()) and len(row.unique()) == T * top
    want = torch.full_like(src, -1)
    want[row] = torch.arange(T * top, device=DEV) // top
    assert torch.equal(src, want)
    assert torch.equal(plan.src_assign.long()[row], torch.arange(T * top, device=DEV))


@pytest.mark.parametrize("E,top", [(5, 2), (64, 4)])
@pytest.mark.parametrize("assignments", [700, 2048, 2064, 4096, 4104, 9000])
def test_numbers_of_no_expert(E, top, assignments):
    """Assignments to -1 or to E are in nobody's rows and change nobody else's."""
    from ithaca_b200.csrc import ops
    T, bn = assignments // top, 32
    g = torch.Generator(device=DEV).manual_seed(assignments)
    chosen = torch.randint(-1, E + 1, (T, top), generator=g, device=DEV, dtype=torch.int32)
    plan = ops.moe_sort_padded(chosen, E, bn)
    flat, row, src = chosen.long().view(-1), plan.row_of.long().view(-1), plan.src_token.long()
    valid = (flat >= 0) & (flat < E)
    counts = torch.bincount(flat[valid], minlength=E)
    tiles = (counts + bn - 1) // bn
    n, first = int(tiles.sum()), (tiles.cumsum(0) - tiles) * bn
    assert torch.equal(plan.tile_group.long()[:n], torch.repeat_interleave(torch.arange(E, device=DEV), tiles)) and bool((plan.tile_group[n:] == -1).all())
    at = row[valid]
    assert bool(((at >= first[flat[valid]]) & (at < first[flat[valid]] + counts[flat[valid]])).all()) and len(at.unique()) == len(at)
    which = torch.arange(T * top, device=DEV)[valid]
    want = torch.full_like(src, -1)
    want[at] = which // top
    assert torch.equal(src, want) and torch.equal(plan.src_assign.long()[at], which) and bool((row[~valid] == 0).all())
