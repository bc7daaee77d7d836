"""Gathering tokens into expert order and adding experts' results up: rows on and off the blocks of four, columns on and off the
blocks' width, few and many tokens (the two ways of cutting the sum), every optional operand; bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T,top,d", [(5, 2, 64), (295, 3, 1028), (296, 1, 8), (700, 5, 2048), (1000, 4, 260), (400, 2, 6)])
def test_sums_of_experts_rows(T, top, d):
    from ithaca_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(T + d)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    rows = T * top + 7
    parts, weight, extra, ew, base = rnd(rows, d), rnd(T, top), rnd(T, d), rnd(T), rnd(T, d)
    row_of = torch.randperm(rows, generator=torch.Generator().manual_seed(1))[:T * top].to(torch.int32).to(DEV)
    for unweighted in (False, True):
        for ex, w in ((None, None), (extra, None), (extra, ew)):
            want = torch.zeros(T, d, device=DEV, dtype=torch.float64)
            for k in range(top):                                  # a fused multiply-add rounds once: exact in float64, then to float32
                row = parts[row_of.view(T, top)[:, k].long()].double()
                want = (want + row * (1.0 if unweighted else weight[:, k, None].double())).float().double()
            if ex is not None:
                want = (want + ex.double() * (1.0 if w is None else w[:, None].double())).float().double()
            got = ops.moe_combine(parts, weight, row_of=row_of, unweighted=unweighted, extra=ex, extra_weight=w)
            assert torch.equal(got, want.float())
            into = ops.moe_combine(parts, weight, out=base.clone(), row_of=row_of, unweighted=unweighted, extra=ex, extra_weight=w, accumulate=True)
            assert torch.equal(into, base + got)
    assert torch.equal(ops.moe_combine(parts[:T * top].contiguous(), weight), ops.moe_combine(parts, weight, row_of=torch.arange(T * top, dtype=torch.int32, device=DEV)))


@pytest.mark.parametrize("T,top,E,bn,d", [(3, 2, 4, 16, 8), (1000, 4, 7, 128, 520), (4099, 5, 32, 128, 64), (2049, 1, 3, 256, 2056)])
def test_tokens_in_expert_order(T, top, E, bn, d):
    from ithaca_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(T)
    chosen = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(i % 97))[:top] for i in range(T)]).to(torch.int32).to(DEV)
    x = torch.randn(T, d, generator=g, device=DEV).to(torch.bfloat16)
    plan = ops.moe_sort_padded(chosen, E, bn)
    xp = ops.moe_gather(x, plan)
    row_of = plan.row_of.view(-1).long()
    assert row_of.unique().numel() == T * top                          # every assignment has a row of its own
    assert torch.equal(xp[row_of], x.repeat_interleave(top, 0))
    assert torch.equal(plan.tile_group.long()[row_of // bn], chosen.view(-1).long())
    rest = torch.ones(xp.shape[0], dtype=torch.bool, device=DEV)
    rest[row_of] = False
    assert float(xp[rest].abs().sum()) == 0


def test_narrow_rows_cost_what_their_bytes_do():
    """Rows of 64 against as many bytes in rows of 512: blocks of one row, or four, whatever their width took four to five times as long."""
    from ithaca_b200.csrc import ops

    def us(call):
        graph = torch.cuda.CUDAGraph()
        call()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            for _ in range(20):
                call()
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b) * 50)
        return min(times)

    gather, combine = [], []
    for T, d in ((16384, 64), (2048, 512)):
        chosen = torch.stack([torch.randperm(8, generator=torch.Generator().manual_seed(i))[:2] for i in range(T)]).to(torch.int32).to(DEV)
        plan = ops.moe_sort_padded(chosen, 8, 128)
        x, parts = torch.ones(T, d, dtype=torch.bfloat16, device=DEV), torch.ones(plan.rows, d, device=DEV)
        weight, out = torch.ones(T, 2, device=DEV), torch.empty(T, d, device=DEV)
        gather.append(us(lambda: ops.moe_gather(x, plan)))
        combine.append(us(lambda: ops.moe_combine(parts, weight, out=out, row_of=plan.row_of)))
    assert gather[0] < 2.5 * gather[1] and combine[0] < 2.5 * combine[1], (gather, combine)
