"""The selective scan of a prompt in pieces, against the token-by-token kernel and float64: sequences of several pieces, of one, of
none, with and without an earlier state, lengths on and off the edges of pieces and tiles."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("inner,N", [(40, 5), (96, 16), (33, 20), (64, 64), (4096, 16)])
@pytest.mark.parametrize("new,start", [([640], [0]), ([3, 0, 257, 192, 64, 65], [5, 0, 0, 12, 0, 1]), ([1, 1025, 2], [4, 7, 0])])
def test_scan_in_pieces(inner, N, new, start):
    from ithaca_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(inner + N)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    T, B, R = sum(new), len(new), 3
    u, dt, bc, z = rnd(T, inner).to(torch.bfloat16), rnd(T, inner) - 2.0, rnd(T, R + 2 * N), rnd(T, 2 * inner)
    A, D, bias = -torch.exp(rnd(inner, N) * 0.5), rnd(inner), rnd(inner) * 0.3
    before = rnd(B + 1, 2, inner, N)
    cu = [sum(new[:i]) for i in range(B + 1)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    slots = list(range(B, 0, -1))
    ends = [a + b for a, b in zip(new, start)]
    made = []
    for longest in (max(new), 0):
        state = before.clone()
        ctx = SimpleNamespace(n_seqs=B, max_new=longest, slots=i32(slots), cu_seqlens=i32(cu), kv_lens=i32(ends), is_decode=False)
        need = ops.lib().ik_selective_scan_scratch(1, T, B, longest, inner, N, 0)
        assert (need > 0) == (longest > 0)
        made.append((ops.selective_scan(u, dt, bias, A, bc, R, R + N, D, z[:, inner:], state, ctx, torch.bfloat16), state))
    (y, state), (y1, state1) = made
    far = lambda a, b: float((a.double() - b.double()).norm() / b.double().norm())
    off, off1 = [], []
    for b in range(B):
        S = before[slots[b], (start[b] - 1) & 1].double() if start[b] > 0 else torch.zeros(inner, N, dtype=torch.float64, device=DEV)
        rows = []
        for t in range(cu[b], cu[b + 1]):
            d = torch.nn.functional.softplus(dt[t].double() + bias.double())
            S = torch.exp(d[:, None] * A.double()) * S + (d * u[t].double())[:, None] * bc[t, R:R + N].double()
            rows.append((S @ bc[t, R + N:].double() + D.double() * u[t].double()) * torch.nn.functional.silu(z[t, inner:].double()))
        if not rows:
            assert torch.equal(state[slots[b]], before[slots[b]])
            continue
        p = (ends[b] - 1) & 1
        off.append(far(state[slots[b], p], S))
        off1.append(far(state1[slots[b], p], S))
        assert far(y[cu[b]:cu[b + 1]], torch.stack(rows)) < 4e-3           # one rounding to 8 bits: 2^-9 at most, 1.7e-3 on average
        if start[b] % 2 == ends[b] % 2:
            continue
        assert torch.equal(state[slots[b], 1 - p], before[slots[b], 1 - p])   # the other parity is left alone
    # the hardware's exponential: some units in the last place; the pieces add roundings of a sum of step sizes, no more
    assert max(off) < 3e-6 and max(off) < 2 * max(off1) + 2e-7, (off, off1)
    assert torch.equal(state[0], before[0])
