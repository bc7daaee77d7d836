"""Attention of prompts with two heads a block and 128 keys a step, against float64 and the warp-level kernel: lengths on and off the tiles
of 128 queries and the steps of 128 keys (an odd number of pages among them), portions behind cached keys, windows."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("nh,nkv", [(4, 1), (6, 3)])
@pytest.mark.parametrize("new,start,window", [([128], [0], 0), ([129, 2, 700], [0, 300, 63], 0), ([64, 65, 1, 191], [0, 0, 64, 129], 0),
                                              ([130, 385], [500, 0], 100), ([700], [1000], 64), ([300], [10], 1)])
def test_two_heads_a_block(hd, nh, nkv, new, start, window):
    from ithaca_b200.csrc import attention_bf16, ops
    B, T = len(new), sum(new)
    g = torch.Generator(device=DEV).manual_seed(T + hd + nh)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
    lens = [a + b for a, b in zip(new, start)]
    cols, n_pages = max(-(-e // 64) for e in lens), sum(-(-e // 64) for e in lens) + 3
    order = torch.randperm(n_pages, generator=torch.Generator().manual_seed(1)).tolist()
    table = torch.full((B, cols), -1, dtype=torch.int32)
    for b, e in enumerate(lens):
        for i in range(-(-e // 64)):
            table[b, i] = order.pop()
    whole = table.clone().to(DEV)
    for b, first in enumerate(start):                              # pages behind the window may have been given back
        if window:
            table[b, :max(0, first + 1 - window) // 64] = -1
    table = table.to(DEV)
    k, v, q = rnd(n_pages, nkv, 64, hd), rnd(n_pages, nkv, 64, hd), rnd(T, nh * hd) * 1.5
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    cu = [sum(new[:i]) for i in range(B + 1)]
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    args = (k, v, i32(cu), i32(lens), table, B, max(new), nh, hd ** -0.5, window, status)
    got = attention_bf16.prefill(q, *args, kind="two_heads")
    one = attention_bf16.prefill(q, *args, kind="mma")
    assert status.item() == 0, ops.wait_records()
    for b, (n, e) in enumerate(zip(new, lens)):
        at = torch.arange(e, device=DEV)
        take = lambda x: x[whole[b, at // 64].long(), :, at % 64].double().repeat_interleave(nh // nkv, 1)
        s = torch.einsum("nha,mha->hnm", q[cu[b]:cu[b + 1]].view(n, nh, hd).double(), take(k)) * hd ** -0.5
        i, j = torch.arange(e - n, e, device=DEV)[:, None], at[None]
        seen = (j <= i) & ((j > i - window) if window else (j >= 0))
        want = torch.einsum("hnm,mhc->nhc", s.masked_fill(~seen, float("-inf")).softmax(-1), take(v)).reshape(n, -1)
        far = lambda x: float((x[cu[b]:cu[b + 1]].double() - want).norm() / want.norm())
        # weights and the result are rounded to 8 bits: 2^-9 relative at most each
        assert far(got) < 2 * 2 ** -9 and far(got) < 1.5 * far(one) + 1e-4, (b, far(got), far(one))


def test_two_heads_a_block_refuses_what_it_does_not_take():
    from ithaca_b200.csrc import attention_bf16, ops
    z = lambda *s: torch.zeros(s, dtype=torch.bfloat16, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    for nh, nkv, more in ((3, 1, {}), (4, 1, {"softcap": 3.0}), (4, 1, {"sink": True}), (4, 2, {"window": 70, "keep": 5})):
        window = more.pop("window", 0)
        with pytest.raises(ops.KernelError):
            attention_bf16.prefill(z(80, nh * 64), z(2, nkv, 64, 64), z(2, nkv, 64, 64), i32([0, 80]), i32([80]), i32([[0, 1]]), 1, 80, nh, 0.125, window,
                                   torch.zeros(1, dtype=torch.int32, device=DEV), kind="two_heads", **more)
