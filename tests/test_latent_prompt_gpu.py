"""Latent attention of prompts over keys and values formed per head, against float64: one and several sequences, portions behind
cached rows, windows, lengths on and off the tiles of 128 and 256 queries and 64 keys, with and without a turning part."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rope", [64, 0])
@pytest.mark.parametrize("new,start,window", [([256], [0], 0), ([257, 1, 640], [0, 300, 63], 0), ([129, 385], [500, 0], 100), ([700], [1000], 64), ([300], [10], 1),
                                              ([1, 63, 64, 65], [0, 1, 64, 200], 0)])
def test_attention_over_formed_keys(rope, new, start, window):
    from ithaca_b200.csrc import attention_latent, ops
    H, rank, B, T = 3, 128, len(new), sum(new)
    hd = rank + rope
    g = torch.Generator(device=DEV).manual_seed(T + rope)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
    lens = [a + b for a, b in zip(new, start)]
    cols = max(-(-e // 64) for e in lens)
    n_pages = sum(-(-e // 64) for e in lens) + 3
    order = torch.randperm(n_pages, generator=torch.Generator().manual_seed(1)).tolist()
    table = torch.full((B, cols), -1, dtype=torch.int32)
    for b, e in enumerate(lens):
        for i in range(-(-e // 64)):
            table[b, i] = order.pop()
    rows, whole = rnd(n_pages, 1, 64, hd), table.clone().to(DEV)
    for b, first in enumerate(start):                              # pages behind the window may have been given back
        if window:
            table[b, :max(0, first + 1 - window) // 64] = -1
    table = table.to(DEV)
    q_plain, q_full, w = rnd(T, H * 128), rnd(T, H * hd) * 1.5, (rnd(2 * H * 128, rank).float() * rank ** -0.5).to(torch.bfloat16)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    cu = [sum(new[:i]) for i in range(B + 1)]
    ctx = SimpleNamespace(n_seqs=B, max_new=max(new), max_kv_len=max(lens), kv_lens=i32(lens), cu_seqlens=i32(cu), host_kv_lens=lens, host_n_new=new)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scale = (128 + rope) ** -0.5
    got = attention_latent.prompt(q_plain, q_full, rows, w, ctx, table, H, rank, scale, window, status)
    again = attention_latent.prompt(q_plain, q_full, rows, w, ctx, table, H, rank, scale, window, status)
    assert status.item() == 0, ops.wait_records()
    assert torch.equal(got, again)
    for b, (n, e) in enumerate(zip(new, lens)):
        at = torch.arange(e, device=DEV)
        x = rows[whole[b, at // 64].long(), 0, at % 64].double()
        kv = (x[:, :rank] @ w.double().T).view(e, 2, H, 128)
        k = torch.cat((kv[:, 0], x[:, None, rank:].expand(-1, H, -1)), -1)
        q = torch.cat((q_plain[cu[b]:cu[b + 1]].view(n, H, 128), q_full[cu[b]:cu[b + 1]].view(n, H, hd)[:, :, rank:]), -1).double()
        s = torch.einsum("nha,mha->hnm", q, k) * scale
        i, j = torch.arange(e - n, e, device=DEV)[:, None], at[None]
        seen = (j <= i) & ((j > i - window) if window else (j >= 0))
        want = torch.einsum("hnm,mhc->nhc", s.masked_fill(~seen, float("-inf")).softmax(-1), kv[:, 1]).reshape(n, -1)
        part = got[cu[b]:cu[b + 1]].double()
        # keys, values, weights and the result are rounded to 8 bits each: 2^-9 relative at most, four of them
        assert float((part - want).norm() / want.norm()) < 4 * 2 ** -9, (b, float((part - want).norm() / want.norm()))


def test_a_missing_page_is_reported():
    from ithaca_b200.csrc import attention_latent
    H, rank, n = 2, 64, 130
    rows, w = torch.ones(4, 1, 64, 128, dtype=torch.bfloat16, device=DEV), torch.ones(2 * H * 128, rank, dtype=torch.bfloat16, device=DEV)
    table = torch.tensor([[1, -1, 9]], dtype=torch.int32, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    ctx = SimpleNamespace(n_seqs=1, max_new=n, max_kv_len=n, kv_lens=i32([n]), cu_seqlens=i32([0, n]), host_kv_lens=[n], host_n_new=[n])
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    q = torch.ones(n, H * 128, dtype=torch.bfloat16, device=DEV)
    attention_latent.prompt(q, q, rows, w, ctx, table, H, rank, 0.1, 0, status)
    assert status.item() == 1 << 2


def test_which_steps_form_keys():
    from ithaca_b200.csrc import attention_latent as a
    rows = torch.empty(4, 1, 64, 576, dtype=torch.bfloat16, device=DEV)
    ctx = lambda new, lens, decode=False: SimpleNamespace(is_decode=decode, n_seqs=len(new), host_n_new=new, host_kv_lens=lens)
    takes = lambda c, dk=128, dr=64, dv=128, dt=torch.bfloat16: a.forms_keys(c, rows, dt, dk, dr, dv, 512)
    assert takes(ctx([4096], [4096])) and takes(ctx([2048, 1], [4096, 200]))
    assert takes(ctx([64], [64])) and not takes(ctx([63], [63])) and not takes(ctx([1, 1], [900, 900], True)) and not takes(ctx([300, 1], [300, 60000]))
    assert not takes(ctx([4096], [4096]), dk=64) and not takes(ctx([4096], [4096]), dr=32) and not takes(ctx([4096], [4096]), dt=torch.float32)
    assert not takes(ctx([200000], [200000]))
    assert not a.forms_keys(ctx([300], [60000]), rows, torch.bfloat16, 128, 64, 128, 512, 1024)       # a window: most keys would be formed for nothing
    assert a.forms_keys(ctx([4096], [4096]), rows, torch.bfloat16, 128, 64, 128, 512, 1024)
