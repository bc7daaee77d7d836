"""Formed keys and values of latent attention stay within their bytes whatever the heads (without a device), sequences taking turns where a
step's are more (on a device, bit for bit)."""
from types import SimpleNamespace

import pytest
import torch


def takes(new, lens, heads, rank=512, scale=0.1):
    from ithaca_b200.csrc import attention_latent as a
    rows = torch.empty(1, 1, 64, rank + 64, dtype=torch.bfloat16)
    ctx = SimpleNamespace(is_decode=False, n_seqs=len(new), host_n_new=new, host_kv_lens=lens)
    return a.forms_keys(ctx, rows, torch.bfloat16, 128, 64, 128, rank, 0, heads, scale)


def test_what_is_formed_is_bounded_in_bytes():
    from ithaca_b200.csrc import attention_latent as a
    for heads in (16, 32, 64, 128):
        keys = a.PROMPT_BYTES_MOST // (2 * (512 + 256 * heads)) // 64 * 64
        assert a.formed_bytes(keys, heads, 512) <= a.PROMPT_BYTES_MOST < a.formed_bytes(keys + 1, heads, 512)
        assert takes([4096], [keys], heads) and not takes([4096], [keys + 1], heads)
        assert takes([4096] * 3, [keys] * 3, heads) and not takes([4096] * 2, [100, keys + 64], heads)
    assert not takes([20000], [20000], 128) and takes([20000], [20000], 64)


def test_a_scale_that_is_not_positive_goes_over_the_rows():
    assert not takes([4096], [4096], 16, scale=0.0) and not takes([4096], [4096], 16, scale=-1.0)


def test_a_small_rank_wants_more_queries():
    assert takes([64] * 16, [564] * 16, 32, rank=128) and not takes([64] * 16, [564] * 16, 32, rank=64) and takes([512], [2512], 32, rank=64)


@pytest.mark.gpu
@pytest.mark.parametrize("window", [0, 100])
def test_sequences_take_turns(window, monkeypatch):
    from ithaca_b200.csrc import attention_latent as a
    dev, H, rank = "cuda:0", 3, 128
    new, start = [130, 1, 257, 64], [70, 300, 0, 129]
    lens, hd = [n + s for n, s in zip(new, start)], rank + 64
    g = torch.Generator(device=dev).manual_seed(7)
    rnd = lambda *s: torch.randn(s, generator=g, device=dev).to(torch.bfloat16)
    cols, T = max(-(-e // 64) for e in lens), sum(new)
    table = torch.randperm(4 * cols, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(4, cols).to(dev)
    rows, w = rnd(4 * cols, 1, 64, hd), (rnd(2 * H * 128, rank).float() * rank ** -0.5).to(torch.bfloat16)
    q_plain, q_full = rnd(T, H * 128), rnd(T, H * hd)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    ctx = SimpleNamespace(n_seqs=4, max_new=max(new), max_kv_len=max(lens), kv_lens=i32(lens), cu_seqlens=i32([sum(new[:i]) for i in range(5)]),
                          host_kv_lens=lens, host_n_new=new)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    made = []
    for most in (1 << 30, a.formed_bytes(max(lens), H, rank), a.formed_bytes(lens[0], H, rank) + a.formed_bytes(lens[1], H, rank)):
        monkeypatch.setattr(a, "PROMPT_BYTES_MOST", most)
        made.append(a.prompt(q_plain, q_full, rows, w, ctx, table, H, rank, 0.07, window, status))
    assert status.item() == 0
    assert torch.equal(made[0], made[1]) and torch.equal(made[0], made[2])
