"""Which prompts run two heads a block: by the tiles of queries that exist and the keys they see, against measured times (without a device);
and that an attention layer takes the kernel the rule names, with the results of the other (on a device)."""
from types import SimpleNamespace

import pytest
import torch


def lengths(text):
    return [int(n) for part in text.split("+") for n in [part.split("x")[1]] * int(part.split("x")[0])]


# measured on B200: head size, heads, new tokens, tokens before them, window, us with one head a block, us with two
MEASURED = [(64, 32, "12x100", 0, 0, 17, 20), (64, 32, "24x100", 0, 0, 25, 29), (64, 32, "128x30", 0, 0, 79, 124), (64, 32, "16x250", 0, 0, 35, 41),
            (64, 32, "8x1000", 0, 0, 98, 105), (64, 32, "1x2048", 0, 0, 49, 42), (64, 32, "1x4096", 0, 0, 134, 121), (64, 32, "1x512", 3000, 0, 51, 57),
            (64, 32, "1x1000+1x300+1x2000+1x50+1x700+1x1500", 0, 0, 112, 92), (64, 32, "1x4096", 0, 128, 45, 56), (64, 32, "1x2048+63x1", 500, 0, 331, 245),
            (128, 32, "12x100", 0, 0, 19, 22), (128, 32, "24x100", 0, 0, 28, 33), (128, 32, "64x100", 0, 0, 68, 82), (128, 32, "64x130", 0, 0, 124, 168),
            (128, 32, "16x300", 0, 0, 60, 75), (128, 32, "8x1000", 0, 0, 114, 128), (128, 32, "1x1024", 0, 0, 23, 27), (128, 32, "1x2048", 0, 0, 52, 49),
            (128, 32, "1x4096", 0, 64, 45, 63), (128, 32, "1x4096", 0, 512, 71, 84), (128, 32, "32x128", 2000, 0, 158, 178),
            (128, 32, "1x1900+1x1200+1x800+1x400+1x200", 0, 0, 111, 100), (128, 16, "1x1024", 0, 0, 21, 25), (128, 16, "1x2048", 0, 0, 36, 41),
            (128, 16, "1x4096", 0, 0, 85, 73), (128, 64, "8x1000", 0, 0, 216, 250), (128, 64, "3x2048", 0, 100, 140, 169)]


@pytest.mark.parametrize("hd,heads,step,before,window,one,two", MEASURED)
def test_prompts_take_the_faster_way(hd, heads, step, before, window, one, two):
    from ithaca_b200.csrc.attention_bf16 import two_heads_pay
    new = lengths(step)
    assert two_heads_pay(new, [n + before for n in new], heads, hd, window, 148) == (two < one)


def test_a_step_without_tokens():
    from ithaca_b200.csrc.attention_bf16 import two_heads_pay
    assert not two_heads_pay([], [], 32, 128, 0, 148)


@pytest.mark.gpu
@pytest.mark.parametrize("new,nh,nkv,options", [([4096], 32, 8, {}), ([100] * 24, 32, 8, {}), ([4096], 32, 32, {}), ([4096], 32, 8, {"softcap": 20.0}),
                                                ([4096], 32, 8, {"sink": True})])
def test_layers_take_the_kernel_of_the_rule(new, nh, nkv, options, monkeypatch):
    from ithaca_b200.csrc import attention_bf16 as A, ops
    dev, hd, B = "cuda:0", 64, len(new)
    g = torch.Generator(device=dev).manual_seed(1)
    rnd = lambda *s: torch.randn(s, generator=g, device=dev).to(torch.bfloat16)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    cols = max(-(-n // 64) for n in new)
    table = torch.arange(cols * B, dtype=torch.int32, device=dev).view(B, cols)
    q, k, v = rnd(sum(new), nh * hd), rnd(cols * B, nkv, 64, hd), rnd(cols * B, nkv, 64, hd)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    ctx = SimpleNamespace(n_seqs=B, max_new=max(new), cu_seqlens=i32([sum(new[:i]) for i in range(B + 1)]), kv_lens=i32(new), host_n_new=new, host_kv_lens=new,
                          is_decode=False, shared={})
    got = A.attend(q, k, v, ctx, table, nh, hd ** -0.5, 0, status, **options)
    takes = not options and nh != nkv and A.two_heads_pay(new, new, nh, hd, 0, ops.sm_count())
    assert takes == (new == [4096] and nkv == 8 and not options)
    args = (q, k, v, ctx.cu_seqlens, ctx.kv_lens, table, B, max(new), nh, hd ** -0.5, 0, status)
    assert torch.equal(got, A.prefill(*args, kind="two_heads" if takes else "tc", **options))
    assert status.item() == 0
