"""What is not finite in attention of prompts shows where it belongs: in its query's row, and behind its key; with two heads a block exactly where
it does with one, and over formed latent keys behind the tile that first sees it."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)


def rnd(seed, *shape):
    return torch.randn(shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV).to(torch.bfloat16)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("where,value", [("q", "nan"), ("q", "inf"), ("k", "nan"), ("v", "inf"), ("v", "nan")])
def test_two_heads_show_what_one_head_shows(hd, where, value):
    from ithaca_b200.csrc import attention_bf16
    nh, nkv, T, at = 4, 2, 450, 200
    table = torch.randperm(8, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(1, 8).to(DEV)
    q, k, v = rnd(1, T, nh * hd), rnd(2, 8, nkv, 64, hd), rnd(3, 8, nkv, 64, hd)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    run = lambda kind: attention_bf16.prefill(q, k, v, i32([0, T]), i32([T]), table, 1, T, nh, hd ** -0.5, 0, status, kind=kind).view(T, nh, hd)
    clean = run("two_heads")
    if where == "q":
        q[at, hd + 3] = float(value)                              # of head 1
    else:
        (k if where == "k" else v)[table[0, at // 64].long(), 1, at % 64, 5] = float(value)
    two, one = run("two_heads"), run("tc")
    assert torch.equal(torch.isfinite(two), torch.isfinite(one)) and status.item() == 0
    if where == "q":
        assert not bool(torch.isfinite(two[at, 1]).all())
        two[at, 1] = clean[at, 1]
        assert torch.equal(two, clean)
    else:
        assert torch.equal(two[:128], clean[:128]) and torch.equal(two[:, :2], clean[:, :2])          # tiles before it, the other kv head's heads
        assert not bool(torch.isfinite(two[at:, 2:]).all(-1).any())


@pytest.mark.parametrize("where", ["q", "turning q", "latent", "turning key"])
def test_formed_keys(where):
    from ithaca_b200.csrc import attention_latent
    H, rank, T, at = 3, 128, 600, 300
    table = torch.randperm(10, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(1, 10).to(DEV)
    rows, w = rnd(4, 10, 1, 64, rank + 64), (rnd(5, 2 * H * 128, rank).float() * rank ** -0.5).to(torch.bfloat16)
    q_plain, q_full = rnd(6, T, H * 128), rnd(7, T, H * (rank + 64))
    ctx = SimpleNamespace(n_seqs=1, max_new=T, max_kv_len=T, kv_lens=i32([T]), cu_seqlens=i32([0, T]), host_kv_lens=[T], host_n_new=[T])
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    run = lambda: attention_latent.prompt(q_plain, q_full, rows, w, ctx, table, H, rank, 0.07, 0, status).view(T, H, 128)
    clean = run()
    nan = float("nan")
    if where == "q":
        q_plain[at, 128 + 7] = nan
    elif where == "turning q":
        q_full[at, (rank + 64) + rank + 1] = nan
    else:
        rows[table[0, at // 64].long(), 0, at % 64, 3 if where == "latent" else rank + 3] = nan
    got = run()
    assert status.item() == 0
    if "q" in where:
        assert not bool(torch.isfinite(got[at, 1]).any())
        got[at, 1] = clean[at, 1]
        assert torch.equal(got, clean)
    else:
        assert torch.equal(got[:256], clean[:256])
        assert not bool(torch.isfinite(got[at:]).any())
