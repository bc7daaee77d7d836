"""32-bit attention of prompts by blocks of 64 rows: bit for bit what the kernel with a token a block gives, over groups of heads, windows, tokens of
several sequences in a block, values that are not finite and missing pages; and which steps go this way."""
import pytest
import torch

DEV = "cuda:0"


def made(nh, nkv, hd, new, old, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    T, B, cols = sum(new), len(new), -(-max(a + b for a, b in zip(new, old)) // 64)
    k, v, q = rnd(B * cols + 1, nkv, 64, hd), rnd(B * cols + 1, nkv, 64, hd), rnd(T, nh * hd)
    table = torch.randperm(B * cols, generator=torch.Generator().manual_seed(seed)).view(B, cols).to(torch.int32).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    seq, pos = i32([i for i, n in enumerate(new) for _ in range(n)]), i32([o + j for n, o in zip(new, old) for j in range(n)])
    return q, k, v, seq, pos, table, nh, hd ** -0.5


@pytest.mark.gpu
@pytest.mark.parametrize("nh,nkv", [(4, 4), (6, 3), (6, 2), (8, 2), (12, 2), (16, 2), (16, 1)])
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("new,old", [([1], [0]), ([130], [0]), ([3, 1, 64, 65, 2], [0, 200, 63, 1, 127]), ([200], [300])])
@pytest.mark.parametrize("window", [0, 1, 70, 129])
def test_same_bits(nh, nkv, hd, new, old, window):
    from ithaca_b200.csrc import ops
    a = made(nh, nkv, hd, new, old, nh + hd)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    assert torch.equal(ops.attention_rows(*a, window, status), ops.attention_simt(*a, window, status)) and status.item() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("what", [float("inf"), float("nan")])
def test_values_that_are_not_finite(what):
    """A key's value reaches the tokens that see the key, and no others of its block."""
    from ithaca_b200.csrc import ops
    q, k, v, seq, pos, table, nh, scale = made(8, 2, 64, [150, 20], [0, 0], 1)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    v[table[0, 1].item(), 0, 10, 5] = what                                     # position 74 of the first sequence
    k[table[1, 0].item(), 1, 12, 7] = what                                     # position 12 of the second
    got, want = (f(q, k, v, seq, pos, table, nh, scale, 0, status) for f in (ops.attention_rows, ops.attention_simt))
    assert torch.equal(got.nan_to_num(7.0, 8.0, 9.0), want.nan_to_num(7.0, 8.0, 9.0)) and bool(torch.isfinite(got[:74]).all())
    assert not bool(torch.isfinite(got[74]).all()) and bool(torch.isfinite(got[150:162]).all())


@pytest.mark.gpu
def test_a_missing_page_is_reported():
    from ithaca_b200.csrc import ops
    q, k, v, seq, pos, table, nh, scale = made(8, 2, 64, [150], [0], 2)
    table[0, 1] = 1 << 20
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    got = ops.attention_rows(q, k, v, seq, pos, table, nh, scale, 0, status)
    assert status.item() != 0 and torch.equal(got, ops.attention_simt(q, k, v, seq, pos, table, nh, scale, 0, status))


@pytest.mark.gpu
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("new,old,window", [([200], [300], 100), ([65, 70], [500, 129], 64), ([3, 90], [640, 200], 129), ([130, 1, 40], [0, 300, 0], 70)])
def test_pages_behind_the_window_may_be_gone(hd, new, old, window):
    """A cache gives back the pages that lie wholly before the first key a window still reaches (their column of the table is -1): nothing is
    missed, and nothing of what the pool's first row holds instead gets into the result."""
    from ithaca_b200.csrc import ops
    q, k, v, seq, pos, table, nh, scale = made(8, 2, hd, new, old, 5)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    gone = 0
    for i, o in enumerate(old):
        n = max(0, o + 1 - window) // 64
        table[i, :n] = -1
        gone += n
    k[0, :, 0], v[0, :, 0] = float("nan"), float("nan")
    table[table == 0] = k.shape[0] - 1
    k[-1], v[-1] = 0.5, 0.25
    rows, simt = (f(q, k, v, seq, pos, table, nh, scale, window, status) for f in (ops.attention_rows, ops.attention_simt))
    assert gone > 0 and status.item() == 0 and torch.equal(rows, simt) and bool(torch.isfinite(rows).all())


# measured on B200: heads, kv heads, new tokens, tokens before them, window, us a token a block, us these
@pytest.mark.parametrize("nh,nkv,new,old,window,simt,rows", [
    (32, 8, [1], [0], 0, 4.5, 8.5), (32, 8, [20], [0], 0, 7.1, 11.5), (32, 8, [64], [0], 0, 13.9, 15.3), (32, 8, [300, 35, 130], [0] * 3, 0, 119, 60),
    (32, 8, [4] * 8, [50] * 8, 0, 12.8, 44.3), (32, 8, [16] * 8, [0] * 8, 0, 10.2, 11.5), (32, 8, [100] * 6, [30] * 6, 0, 95, 48), (32, 8, [700], [0], 100, 154, 66),
    (32, 8, [40], [2000], 0, 302, 215), (16, 16, [16] * 8, [0] * 8, 0, 8.2, 34.5), (16, 16, [100] * 6, [30] * 6, 0, 91, 54), (40, 40, [4] * 8, [50] * 8, 0, 18.6, 131)])
def test_steps_take_the_faster_way(nh, nkv, new, old, window, simt, rows):
    from ithaca_b200.csrc import ops
    assert ops.attention_rows_pay(new, [a + b for a, b in zip(new, old)], nh, nkv, window) == (rows < simt)
