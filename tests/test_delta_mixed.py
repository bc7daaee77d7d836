"""Steps that mix long and short sequences through the gated delta rule: which of them go through the chunks (without a device), and that a
sequence's results do not depend on what else the step brings or on which way the others go (on a device)."""
import pytest
import torch


def lengths(text):
    return [int(n) for part in text.split("+") for n in [part.split("x")[1]] * int(part.split("x")[0])]


# measured on B200, heads of 128 x 128 (us: every token by itself, every sequence in chunks of 64)
MEASURED = [(16, "1x64", 27, 29), (16, "1x128", 51, 37), (16, "1x2000", 743, 285), (16, "16x64", 107, 115), (16, "8x70", 70, 115), (16, "32x70", 227, 407),
            (16, "32x128", 401, 416), (16, "8x512", 465, 427), (16, "16x2000", 3104, 2886), (16, "1x64+63x1", 69, 439), (32, "1x64+63x1", 106, 863),
            (32, "16x64", 207, 228), (32, "32x70", 446, 790), (32, "2x2000", 1028, 812), (32, "16x2000", 6087, 5744), (4, "8x70", 30, 44), (4, "16x2000", 1029, 812)]


@pytest.mark.parametrize("heads,step,token,chunks", MEASURED)
def test_steps_of_one_kind_take_the_faster_way(heads, step, token, chunks):
    from ithaca_b200.csrc.ops import delta_chunks_from
    least = delta_chunks_from(lengths(step), heads, 128, 128, 148)
    if chunks > 1.05 * token:
        assert least == 0
    elif token > 1.05 * chunks:
        assert 0 < least <= min(lengths(step))


@pytest.mark.parametrize("heads", [4, 16, 32])
def test_short_sequences_stay_out_of_the_chunks(heads):
    from ithaca_b200.csrc.ops import delta_chunks_from
    for step in ("1x2000+63x1", "1x2000+15x30", "1x512+16x1"):
        assert 1 < delta_chunks_from(lengths(step), heads, 128, 128, 148) <= 512
    assert delta_chunks_from([1] * 200, heads, 128, 128, 148) == 0 and delta_chunks_from([], heads, 128, 128, 148) == 0
    assert delta_chunks_from([63] * 9, heads, 128, 128, 148) == 0


NEW = [1, 64, 31, 130, 0, 33, 200, 1] + [1, 2] * 16 + [65, 1, 0, 129, 32]           # more than one warp's worth of sequences


@pytest.mark.gpu
@pytest.mark.parametrize("H,G,dk,dv", [(4, 2, 128, 128), (2, 2, 64, 36), (40, 8, 64, 64)])
@pytest.mark.parametrize("least", [None, 0, 1, 32, 64, 129, 500])
def test_a_sequence_does_not_see_the_others(H, G, dk, dv, least):
    from types import SimpleNamespace
    from ithaca_b200.csrc import ops
    from test_delta_chunks_gpu import far, make
    start = [(7 * i) % 3 for i in range(len(NEW))]
    u, bg, before, ctx, cu, slots = make(H, G, dk, dv, NEW, start, dk + dv, "usual")
    ctx.host_n_new = NEW
    args = (4, 4 + G * dk, 4 + 2 * G * dk)
    state, state1 = before.clone(), before.clone()
    got = ops.delta_rule(u, *args, bg, state, ctx, H, G, dk, dv, chunks=True, chunks_from=least)
    token = ops.delta_rule(u, *args, bg, state1, ctx, H, G, dk, dv)
    cut = least if least is not None else ops.delta_chunks_from(NEW, H, dk, dv, ops.sm_count())
    for b, n in enumerate(NEW):
        rows = slice(cu[b], cu[b + 1])
        if n == 0 or cut == 0 or n < cut:
            assert torch.equal(got[rows], token[rows]) and torch.equal(state[slots[b]], state1[slots[b]])
            continue
        i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=u.device)
        alone = SimpleNamespace(n_seqs=1, max_new=max(n, 64), slots=i32([slots[b]]), cu_seqlens=i32([0, n]), kv_lens=i32([n + start[b]]), is_decode=False)
        s = before.clone()
        o = ops.delta_rule(u[rows], *args, bg[rows], s, alone, H, G, dk, dv, chunks=True)
        assert torch.equal(got[rows], o) and torch.equal(state[slots[b]], s[slots[b]])
        assert far(got[rows], token[rows]) < 5e-6                 # the bound that either way keeps to float64
    assert torch.equal(state[0], before[0])


@pytest.mark.gpu
def test_rows_off_sixteen_bytes_go_token_by_token():
    from ithaca_b200.csrc import ops
    from test_delta_chunks_gpu import make
    H, G, dk, dv = 2, 1, 64, 64
    u, bg, before, ctx, cu, slots = make(H, G, dk, dv, [150, 3], [0, 4], 1, "usual")
    off = torch.empty(u.shape[0] * u.shape[1] + 1, device=u.device)[1:].view(u.shape)
    off.copy_(u)
    made = []
    for x, chunks in ((off, True), (u, False)):
        s = before.clone()
        made.append((ops.delta_rule(x, 4, 4 + G * dk, 4 + 2 * G * dk, bg, s, ctx, H, G, dk, dv, chunks=chunks), s))
    assert torch.equal(made[0][0], made[1][0]) and torch.equal(made[0][1], made[1][1])
