"""The gated delta rule of a prompt in chunks of 64 tokens, against float64 and the token-by-token kernel: sequences of several chunks,
of one, of none, with and without an earlier state, lengths on and off the chunks' edges, decays near 0 and 1."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def make(H, G, dk, dv, new, start, seed, decay):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    T, B = sum(new), len(new)
    u = rnd(T, 4 + 2 * G * dk + H * dv)
    for off, mult in ((4, dk ** -0.5), (4 + G * dk, 1.0)):
        x = u[:, off:off + G * dk].view(T, G, dk)
        u[:, off:off + G * dk] = (x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6) * mult).view(T, -1)
    bg = torch.sigmoid(rnd(T, 2, H))
    bg[:, 1] = {"usual": 1 - 0.2 * bg[:, 1] ** 2, "near one": 1 - 1e-4 * bg[:, 1], "small": bg[:, 1] ** 8}[decay]
    if decay == "small":
        bg[::7, 1] = 0.0
    state = rnd(B + 1, 2, H, dv, dk)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    cu = [sum(new[:i]) for i in range(B + 1)]
    slots = list(range(B, 0, -1))
    ctx = SimpleNamespace(n_seqs=B, max_new=max(new), slots=i32(slots), cu_seqlens=i32(cu), kv_lens=i32([a + b for a, b in zip(new, start)]),
                          is_decode=False)
    return u, bg.contiguous(), state, ctx, cu, slots


def far(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


@pytest.mark.parametrize("H,G,dk,dv", [(4, 2, 128, 128), (2, 2, 64, 64), (3, 1, 128, 36), (2, 1, 64, 20), (40, 8, 128, 128)])
@pytest.mark.parametrize("new,start", [([200], [0]), ([3, 0, 129, 64, 63], [5, 0, 0, 12, 0])])
@pytest.mark.parametrize("decay", ["usual", "near one", "small"])
def test_delta_rule_in_chunks(H, G, dk, dv, new, start, decay):
    from ithaca_b200.csrc import ops
    u, bg, before, ctx, cu, slots = make(H, G, dk, dv, new, start, dk + dv, decay)
    assert ops.lib().ik_delta_chunks_scratch(cu[-1], len(new), max(new), H, dk, dv) > 0
    args = (4, 4 + G * dk, 4 + 2 * G * dk, bg)
    state, state1 = before.clone(), before.clone()
    o = ops.delta_rule(u, *args, state, ctx, H, G, dk, dv, chunks=True)
    o1 = ops.delta_rule(u, *args, state1, ctx, H, G, dk, dv)
    ud, bd = u.double(), bg.double()
    for b, (n, first) in enumerate(zip(new, start)):
        if n == 0:
            assert torch.equal(state[slots[b]], before[slots[b]])
            continue
        S = before[slots[b], (first - 1) & 1].double() if first > 0 else torch.zeros(H, dv, dk, dtype=torch.float64, device=DEV)
        want = []
        for t in range(cu[b], cu[b + 1]):
            q, k = (ud[t, off:off + G * dk].view(G, dk).repeat_interleave(H // G, 0) for off in (4, 4 + G * dk))
            S = S * bd[t, 1][:, None, None]
            x = bd[t, 0][:, None] * (ud[t, 4 + 2 * G * dk:].view(H, dv) - torch.einsum("hvk,hk->hv", S, k))
            S = S + x[:, :, None] * k[:, None, :]
            want.append(torch.einsum("hvk,hk->hv", S, q).reshape(-1))
        rows, p = slice(cu[b], cu[b + 1]), (first + n - 1) & 1
        want = torch.stack(want)
        # float sums of at most dk + 64 products, carried on by the decays: as far off as token by token, give or take
        assert far(o[rows], want) < max(1.5 * far(o1[rows], want), 1e-6) and far(o[rows], want) < 5e-6
        assert far(state[slots[b], p], S) < max(1.5 * far(state1[slots[b], p], S), 1e-6)
        if (first - 1) & 1 != p:
            assert torch.equal(state[slots[b], 1 - p], before[slots[b], 1 - p])
    assert torch.equal(state[0], before[0])


@pytest.mark.parametrize("where", ["k", "v", "decay", "factor"])
def test_what_is_not_finite_stays_behind_its_token(where):
    from ithaca_b200.csrc import ops
    H, G, dk, dv = 2, 1, 128, 64
    u, bg, before, ctx, cu, slots = make(H, G, dk, dv, [150], [0], 3, "usual")
    args = (4, 4 + G * dk, 4 + 2 * G * dk)
    whole = ops.delta_rule(u, *args, bg, before.clone(), ctx, H, G, dk, dv, chunks=True)
    bad_u, bad_bg = u.clone(), bg.clone()
    if where in ("decay", "factor"):
        bad_bg[101, int(where == "decay")] = float("nan")
    else:
        bad_u[101, 4 + G * dk if where == "k" else 4 + 2 * G * dk + 5] = float("inf") if where == "v" else float("nan")
    got = ops.delta_rule(bad_u, *args, bad_bg, before.clone(), ctx, H, G, dk, dv, chunks=True)
    assert torch.equal(got[:101], whole[:101])
    assert not torch.isfinite(got[101]).all() and not torch.isfinite(got[149]).all()


@pytest.mark.parametrize("H,G,dk,dv", [(3, 1, 128, 36), (2, 2, 64, 64), (40, 8, 128, 64)])            # 16 and 32 columns a block
def test_columns_beside_one_that_is_not_finite(H, G, dk, dv):
    from ithaca_b200.csrc import ops
    u, bg, before, ctx, cu, slots = make(H, G, dk, dv, [200, 64], [0, 9], 4, "usual")
    args = (4, 4 + G * dk, 4 + 2 * G * dk, bg)
    state, state1, bad = before.clone(), before.clone(), u.clone()
    whole = ops.delta_rule(u, *args, state, ctx, H, G, dk, dv, chunks=True)
    col = (H - 1) * dv + 19
    bad[77, 4 + 2 * G * dk + col] = float("-inf")
    got = ops.delta_rule(bad, *args, state1, ctx, H, G, dk, dv, chunks=True)
    others = torch.arange(H * dv, device=DEV) != col
    assert torch.equal(got[:, others], whole[:, others]) and torch.equal(got[:77], whole[:77]) and torch.equal(got[200:], whole[200:])
    assert not torch.isfinite(got[77:200, col]).any()
    p = 199 & 1
    assert not torch.isfinite(state1[slots[0], p, H - 1, 19]).any()
    state1[slots[0], p, H - 1, 19] = state[slots[0], p, H - 1, 19]
    assert torch.equal(state1, state)


@pytest.mark.parametrize("at", [77, 127, 149])                    # within a chunk, a chunk's last token, the prompt's
@pytest.mark.parametrize("what", [float("inf"), float("-inf"), float("nan")])
def test_an_infinity_is_what_it_is_token_by_token(at, what):
    """Its own token's results, and the state behind the last token, stay infinite; later ones are NaN."""
    from ithaca_b200.csrc import ops
    H, G, dk, dv = 2, 1, 128, 64
    u, bg, before, ctx, cu, slots = make(H, G, dk, dv, [150], [0], 3, "usual")
    col = dv + 5
    u[at, 4 + 2 * G * dk + col] = what
    made = []
    for chunks in (True, False):
        state = before.clone()
        o = ops.delta_rule(u, 4, 4 + G * dk, 4 + 2 * G * dk, bg, state, ctx, H, G, dk, dv, chunks=chunks)
        made.append((o[at:, col], state[slots[0], 1, 1, 5]))
    for got, want in zip(*made):
        assert not torch.isfinite(want).any()
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got == float("inf"), want == float("inf")) and torch.equal(got.isinf(), want.isinf())


@pytest.mark.parametrize("decay", [0.01, 0.1])
def test_strong_decays(decay):
    """A state that is a few tokens' products is not further from 64 bits than token by token."""
    from ithaca_b200.csrc import ops
    H, G, dk, dv, T = 4, 2, 128, 128, 360
    u, bg, before, ctx, cu, slots = make(H, G, dk, dv, [T], [0], 7, "usual")
    bg[:, 1] = decay * (0.8 + 0.4 * torch.rand((T, H), generator=torch.Generator(device=DEV).manual_seed(1), device=DEV))
    made = []
    for chunks in (True, False):
        state = before.clone()
        ops.delta_rule(u, 4, 4 + G * dk, 4 + 2 * G * dk, bg, state, ctx, H, G, dk, dv, chunks=chunks)
        made.append(state[slots[0], 1])
    S = torch.zeros(H, dv, dk, dtype=torch.float64, device=DEV)
    for t in range(T):
        k = u[t, 4 + G * dk:4 + 2 * G * dk].double().view(G, dk).repeat_interleave(H // G, 0)
        S = S * bg[t, 1].double()[:, None, None]
        x = bg[t, 0].double()[:, None] * (u[t, 4 + 2 * G * dk:].double().view(H, dv) - torch.einsum("hvk,hk->hv", S, k))
        S = S + x[:, :, None] * k[:, None, :]
    # about four roundings to nearest of terms that are hardly ever as large as the sum: 2 * 2^-24 / sqrt(3)
    assert far(made[0], S) < 6e-8 and far(made[0], S) < far(made[1], S)
