"""The selective scan of whole sequences whose blocks share their work between warps, against float64: lengths on and off the edges of tiles and of
the four places a tile may lie in, channels and states off the edges of blocks and lanes, every optional input left out; and which steps take pieces."""
from types import SimpleNamespace

import pytest
import torch

DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("inner,N", [(3, 1), (33, 5), (64, 16), (40, 17), (32, 32), (20, 33), (24, 64)])
@pytest.mark.parametrize("new,start", [([1], [0]), ([16], [3]), ([17, 0, 15], [0, 4, 1]), ([31, 32, 33], [0, 0, 2]), ([64, 65, 95, 200], [1, 0, 0, 5])])
@pytest.mark.parametrize("less", [(), ("z",), ("D", "bias"), ("rows",)])
@pytest.mark.parametrize("odt", [torch.bfloat16, torch.float32])
def test_stream(inner, N, new, start, less, odt):
    from ithaca_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(inner + N)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    T, B, R = sum(new), len(new), 4 if "rows" not in less else 3              # (3: rows of B and C off 16 bytes)
    u, dt, bc, z = rnd(T, inner).to(torch.bfloat16), rnd(T, inner) - 2.0, rnd(T, R + 2 * N), rnd(T, 2 * inner)[:, inner:]
    A, D, bias = -torch.exp(rnd(inner, N) * 0.5), rnd(inner), rnd(inner) * 0.3
    A[0, 0] = -float("inf")                                                    # a state that forgets at once
    z, D, bias = (None if n in less else t for n, t in (("z", z), ("D", D), ("bias", bias)))
    before = rnd(B + 1, 2, inner, N)
    state = before.clone()
    cu = [sum(new[:i]) for i in range(B + 1)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    slots, ends = list(range(B, 0, -1)), [a + b for a, b in zip(new, start)]
    ctx = SimpleNamespace(n_seqs=B, max_new=max(new), slots=i32(slots), cu_seqlens=i32(cu), kv_lens=i32(ends), is_decode=False)
    y = ops.selective_scan(u, dt, bias, A, bc, R, R + N, D, z, state, ctx, odt, pieces=False)
    # The hardware's logarithm is off by 2^-21.4 at most for arguments between 1/2 and 2 (CUDA's documentation), so a step size is by 4e-7, which moves
    # a state by 4e-7 of W: the sum of what a step size multiplies, decayed.  Everything else is relative: 2e-6 of the sum of magnitudes.
    for b in range(B):
        S = before[slots[b], (start[b] - 1) & 1].double() if start[b] > 0 else torch.zeros(inner, N, dtype=torch.float64, device=DEV)
        mag, W = S.abs(), torch.zeros_like(S)
        for t in range(cu[b], cu[b + 1]):
            d = torch.nn.functional.softplus(dt[t].double() + (bias.double() if bias is not None else 0.0))
            xB, C = u[t].double()[:, None] * bc[t, R:R + N].double(), bc[t, R + N:].double()
            e = torch.exp(d[:, None] * A.double())
            W = e * W + xB.abs() + e * mag * A.double().abs().clamp(max=1e30)
            S, mag = e * S + d[:, None] * xB, e * mag + (d[:, None] * xB).abs()
            Du = D.double() * u[t].double() if D is not None else 0.0 * d
            g = torch.nn.functional.silu(z[t].double()) if z is not None else 1.0 + 0.0 * d
            want, size = (S @ C + Du) * g, (mag @ C.abs() + Du.abs()) * g.abs()
            bound = 4e-7 * (W @ C.abs()) * g.abs() + 2e-6 * size
            off = (y[t].double() - want).abs()
            assert bool((off <= bound + (2.0 ** -8 * want.abs() if odt == torch.bfloat16 else 0.0)).all())        # (rounded to 8 bits: half of the last place)
        if not new[b]:
            assert torch.equal(state[slots[b]], before[slots[b]])
            continue
        p = (ends[b] - 1) & 1
        assert bool(((state[slots[b], p].double() - S).abs() <= 4e-7 * W + 2e-6 * mag).all())
        if start[b] % 2 != ends[b] % 2:
            assert torch.equal(state[slots[b], 1 - p], before[slots[b], 1 - p])
    assert torch.equal(state[0], before[0])


@pytest.mark.gpu
@pytest.mark.parametrize("inner,N", [(40, 17), (64, 16)])                      # values one by one, and by fours
@pytest.mark.parametrize("T", [16, 21])
def test_numbers_that_are_not_finite(inner, N, T):
    """A NaN in A makes its channel's results and that state NaN; an infinite last input makes its channel's states infinite, also where the last tile
    is not full.  Other channels keep their bits."""
    from ithaca_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(T)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    u, dt, bc, z = rnd(T, inner).to(torch.bfloat16), rnd(T, inner), rnd(T, 4 + 2 * N), rnd(T, 2 * inner)[:, inner:]
    A, D, before = -torch.exp(rnd(inner, N) * 0.5), rnd(inner), rnd(1, 2, inner, N)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    ctx = SimpleNamespace(n_seqs=1, max_new=T, slots=i32([0]), cu_seqlens=i32([0, T]), kv_lens=i32([T + 2]), is_decode=False)

    def run(u, A):
        state = before.clone()
        return ops.selective_scan(u, dt, None, A, bc, 4, 4 + N, D, z, state, ctx, torch.float32, pieces=False), state[0, (T + 1) & 1]
    y0, S0 = run(u, A)
    bad_A, bad_u = A.clone(), u.clone()
    bad_A[3, 2], bad_u[T - 1, 7] = float("nan"), float("inf")
    y, S = run(bad_u, bad_A)
    assert bool(y[:, 3].isnan().all()) and bool(S[3, 2].isnan()) and int(S.isnan().sum()) == 1
    assert torch.equal(S[7], torch.copysign(torch.full_like(S[7], float("inf")), bc[T - 1, 4:4 + N])) and not bool(torch.isfinite(y[T - 1, 7]))
    same = torch.ones(inner, dtype=torch.bool, device=DEV)
    same[3] = same[7] = False
    assert torch.equal(y[:, same], y0[:, same]) and torch.equal(S[same], S0[same]) and torch.equal(y[:T - 1, 7], y0[:T - 1, 7])


# measured on B200: channels, states, step's longest and number of sequences, us whole, us in pieces
MEASURED = [(256, 16, 4000, 1, 152, 55), (512, 16, 8000, 1, 297, 110), (512, 16, 2000, 8, 86, 179), (2048, 16, 2000, 1, 80, 98), (2048, 16, 2000, 2, 86, 174),
            (4096, 16, 4000, 1, 167, 325), (64, 16, 2000, 1, 79, 41), (256, 64, 4000, 1, 177, 91), (1024, 64, 4000, 1, 179, 282), (1024, 64, 2000, 8, 504, 1001)]


@pytest.mark.parametrize("inner,N,longest,B,whole,pieces", MEASURED)
def test_steps_take_the_faster_way(inner, N, longest, B, whole, pieces):
    from ithaca_b200.csrc.ops import scan_pieces_beat_stream
    assert scan_pieces_beat_stream(longest * B, B, longest, inner, N, 148) == (pieces < whole)
