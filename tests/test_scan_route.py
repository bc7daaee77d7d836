"""Which steps run the selective scan in pieces (without a device), and the pieces against whole sequences where the rule would not take them
(on a device): many short sequences beside a long one, more sequences than pieces."""
import pytest
import torch


def lengths(text):
    return [int(n) for part in text.split("+") for n in [part.split("x")[1]] * int(part.split("x")[0])]


# measured on B200: channels, states, step, us in whole sequences, us in pieces
MEASURED = [(4096, 16, "1x200", 26, 39), (4096, 16, "1x1000", 116, 88), (4096, 16, "1x4000", 454, 318), (4096, 16, "2x2000", 287, 318),
            (4096, 16, "3x2000", 381, 451), (4096, 16, "8x2000", 790, 1083), (4096, 16, "1x2000+63x1", 352, 250), (4096, 16, "1x200+63x1", 46, 122),
            (4096, 16, "4x512+32x1", 147, 201), (8192, 16, "1x4000", 569, 622), (8192, 16, "4x2000", 790, 1084), (2048, 16, "1x2000", 214, 92),
            (2048, 16, "2x2000", 229, 168), (2048, 16, "8x2000", 538, 614), (512, 16, "8x2000", 229, 172), (2048, 32, "2x2000", 339, 290),
            (2048, 32, "8x2000", 771, 1038), (1024, 64, "1x4000", 587, 275), (1024, 64, "8x2000", 647, 995), (4096, 64, "1x2000", 406, 515)]


@pytest.mark.parametrize("inner,N,step,whole,pieces", MEASURED)
def test_steps_take_the_faster_way(inner, N, step, whole, pieces):
    from ithaca_b200.csrc.ops import scan_pieces_pay
    new = lengths(step)
    pays = scan_pieces_pay(sum(new), len(new), max(new), inner, N, 148)
    if max(whole, pieces) > 1.06 * min(whole, pieces):
        assert pays == (pieces < whole)


def test_a_step_that_does_not_say_its_longest_goes_whole():
    from ithaca_b200.csrc.ops import scan_pieces_pay
    assert not scan_pieces_pay(5000, 1, 0, 4096, 16, 148)


@pytest.mark.gpu
@pytest.mark.parametrize("inner,N", [(40, 5), (4096, 16), (33, 20), (64, 64)])
@pytest.mark.parametrize("new", [[3, 0, 257, 192, 64, 65], [1] * 40 + [700] + [2] * 30, [200] * 5])
def test_pieces_asked_for(inner, N, new):
    from types import SimpleNamespace
    from ithaca_b200.csrc import ops
    dev = "cuda:0"
    g = torch.Generator(device=dev).manual_seed(inner + N)
    rnd = lambda *s: torch.randn(s, generator=g, device=dev)
    T, B = sum(new), len(new)
    u, dt, bc, z = rnd(T, inner).to(torch.bfloat16), rnd(T, inner) - 2.0, rnd(T, 2 * N), rnd(T, inner)
    A, D = -torch.exp(rnd(inner, N) * 0.5), rnd(inner)
    before = rnd(B, 2, inner, N)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    start = [i % 3 for i in range(B)]
    ctx = SimpleNamespace(n_seqs=B, max_new=max(new), slots=i32(list(range(B))), cu_seqlens=i32([sum(new[:i]) for i in range(B + 1)]),
                          kv_lens=i32([a + b for a, b in zip(new, start)]), is_decode=False)
    made = []
    for pieces in (True, False):
        state = before.clone()
        made.append((ops.selective_scan(u, dt, None, A, bc, 0, N, D, z, state, ctx, torch.bfloat16, pieces=pieces).double(), state.double()))
    (y, s), (y1, s1) = made
    assert float((y - y1).norm() / y1.norm()) < 3e-3              # either is rounded to 8 bits once: 1.7e-3 on average if all fell differently
    assert float((s - s1).norm() / s1.norm()) < 6e-6              # twice the bound that either keeps to float64
