"""Kernels around the mixers that take several values a thread, at the sizes that choose each of their forms: the same bits as the value-at-a-time
form gives, and against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(shape, seed, std=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV) * std


# fewer fours than threads, more than a thread asks for ahead; a turning part of one four
@pytest.mark.parametrize("H,dk,dr,rank", [(1, 4, 4, 8), (16, 128, 64, 512), (40, 128, 64, 64), (3, 64, 0, 128)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_latent_prepare(H, dk, dr, rank, dtype):
    from ithaca_b200.csrc import ops
    T, cols = 67, 2
    made = []
    inv = (10000.0 ** (-torch.arange(dr // 2, device=DEV, dtype=torch.float32) * 2 / max(dr, 1))) if dr else None
    body, w = rnd((T, H * (dk + dr) + rank + dr), 1), rnd((rank,), 2)
    seq, pos = torch.zeros(T, dtype=torch.int32, device=DEV), torch.arange(T, dtype=torch.int32, device=DEV)
    table = torch.tensor([[1, 0]], dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    for lead in (0, 1):                                                         # (a row off 16 bytes goes a value at a time)
        p = torch.zeros((T, body.shape[1] + 4), device=DEV)
        p[:, lead:lead + body.shape[1]] = body
        qp, qf = torch.zeros((T, H * dk), dtype=dtype, device=DEV), torch.zeros((T, H * (rank + dr)), dtype=dtype, device=DEV)
        pages = torch.zeros((cols, 1, 64, rank + dr), dtype=dtype, device=DEV)
        ops.latent_prepare(p, lead, lead + H * (dk + dr), w, 1e-6, qp, qf, pages, seq, pos, table, inv, H, dk, dr, rank, True, status)
        made.append((qp, qf, pages))
    assert status.item() == 0 and all(torch.equal(a, b) for a, b in zip(*made))
    assert torch.equal(made[0][0], body[:, :H * (dk + dr)].view(T, H, dk + dr)[:, :, :dk].reshape(T, -1).to(dtype))


@pytest.mark.parametrize("T,H", [(3, 5), (1100, 9), (9473, 1)])               # an odd number of heads in all, one and two a warp
@pytest.mark.parametrize("dv", [64, 128, 96])
@pytest.mark.parametrize("gate", ["silu", "sigmoid"])
def test_head_norm_gate(T, H, dv, gate):
    from ithaca_b200.csrc import ops
    x, p, w = rnd((T, H * dv), 3), rnd((T, H * dv + 3), 4), rnd((dv,), 5)
    got = ops.head_norm_gate(x, w, 1e-6, p, 3, H, torch.float32, gate=gate)
    xd, g = x.double().view(T, H, dv), p[:, 3:].double().view(T, H, dv)
    want = xd * torch.rsqrt((xd * xd).mean(-1, keepdim=True) + 1e-6) * w.double() * (torch.sigmoid(g) * (g if gate == "silu" else 1.0))
    # a sum of dv squares, a root, a quotient, an exponential and four products: some 2^-24 each
    assert float(((got.double().view(T, H, dv) - want).abs() - 2e-6 * want.abs()).max()) <= 1e-30


@pytest.mark.parametrize("T,H,hdv", [(1, 1, 4), (5, 3, 64), (300, 16, 128), (2, 9, 132)])
@pytest.mark.parametrize("wide", [True, False])
@pytest.mark.parametrize("off", [0, 4, 3])
def test_head_gate(T, H, hdv, wide, off):
    from ithaca_b200.csrc import ops
    n = H * hdv if wide else H
    att, p = rnd((T, H * hdv), 6), rnd((T, off + n + 4 - (off + n) % 4), 7)
    out = torch.empty_like(att)
    ops.head_gate(att, p, off, out, H, mult=0.5, wide=wide)
    g = torch.sigmoid(p[:, off:off + n].double())
    want = att.double() * (g if wide else g.repeat_interleave(hdv, 1)) * 0.5
    assert float(((out.double() - want).abs() - 1e-6 * want.abs()).max()) <= 1e-30
