"""The 32-bit path's product on the tensor cores (three bfloat16 planes of the tokens) at the edges of its tiles, K steps and slices: against 64
bits, the same bits from every tile and for a row alone, and where numbers are not finite."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(shape, seed, dtype=torch.float32):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV).to(dtype)


# one row to three tiles of 256, features about 256, K of less than a step, ragged steps, two and eight slices
@pytest.mark.parametrize("M", [1, 31, 33, 129, 257, 513])
@pytest.mark.parametrize("N,K", [(1, 256), (255, 264), (257, 1000), (130, 40), (300, 4104), (64, 16392)])
def test_every_tile(M, N, K):
    from ithaca_b200.csrc import ops
    x, w = rnd((M, K + 3), 1)[:, 3:], rnd((N, K + 8), 2, torch.bfloat16)[:, 8:]
    got = ops.gemm_split(x, w)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # an instruction drops less than 2^-23 of its largest term for the alignment and again for the sum: 24 in a chain of 12; then K / 64
    # roundings of 2^-24 between chains and at most eight between slices
    assert bool(((got.double() - want).abs() <= (24 + (K // 64 + 9) / 2) * 2.0 ** -23 * size).all())
    assert float((got.double() - want).norm() / want.norm()) < 2.5e-7          # (measured 0.8 to 1.4e-7)
    for tile in (32, 64, 128, 256):
        for side in (False, True):
            assert torch.equal(ops.gemm_split(x, w, tile=tile, side_by_side=side), got), (tile, side)
    for r in {0, M // 2, M - 1}:
        assert torch.equal(ops.gemm_split(x[r:r + 1], w)[0], got[r])
    wide = rnd((M, N + 5), 3)
    base, into = wide.clone(), wide[:, 2:2 + N]
    ops.gemm_split(x, w, out=into, accumulate=True)
    assert float((into.double() - base[:, 2:2 + N].double() - want).norm()) < 4e-7 * float((base[:, 2:2 + N].double() + want).norm() + want.norm())
    assert torch.equal(wide[:, :2], base[:, :2]) and torch.equal(wide[:, 2 + N:], base[:, 2 + N:])
    for side in (False, True):
        again = base.clone()
        ops.gemm_split(x, w, out=again[:, 2:2 + N], accumulate=True, tile=64, side_by_side=side)
        assert torch.equal(again, wide)
    assert ops.device_status(torch.device(DEV)).item() == 0


def test_rows_in_turns(monkeypatch):
    from ithaca_b200.csrc import ops
    x, w = rnd((150, 320), 4), rnd((70, 320), 5, torch.bfloat16)
    got = ops.gemm_split(x, w)
    monkeypatch.setattr(ops, "SPLIT_ROWS", 64)
    assert torch.equal(ops.gemm_split(x, w), got)
    assert ops.gemm_split(x[:0], w).shape == (0, 70)


def test_numbers_that_are_not_finite():
    """Infinities and NaN in the tokens and in the weights come out where the CUDA-core product has them."""
    from ithaca_b200.csrc import ops
    x, w = rnd((40, 512), 6), rnd((300, 512), 7, torch.bfloat16)
    inf, nan = float("inf"), float("nan")
    x[3, 5], x[4, 7], x[5, 9], x[6], x[7, 1] = inf, nan, -inf, 0.0, 3e38
    x[8, 11] = torch.tensor([0x7f800001], dtype=torch.int32, device=DEV).view(torch.float32)[0]
    x[9] = x[9].bfloat16().float()                                             # two of its planes are zeros
    w[10, 3], w[11, 4], w[12, 6], w[13] = inf, nan, -inf, 0.0
    a, b = ops.gemm_simt(x, w), ops.gemm_split(x, w)
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a == inf, b == inf) and torch.equal(a == -inf, b == -inf)
    assert int(a[[3, 5]].isinf().sum()) >= 2 * 296 and bool(a[[4, 8]].isnan().all())


def test_small_numbers():
    """Every plane of a small number is there: the same bits as of a larger one, down to where a float itself has fewer."""
    from ithaca_b200.csrc import ops
    x, w = rnd((40, 512), 10), rnd((300, 512), 11, torch.bfloat16)
    x = torch.where(x.abs() < 2.0 ** -8, torch.ones_like(x), x)
    got = ops.gemm_split(x, w)
    assert torch.equal(ops.gemm_split(x * 2.0 ** -110, w * 2.0 ** 60) * 2.0 ** 50, got)
    tiny = (torch.randint(-2 ** 22, 2 ** 22, (40, 512), generator=torch.Generator().manual_seed(1)) * 2).double().to(DEV) * 2.0 ** -149
    small = tiny.float()
    assert torch.equal(small.double(), tiny)
    want = tiny @ (w.double() * 2.0 ** 100).T
    assert float((ops.gemm_split(small, w * 2.0 ** 100).double() - want).norm() / want.norm()) < 2.5e-7


def test_dispatch():
    """The rule asks for nothing but the weight's form, so that rows do not change with the rows beside them."""
    from ithaca_b200.csrc import ops
    from ithaca_b200.parts import linear
    w = rnd((64, 512), 8, torch.bfloat16)
    for rows in (1, 40):
        x = rnd((rows, 512), 9)
        assert ops.split_takes(x, w) and torch.equal(linear.gemm(x, w), ops.gemm_split(x, w))
        for other in (w.float(), rnd((64, 516), 8, torch.bfloat16)[:, 4:], rnd((64, 513), 8, torch.bfloat16)[:, :512]):
            assert not ops.split_takes(x, other) and torch.equal(linear.gemm(x, other), ops.gemm_simt(x, other))
        short = rnd((64, 248), 8, torch.bfloat16)
        assert not ops.split_takes(x[:, :248], short) and not ops.split_takes(x.bfloat16(), w) and not ops.split_takes(x, w, torch.bfloat16)
        assert torch.equal(linear.gemm(x[:, :248], short), ops.gemm_simt(x[:, :248], short))
