"""The CUDA-core product and attention at the sizes that choose each of their launch shapes: every tile of the product, ragged sizes, rows off
16 bytes, and one, two and four heads a block of the attention with every option; a row bit for bit as it is alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(shape, seed, dtype=torch.float32):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV).to(dtype)


# tiles of 64 x 64, 128 x 64 and 128 x 128 on 148 SMs
@pytest.mark.parametrize("M,N", [(37, 129), (465, 2050), (465, 8200)])
@pytest.mark.parametrize("K,lead", [(1, 0), (3, 1), (17, 3), (48, 0), (48, 1), (301, 0), (300, 4)])
@pytest.mark.parametrize("xdt,wdt", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
def test_every_tile_of_the_product(M, N, K, lead, xdt, wdt):
    from ithaca_b200.csrc import ops
    x, w = rnd((M, K + lead), 1, xdt)[:, lead:], rnd((N, K + lead), 2, wdt)[:, lead:]
    got = ops.gemm_simt(x, w, out_dtype=torch.float32)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # float products summed in order: K roundings of at most 2^-24 of the sum of magnitudes each
    assert bool(((got.double() - want).abs() <= (K + 1) * 2.0 ** -24 * size).all())
    for r in (0, 5, M // 2, M - 1):
        assert torch.equal(ops.gemm_simt(x[r:r + 1], w, out_dtype=torch.float32)[0], got[r])
    base = rnd((M, N), 3)
    assert torch.equal(ops.gemm_simt(x, w, out=base.clone(), accumulate=True), base + got)


OPTIONS = [{}, {"softcap": 3.0}, {"sink": True}, {"sink": "learned"}, {"slopes": True}, {"scales": True}, {"window": 70}, {"window": 70, "keep": 5}, {"own": 24}, {"inside": True}]


@pytest.mark.parametrize("nh,nkv,hd", [(8, 2, 80), (8, 2, 50), (6, 3, 64), (8, 1, 512), (4, 1, 3072)])
@pytest.mark.parametrize("options", OPTIONS)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_heads_that_share_a_block(nh, nkv, hd, options, dtype):
    from ithaca_b200.csrc import ops
    T, start = 1200 if nh == 6 else 600, 9
    cols = -(-(T + start) // 64)
    o = dict(options)
    own = o.pop("own", 32 if hd > 512 else hd)
    k, q = rnd((cols + 2, nkv, 64, hd), 4, dtype), rnd((T, nh * hd), 5, dtype)
    v = rnd((cols + 2, nkv, 64, own), 6, dtype)
    more = {"softcap": o.get("softcap", 0.0), "keep": o.get("keep", 0)}
    if o.get("inside"):
        more["values_in_keys"] = min(hd, 48)
    if "sink" in o:
        more["sink"] = rnd((nh,), 7) if o["sink"] == "learned" else True
    if o.get("slopes"):
        more["slopes"] = rnd((nh,), 8).abs() * 0.1
    if o.get("scales"):
        more["key_scales"] = rnd((cols + 2, nkv, 64), 9).abs()
    table = torch.randperm(cols + 2, generator=torch.Generator().manual_seed(1))[:cols].to(torch.int32).view(1, cols).to(DEV)
    pos = torch.arange(start, start + T, dtype=torch.int32, device=DEV)
    seq = torch.zeros(T, dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    run = lambda at: ops.attention_simt(q[at], k, None if o.get("inside") else v, seq[at], pos[at], table, nh, hd ** -0.5, o.get("window", 0), status, **more)
    got = run(slice(0, T))
    for lo in (0, 1, 127, 300, T - 3):
        assert torch.equal(run(slice(lo, lo + 3)), got[lo:lo + 3]), lo
    assert status.item() == 0 and bool(torch.isfinite(got).all())
