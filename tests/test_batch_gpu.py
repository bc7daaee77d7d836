"""The product for up to 128 tokens in every way it shares out its work (blocks to a tile x slices of K): against 64 bits at the edges of tokens, features and
K steps, what the epilogues make of the sums, rotary results and cache rows, and which products come here."""
import pytest
import torch

DEV = "cuda:0"
WAYS = [0] + [16 * cg + s for cg in (1, 2) for s in (1, 2, 4)]


def rnd(shape, seed, dtype=torch.bfloat16, std=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(shape, generator=g, device=DEV) * std).to(dtype)


def takes(way, K):
    s, steps = max(way % 16, 1), -(-K // 64)
    return (s - 1) * -(-steps // s) < steps


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 9, 63, 64, 65, 128])
@pytest.mark.parametrize("N,K", [(2, 64), (130, 520), (257, 1096), (300, 4096), (5000, 200)])
@pytest.mark.parametrize("way", WAYS)
def test_product(M, N, K, way):
    from ithaca_b200.csrc import ops
    if not takes(way, K):
        pytest.skip("a slice would hold no K step: refused")
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    x, w = rnd((M, K + 8), 1)[:, 8:], rnd((N, K + 16), 2)[:, :K]
    more = {"batch": way, "status": status}
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    got = ops.gemm_tcgen05(x, w, **more)
    # exact products; an instruction of 16 drops less than 2^-23 of its largest term twice, slices are added in float
    assert bool(((got.double() - want).abs() <= (2 * -(-K // 16) + 4) * 2.0 ** -23 * size).all())
    wide = rnd((M, N + 5), 3, torch.float32)
    into = wide.clone()
    ops.gemm_tcgen05(x, w, out=into[:, 3:3 + N], accumulate=True, **more)
    assert torch.equal(into[:, 3:3 + N], wide[:, 3:3 + N] + got) and torch.equal(into[:, :3], wide[:, :3]) and torch.equal(into[:, 3 + N:], wide[:, 3 + N:])
    assert torch.equal(ops.gemm_tcgen05(x, w, out_dtype=torch.bfloat16, **more), got.bfloat16())
    for act, f in (("relu2", lambda v: torch.relu(v) ** 2), ("gelu_tanh", lambda v: torch.nn.functional.gelu(v, approximate="tanh"))):
        if act in ops.PLAIN_ACTS:
            a = ops.gemm_tcgen05(x, w, out_dtype=torch.bfloat16, act=act, **more)
            assert bool(((a.double() - f(got.double())).abs() <= 2.0 ** -8 * f(got.double()).abs() + 1e-5 * got.double().abs()).all())     # (one rounding to 8 bits, tanh's error)
    if N % 2 == 0:
        for glu in (None, (1.5, 2.0, 1.0)):
            j = ops.gemm_tcgen05(x, w, out_dtype=torch.bfloat16, swiglu=True, glu=glu, **more)
            gate, up = got[:, 0::2].double(), got[:, 1::2].double()
            a, limit, shift = glu or (1.0, 1e30, 0.0)
            gate, up = gate.clamp(max=limit), up.clamp(-limit, limit)
            r = gate * torch.sigmoid(a * gate) * (up + shift)
            assert bool(((j.double() - r).abs() <= 2.0 ** -8 * r.abs() + 1e-6).all())
    assert status.item() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M", [5, 64, 77, 128])
@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 64), (3, 1, 80), (8, 8, 128)])
@pytest.mark.parametrize("way", WAYS)
@pytest.mark.parametrize("bias", [False, True])
def test_rotary_results(M, nh, nkv, hd, way, bias):
    """The same bits as the product of gemm_tcgen05.cu rounded the same way: compared with the plain product's sums."""
    from ithaca_b200.csrc import ops
    K, N, cols = 1600, (nh + 2 * nkv) * hd, 3
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    x, w, b = rnd((M, K), 4), rnd((N, K), 5, std=K ** -0.5), rnd((N,), 6, torch.float32) if bias else None
    seq = torch.arange(M, dtype=torch.int32, device=DEV) % 5
    pos = torch.arange(M, dtype=torch.int32, device=DEV) * 7 % (64 * cols)
    table = torch.randperm(5 * cols, generator=torch.Generator().manual_seed(1)).view(5, cols).to(torch.int32).to(DEV)
    cos_sin = ops.rope_table(pos, 10000.0 ** (-torch.arange(hd // 2, device=DEV, dtype=torch.float32) * 2 / hd))
    q, k, v = torch.zeros((M, nh * hd), dtype=torch.bfloat16, device=DEV), *(torch.zeros((5 * cols, nkv, 64, hd), dtype=torch.bfloat16, device=DEV) for _ in range(2))
    assert ops.gemm_qkv_rope(x, w, q, k, v, cos_sin, seq, pos, table, nh, nkv, hd, True, status, skinny_max=0, bias=b, batch=way)
    s = ops.gemm_tcgen05(x, w, batch=way, status=status).double() + (b.double() if bias else 0.0)
    s = s.view(M, nh + 2 * nkv, hd // 2, 2)
    c, sn = cos_sin[:, None, :, 0].double(), cos_sin[:, None, :, 1].double()
    turned = torch.stack((s[..., 0] * c - s[..., 1] * sn, s[..., 0] * sn + s[..., 1] * c), -1).view(M, nh + 2 * nkv, hd)
    plain = s.reshape(M, nh + 2 * nkv, hd)
    near = lambda got, want: bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all())
    assert near(q.view(M, nh, hd), turned[:, :nh])
    page, at = table[seq.long(), pos.long() // 64].long(), pos.long() % 64
    last = {(p, a): i for i, (p, a) in enumerate(zip(page.tolist(), at.tolist()))}             # (of two tokens at one place either may stand)
    rows = torch.tensor(sorted(last.values()), device=DEV)
    if len(rows) == M:
        assert near(k[page, :, at], turned[:, nh:nh + nkv]) and near(v[page, :, at], plain[:, nh + nkv:])
    assert status.item() == 0


@pytest.mark.gpu
def test_what_it_refuses():
    from ithaca_b200.csrc import ops
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    x, w = rnd((129, 256), 7), rnd((256, 256), 8)
    assert torch.equal(ops.gemm_tcgen05(x, w, batch=0, status=status), ops.gemm_tcgen05(x, w, status=status))     # more tokens: the ways there were
    with pytest.raises(ops.KernelError):
        ops.gemm_tcgen05(x[:5], w, batch=16 * 3 + 1, status=status)
    assert status.item() == 0


# measured on B200: tokens, features, K, us in the ways of gemm_tcgen05.cu, us here
@pytest.mark.parametrize("M,N,K,other,here", [(17, 28672, 4096, 43.5, 41.2), (64, 4096, 4096, 17.0, 11.5), (128, 6144, 4096, 26.6, 15.8), (17, 2048, 8192, 11.4, 13.6),
                                              (48, 2048, 8192, 12.8, 13.7), (100, 2048, 8192, 17.1, 15.9), (24, 1536, 6144, 9.7, 11.1), (24, 128256, 2048, 82.7, 84.4),
                                              (100, 128256, 2048, 94.1, 90.3), (65, 1024, 512, 8.8, 5.1),
                                              (80, 2048, 8192, 16.0, 16.4), (104, 2048, 8192, 17.7, 16.4), (96, 768, 16384, 16.4, 22.5), (64, 2048, 16384, 20.1, 21.8), (17, 2304, 6144, 10.9, 12.6),
                                              (104, 1280, 10240, 16.0, 17.4), (40, 1024, 4096, 10.7, 9.0), (80, 512, 4096, 11.3, 11.0), (65, 2560, 16384, 25.0, 26.9), (65, 3072, 16384, 28.5, 28.1),
                                              (48, 2560, 10240, 20.2, 16.7), (64, 128256, 4096, 179.2, 174.6), (32, 96000, 2048, 69.9, 66.2)])
def test_products_take_the_faster_way(M, N, K, other, here, monkeypatch):
    from ithaca_b200.csrc import ops
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    assert ops.batch_takes(M, N, K) == (here < other)


@pytest.mark.gpu
def test_two_threads_with_other_shares():
    """Two shares of one instance want other amounts of shared memory: neither thread's launch is refused for what the other asked for."""
    import threading

    from ithaca_b200.csrc import ops
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    x, w = rnd((40, 1024), 1), rnd((256, 1024), 2)
    want = {way: ops.gemm_tcgen05(x, w, batch=way, status=status) for way in (17, 18, 20)}
    failed = []

    def work(way):
        y = torch.zeros_like(want[way])                         # (a kernel: the thread has the device's context from here on)
        try:
            for _ in range(3000):
                ops.gemm_tcgen05(x, w, out=y, batch=way, status=status)
            torch.cuda.synchronize()
            if not torch.equal(y, want[way]):
                failed.append(f"{way}: other bits")
        except Exception as e:
            failed.append(f"{way}: {e}")
    threads = [threading.Thread(target=work, args=(way,)) for way in (17, 18, 20)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed and status.item() == 0
