"""The product for many tokens (two SMs to a tile): every epilogue and tile width at the edges of its tiles, against float64 and,
bit for bit, against the one-SM kernel, whose sums run in the same order."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from ithaca_b200.csrc import ops as o
    return o


def rnd(shape, seed, dtype=torch.bfloat16):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV).to(dtype)


# one token more or less than a tile, a block's half tile empty, features off every tile width, K off a step, fewer K steps than
# stages, more tiles than SMs
SHAPES = [(129, 128, 64), (256, 256, 512), (257, 320, 520), (300, 144, 72), (513, 1008, 1032), (1300, 4160, 200), (2100, 10288, 136)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("bn", [0, 128, 192, 256])
def test_gemm_wide(M, N, K, bn):
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    x, w = rnd((M, K), 1), rnd((N, K), 2)
    ref = x.double() @ w.double().T
    one = dict(status=status, wide=False, splits=1, pairs=False)
    two = dict(status=status, wide=True, wide_tile=bn)
    got = ops().gemm_tcgen05(x, w, **two)
    # float sums of K products in blocks of 16: the bound of the tests of the one-SM kernel
    assert float((got.double() - ref).abs().max() / ref.abs().max()) < 2e-5
    assert torch.equal(got, ops().gemm_tcgen05(x, w, **one))
    base = rnd((M, N), 3, torch.float32)
    assert torch.equal(ops().gemm_tcgen05(x, w, out=base.clone(), accumulate=True, **two),
                       ops().gemm_tcgen05(x, w, out=base.clone(), accumulate=True, **one))
    for more in ({}, {"act": "relu2"}, {"act": "gelu_tanh"}, {"swiglu": True}, {"swiglu": True, "glu": (1.5, 2.0, 1.0)}):
        assert torch.equal(ops().gemm_tcgen05(x, w, out_dtype=torch.bfloat16, **more, **two),
                           ops().gemm_tcgen05(x, w, out_dtype=torch.bfloat16, **more, **one)), more
    # rows of a wider matrix, and a destination whose rows are not on 16 bytes (another kernel takes it)
    big = torch.full((M, N + 5), 7.0, device=DEV)
    ops().gemm_tcgen05(x, w, out=big[:, :N], splits=1, **two)
    assert torch.equal(big[:, :N], got) and float((big[:, N:] - 7).abs().max()) == 0
    assert status.item() == 0


@pytest.mark.parametrize("M,hd,nh,nkv", [(257, 64, 5, 1), (700, 128, 8, 2), (1025, 192, 3, 3)])
@pytest.mark.parametrize("biased", [False, True])
def test_gemm_wide_rotary_epilogue(M, hd, nh, nkv, biased):
    K, N, n_pages = 264, (nh + 2 * nkv) * hd, 40
    x, w = rnd((M, K), 4), rnd((N, K), 5)
    seq = (torch.arange(M, device=DEV) >= 200).to(torch.int32)
    pos = torch.where(seq == 0, torch.arange(M, device=DEV), torch.arange(M, device=DEV) - 200 + 77).to(torch.int32)
    table = torch.randperm(n_pages, generator=torch.Generator().manual_seed(1))[:40].to(torch.int32).view(2, 20).to(DEV)
    cos_sin = ops().rope_table(pos, torch.rand(hd // 2, device=DEV))
    bias = rnd((N,), 6, torch.float32) if biased else None
    made = []
    for splits in (None, 1):
        q = torch.zeros((M, nh * hd), dtype=torch.bfloat16, device=DEV)
        k, v = (torch.zeros((n_pages, nkv, 64, hd), dtype=torch.bfloat16, device=DEV) for _ in range(2))
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        if splits is None:
            rs = ops().RopeStore(q.data_ptr(), k.data_ptr(), v.data_ptr(), cos_sin.data_ptr(), seq.data_ptr(), pos.data_ptr(), table.data_ptr(),
                                 status.data_ptr(), bias.data_ptr() if biased else 0, table.stride(0), nh, nkv, hd, 64, n_pages, 1)
            assert ops().lib().ik_gemm_qkv_rope_wide(x.data_ptr(), w.data_ptr(), M, N, K, K, K, 0, status.data_ptr(), ctypes.byref(rs),
                                                     torch.cuda.current_stream().cuda_stream) == 0
        else:
            assert ops().gemm_qkv_rope(x, w, q, k, v, cos_sin, seq, pos, table, nh, nkv, hd, True, status, splits=splits, bias=bias)
        assert status.item() == 0
        made.append((q, k, v))
    for a, b in zip(*made):
        # the rotation is compiled twice (a product and a sum may contract differently): one rounding to 8 bits apart at most
        assert float((a.float() - b.float()).abs().max()) <= 2 ** -7 * float(b.float().abs().max())
        assert float(((a != b).float()).mean()) < 1e-2
        assert torch.equal(a == 0, b == 0)


@pytest.mark.parametrize("rows", [128, 256])
@pytest.mark.parametrize("N,K,join", [(200, 72, 0), (1024, 520, 1), (144, 2048, 17)])
def test_gemm_wide_grouped(rows, N, K, join):
    E, tiles = 5, 9
    groups = torch.tensor([3, -1, 0, 0, 4, -1, 1, 2, -1], dtype=torch.int32, device=DEV)
    x, w = rnd((tiles * rows, K), 7), rnd((E * N, K), 8)
    made = []
    for name in ("ik_gemm_wide_grouped", "ik_gemm_tcgen05_grouped"):
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        dt = torch.bfloat16 if join else torch.float32
        y = torch.full((tiles * rows, N // 2 if join == 1 else N), 3.0, dtype=dt, device=DEV)
        assert getattr(ops().lib(), name)(x.data_ptr(), w.data_ptr(), y.data_ptr(), 1 if join else 0, groups.data_ptr(), E, rows, tiles * rows, N, K, K, K,
                                          y.stride(0), join, status.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        assert status.item() == 0
        made.append(y)
    assert torch.equal(*made)
    assert float((made[0][rows:2 * rows].float() - 3).abs().max()) == 0


@pytest.mark.parametrize("M,N,K", [(2048, 2048, 2048), (513, 8192, 256)])
def test_results_without_an_activation_cost_no_more_than_floats(M, N, K):
    """Half the bytes and no more arithmetic: 16-bit results once took up to 2.6 times the time of float ones."""
    x, w, status = rnd((M, K), 1), rnd((N, K), 2), torch.zeros(1, dtype=torch.int32, device=DEV)
    best = {}
    for dtype in (torch.float32, torch.bfloat16):
        out = torch.empty((M, N), dtype=dtype, device=DEV)
        graph = torch.cuda.CUDAGraph()
        run = lambda: ops().gemm_tcgen05(x, w, out=out, wide=True, status=status)
        run()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            for _ in range(10):
                run()
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        best[dtype] = min(times)
    assert best[torch.bfloat16] < 1.25 * best[torch.float32], best


def test_which_products_run_on_pairs_of_SMs():
    takes = ops().wide_takes
    assert takes(2048, 4096, 4096) and takes(300, 4096, 4096) and takes(130, 28672, 4096)
    assert not takes(128, 28672, 4096) and not takes(130, 6144, 4096) and not takes(256, 4096, 14336)
    assert takes(400, 8192, 256) and not takes(192, 8192, 256) and not takes(257, 8192, 512) and takes(257, 8192, 1024)


@pytest.mark.parametrize("M,hd,nh,nkv", [(513, 128, 16, 4), (700, 64, 24, 4), (900, 80, 16, 4)])
def test_rotary_products_as_they_are_dispatched(M, hd, nh, nkv):
    """Heads of a multiple of 64 go to the pairs of SMs, others to the kernel that takes them."""
    K, N, n_pages = 1032, (nh + 2 * nkv) * hd, 40
    x, w = rnd((M, K), 4), rnd((N, K), 5)
    seq, pos = torch.zeros(M, dtype=torch.int32, device=DEV), torch.arange(M, dtype=torch.int32, device=DEV)
    table = torch.randperm(n_pages, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(1, n_pages).to(DEV)
    cos_sin = ops().rope_table(pos, torch.rand(hd // 2, device=DEV))
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    made = []
    for way in ("dispatched", "wide", "other"):
        q = torch.zeros((M, nh * hd), dtype=torch.bfloat16, device=DEV)
        k, v = (torch.zeros((n_pages, nkv, 64, hd), dtype=torch.bfloat16, device=DEV) for _ in range(2))
        if way == "wide":
            rs = ops().RopeStore(q.data_ptr(), k.data_ptr(), v.data_ptr(), cos_sin.data_ptr(), seq.data_ptr(), pos.data_ptr(), table.data_ptr(),
                                 status.data_ptr(), 0, table.stride(0), nh, nkv, hd, 64, n_pages, 1)
            st = ops().lib().ik_gemm_qkv_rope_wide(x.data_ptr(), w.data_ptr(), M, N, K, K, K, 0, status.data_ptr(), ctypes.byref(rs),
                                                   torch.cuda.current_stream().cuda_stream)
            assert st == (-2 if hd % 64 else 0)
        else:
            assert ops().gemm_qkv_rope(x, w, q, k, v, cos_sin, seq, pos, table, nh, nkv, hd, True, status, splits=None if way == "dispatched" else 1)
        made.append((q, k, v))
    assert status.item() == 0 and ops().wide_takes(M, N, K)
    for a, b in zip(made[0], made[2 if hd % 64 else 1]):
        assert torch.equal(a, b) and float(a.float().abs().max()) > 0
