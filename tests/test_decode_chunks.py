"""Pages per decode block for sequences of unequal lengths: the shapes that were measured, within the measured times; equal lengths as before."""
import random

import pytest

from ithaca_b200.csrc.attention_bf16 import decode_chunk_pages, decode_chunk_pages_uneven


def pages(n, longest):
    r = random.Random(f"{longest} {n}")
    return [-(-(r.randint(max(1, longest // 4), longest) + 1) // 64) for _ in range(n - 1)] + [-(-(longest + 1) // 64)]


# heads, kv heads, sequences, longest, us by chunk as measured on B200
MEASURED = [(32, 8, 8, 4000, {16: 30.4, 5: 21.0, 6: 20.6, 8: 23.1, 4: 24.7, 12: 29.2}), (32, 8, 16, 3000, {24: 41.5, 10: 28.0, 12: 31.2, 8: 33.8}),
            (32, 8, 10, 6000, {32: 53.7, 12: 34.3, 8: 42.4}), (32, 8, 24, 2000, {20: 39.7, 12: 31.8, 13: 33.4}), (32, 8, 20, 600, {8: 18.4, 4: 15.0, 3: 13.9}),
            (32, 8, 2, 5000, {5: 15.4, 3: 16.9}), (32, 8, 48, 3500, {20: 87.1, 12: 85.6}), (40, 40, 3, 8000, {63: 97.0, 12: 65.3}),
            (40, 40, 10, 6000, {20: 126.7, 12: 129.0}), (40, 40, 2, 5000, {27: 46.3, 12: 35.1}), (16, 2, 3, 8000, {4: 16.4, 2: 20.6})]


@pytest.mark.parametrize("nh,nkv,n,longest,us", MEASURED)
def test_measured_shapes(nh, nkv, n, longest, us):
    p = pages(n, longest)
    before = decode_chunk_pages(n, nh, nkv, max(p) * 64, n_sm=148)
    got = decode_chunk_pages_uneven(p, nh, nkv, before, 148)
    assert got in us and us[got] <= 1.12 * min(us.values()) and us[got] <= us[before]


@pytest.mark.parametrize("n", [1, 2, 8, 33, 64, 200])
@pytest.mark.parametrize("nh,nkv", [(32, 8), (40, 40), (6, 2), (64, 1)])
@pytest.mark.parametrize("longest", [1, 64, 700, 4096, 20000])
def test_bounds(n, nh, nkv, longest):
    most = -(-longest // 64)
    before = decode_chunk_pages(n, nh, nkv, longest, n_sm=148)
    assert decode_chunk_pages_uneven([most] * n, nh, nkv, before, 148) == before
    for p in (pages(n, longest), [most] + [1] * (n - 1)):
        assert 1 <= decode_chunk_pages_uneven(p, nh, nkv, before, 148) <= before
