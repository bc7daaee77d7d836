"""The width of tiles of the products on pairs of SMs (a host function of the kernel library; no device)."""
import pytest


@pytest.fixture(scope="module")
def width():
    from ithaca_b200.csrc import ops
    return ops.lib().ik_gemm_wide_tile_width


def test_widths_of_plain_products(width):
    assert width(8, 0, 28672, 74) == 256 and width(8, 0, 4096, 74) == 256 and width(2, 0, 4096, 74) == 128


@pytest.mark.parametrize("tokens,top,experts,N,fastest", [(300, 2, 8, 4096, 256), (2048, 2, 8, 4096, 256), (600, 2, 16, 1024, 128)])
def test_a_plan_is_cut_for_the_tiles_in_use(width, tokens, top, experts, N, fastest):
    plan = tokens * top // 128 + experts                       # as the sort makes it: one tile to spare for every expert
    assert width(plan, experts, N, 148) == fastest             # measured; counted in full the plan got 192, 192 and 256
    assert width(plan, 0, N, 148) != fastest


def test_what_is_not_a_product_has_no_width(width):
    assert width(0, 0, 128, 74) == 0 and width(1, 0, 0, 74) == 0 and width(4, 100, 128, 74) in (128, 192, 256)
