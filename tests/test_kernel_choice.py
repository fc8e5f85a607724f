"""Rules that choose a kernel from a step's sizes, where they need no GPU."""
import pytest
import torch

from herbert_rs_b200 import ops


@pytest.mark.parametrize("top,E,D,F,gated,loses,pays", [
    (4, 32, 2048, 1408, 0, 0, 1), (4, 32, 2048, 1408, 2, 0, 1), (2, 16, 1024, 768, 0, 4, 8), (2, 16, 1024, 768, 2, 2, 4),
    (2, 8, 1024, 512, 0, 8, 12), (8, 128, 2048, 768, 0, 0, 1)])
def test_experts_are_read_once_where_a_step_shares_them(top, E, D, F, gated, loses, pays):
    """`loses`, `pays`: tokens at which a warp per output number and experts read once for all tokens were measured to be faster."""
    assert not any(ops.moe_few_pays(t, top, E, D, F, gated) for t in range(1, loses + 1))
    assert all(ops.moe_few_pays(t, top, E, D, F, gated) for t in range(pays, 33))


@pytest.mark.parametrize("top,E,D,F", [(1, 4, 256, 128), (2, 4, 64, 96), (1, 1, 64, 64)])
def test_small_experts_keep_a_warp_per_output_number(top, E, D, F):
    assert not any(ops.moe_few_pays(t, top, E, D, F, g) for t in range(1, 33) for g in (0, 2))


@pytest.mark.parametrize("E,top,T,D,F,want", [(32, 4, 128, 2048, 1408, True), (1024, 8, 64, 2048, 1408, True), (1024, 8, 64, 64, 32, False),
                                              (1024, 1, 65535, 64, 32, True), (16, 4, 130, 264, 392, True), (256, 2, 256, 128, 64, False)])
def test_padding_of_plain_experts_stays_small(E, top, T, D, F, want):
    h, up = torch.empty(T, D, dtype=torch.bfloat16), torch.empty(1, dtype=torch.bfloat16).expand(E, F, D)
    assert ops.moe_tc_ok(h, up, top, 0, ops.ACT_SILU) == want


def test_padded_rows_hold_every_way_to_spread_the_pairs():
    """m experts with c_1 .. c_m pairs need the sum of ceil(c_i / 128) tiles: most where all but one have a single pair, or 128 k + 1."""
    rows = lambda T, E, top: ops._fn("hb_moe_experts_tc_rows")(T, E, top)
    for T, E, top in ((1, 1, 1), (128, 32, 4), (513, 7, 1), (64, 1024, 8), (300, 2, 2), (65535, 1024, 8), (129, 1, 1)):
        P = T * top
        m = min(E, P)
        spread = [1] * (m - 1) + [P - (m - 1)]
        odd = [1 + 128 * ((P - m) // 128 // m)] * m
        odd[0] += P - sum(odd)
        for c in (spread, odd):
            assert sum(c) == P and min(c) >= 1
            assert sum(-(-n // 128) for n in c) * 128 <= rows(T, E, top)
        assert rows(T, E, top) <= P + 127 * m
