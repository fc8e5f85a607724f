"""Rules that choose a kernel from a step's sizes, where they need no GPU."""
import pytest

from herbert_rs_b200 import ops


@pytest.mark.parametrize("top,E,D,F,gated,loses,pays", [
    (4, 32, 2048, 1408, 0, 2, 3), (4, 32, 2048, 1408, 2, 1, 4), (2, 16, 1024, 768, 0, 8, 12), (2, 16, 1024, 768, 2, 4, 8),
    (2, 8, 1024, 512, 0, 8, 12), (8, 128, 2048, 768, 0, 2, 4), (2, 8, 4096, 14336, 0, 1, 3)])
def test_experts_are_read_once_where_a_step_shares_them(top, E, D, F, gated, loses, pays):
    """`loses`, `pays`: tokens at which a warp per output number and experts read once for all tokens were measured to be faster."""
    assert not any(ops.moe_few_pays(t, top, E, D, F, gated) for t in range(1, loses + 1))
    assert all(ops.moe_few_pays(t, top, E, D, F, gated) for t in range(pays, 33))


@pytest.mark.parametrize("top,E,D,F", [(1, 4, 256, 128), (2, 4, 64, 96), (1, 1, 64, 64)])
def test_small_experts_keep_a_warp_per_output_number(top, E, D, F):
    assert not any(ops.moe_few_pays(t, top, E, D, F, g) for t in range(1, 33) for g in (0, 2))
