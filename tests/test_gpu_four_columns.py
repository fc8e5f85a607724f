"""Elementwise kernels that take four columns at a time: the same bits as the general kernels, which rows off 16 bytes go to."""
import pytest
import torch

from herbert_rs_b200 import ops

pytestmark = pytest.mark.gpu


def _off16(t):
    """The same rows, four bytes behind a 16-byte boundary."""
    flat = torch.empty(t.numel() + 4, device="cuda", dtype=t.dtype)
    out = flat[1:1 + t.numel()].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("tokens", [64, 65, 201])
@pytest.mark.parametrize("inter,interleave", [(4, 0), (1028, 0), (2048, 8), (48, 4)])
@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_tanh", "relu", "swish_clamp"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_bias_glu(tokens, inter, interleave, act, dtype):
    g = torch.Generator("cuda").manual_seed(tokens + inter)
    gu = torch.randn(tokens, 2 * inter, device="cuda", generator=g) * 3
    gu[0, 0], gu[1, inter], gu[2, 1] = float("inf"), float("nan"), -1e30
    for bias in (None, torch.randn(2 * inter, device="cuda", generator=g)):
        outs = []
        for rows in (gu, _off16(gu)):
            out = torch.empty(tokens, inter, device="cuda", dtype=dtype)
            ops.bias_glu(rows, bias, out, interleave, ops.ACTIVATIONS[act], 7.0)
            outs.append(torch.nan_to_num(out.float(), nan=12345.0, posinf=1e38, neginf=-1e38))
        assert torch.equal(*outs)


@pytest.mark.parametrize("rows", [64, 65, 201])
@pytest.mark.parametrize("col0,cols", [(0, 4), (8, 1028), (4, 2048)])
def test_silu_columns(rows, col0, cols):
    x = torch.randn(rows, col0 + cols + 4, device="cuda") * 5
    x[0, col0], x[1, col0 + 1] = float("-inf"), float("nan")
    a, b = x.clone(), _off16(x)
    ops.silu_columns(a, col0, cols)
    ops.silu_columns(b, col0, cols)
    assert torch.equal(torch.nan_to_num(a, nan=12345.0), torch.nan_to_num(b, nan=12345.0))
    assert torch.equal(a[:, :col0], x[:, :col0]) and torch.equal(a[:, col0 + cols:], x[:, col0 + cols:])


@pytest.mark.parametrize("extra", [0, 1, 138])
@pytest.mark.parametrize("inter,interleave", [(12, 0), (1028, 0), (2048, 8), (48, 4), (8192, 0)])
@pytest.mark.parametrize("act", ["silu", "swish_clamp"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_bias_glu_from_half_a_million_numbers_on(extra, inter, interleave, act, dtype):
    test_bias_glu(-(-512 * 1024 // inter) + extra, inter, interleave, act, dtype)


@pytest.mark.parametrize("extra", [0, 1, 138])
@pytest.mark.parametrize("col0,cols", [(0, 4), (8, 1028), (4, 2048), (0, 6144)])
def test_silu_columns_from_half_a_million_numbers_on(extra, col0, cols):
    test_silu_columns(-(-512 * 1024 // cols) + extra, col0, cols)
