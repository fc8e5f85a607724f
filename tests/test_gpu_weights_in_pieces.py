"""Small products inside the preparing kernels of the recurrences: sixteen weights at a time where rows are pieces of 16 bytes, the same
bits as a weight at a time, which weights off 16 bytes go to."""
import pytest
import torch

from herbert_rs_b200 import ops

pytestmark = pytest.mark.gpu


def _off16(t):
    flat = torch.empty(t.numel() + 8, device="cuda", dtype=t.dtype)
    out = flat[1:1 + t.numel()].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("tokens", [1, 8, 67])
@pytest.mark.parametrize("channels,rank", [(130, 16), (1024, 32), (97, 40), (256, 24)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gla_decay(tokens, channels, rank, dtype):
    low, w2 = torch.randn(tokens, rank, device="cuda"), torch.randn(channels, rank, device="cuda").to(dtype)
    bias = torch.randn(channels, device="cuda")
    outs = [torch.empty(tokens, channels, device="cuda") for _ in range(2)]
    for w, out in zip((w2, _off16(w2)), outs):
        ops.gla_decay(low, w, bias, 16.0, out)
    assert torch.equal(*outs)
    want = torch.sigmoid(low.double() @ w2.double().T + bias.double()) ** (1 / 16)
    assert ((outs[0].double() - want).abs() <= 1e-5).all()      # sums of at most 40 products, a sigmoid and its sixteenth root


@pytest.mark.parametrize("tokens", [1, 5, 70])
@pytest.mark.parametrize("heads,dk,rank", [(2, 64, 16), (3, 40, 48), (1, 300, 24), (2, 128, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_general_delta_prepare(tokens, heads, dk, rank, dtype):
    n = heads * dk
    rows = torch.randn(tokens, 3 * n + rank, device="cuda")
    w2, w0, a0 = (torch.randn(n, rank, device="cuda") * 0.3).to(dtype), torch.randn(n, device="cuda"), torch.randn(n, device="cuda")
    outs = [torch.empty(tokens, heads, 5, dk, device="cuda") for _ in range(2)]
    for w, out in zip((w2, _off16(w2)), outs):
        ops.general_delta_prepare(rows, 0, n, 2 * n, 3 * n, w, w0, a0, 0.6, 1e-6, out, heads, dk)
    assert torch.equal(*outs)
    want = torch.exp(-0.6 * torch.sigmoid(torch.tanh(rows[:, 3 * n:].double()) @ w2.double().T + w0.double())).view(tokens, heads, dk)
    assert ((outs[0][:, :, 2].double() - want).abs() <= 1e-5).all()
