"""Products per head of many tokens against float64, at the edges of their tiles."""
import pytest
import torch

from herbert_rs_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T,H,K,N", [(128, 2, 128, 512), (257, 3, 512, 130), (300, 1, 40, 128), (129, 2, 8, 200)])
def test_product_per_head_of_many_tokens(T, H, K, N):
    g = torch.Generator(device=DEV).manual_seed(T + K + N)
    src = torch.randn(T, H * (K + 4), generator=g, device=DEV)
    w = (torch.randn(H, N, K, generator=g, device=DEV) / K ** 0.5).bfloat16()
    gate = torch.randn(T, H * N, generator=g, device=DEV)
    ref = torch.einsum("thk,hnk->thn", src.view(T, H, K + 4)[:, :, :K].bfloat16().double(), w.double()) * 0.7
    for gap in (0, 3):                                           # pairs of results side by side, and one by one
        out = torch.full((T, H * (N + gap)), 5.0, device=DEV)
        ops.headwise_gemm(src, K + 4, w, out, N + gap, scale=0.7)
        got = out.view(T, H, N + gap)
        assert float((got[:, :, :N].double() - ref).abs().max()) <= 2e-5      # float sums of up to 512 products of unit size
        assert gap == 0 or (got[:, :, N:] == 5.0).all()
    out = torch.empty(T, H * N, dtype=torch.bfloat16, device=DEV)
    ops.headwise_gemm(src, K + 4, w, out, N, scale=0.7, gate=gate)
    want = ref * torch.sigmoid(gate.double()).view(T, H, N)
    assert ((out.view(T, H, N).double() - want).abs() <= want.abs() * 2.0 ** -8 + 2e-5).all()
