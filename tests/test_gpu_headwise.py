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


@pytest.mark.parametrize("T,H,K,N,gap", [(128, 1, 16, 131, 0), (200, 3, 64, 190, 1), (130, 2, 128, 128, 0), (257, 2, 24, 258, 2)])
def test_gates_of_a_row_in_pairs_and_one_by_one(T, H, K, N, gap):
    """Gates two at a time (an even width, rows on even columns) and one by one, at the last outputs of a tile."""
    g = torch.Generator(device=DEV).manual_seed(T + K + N)
    src = torch.randn(T, H * K, generator=g, device=DEV)
    w = (torch.randn(H, N, K, generator=g, device=DEV) / K ** 0.5).bfloat16()
    gate = torch.randn(T, H * N + gap, generator=g, device=DEV)[:, :H * N]
    out = torch.full((T, H * N), 5.0, device=DEV)
    ops.headwise_gemm(src, K, w, out, N, scale=0.7, gate=gate)
    ref = torch.einsum("thk,hnk->thn", src.view(T, H, K).bfloat16().double(), w.double()) * 0.7
    want = ref * torch.sigmoid(gate.double()).reshape(T, H, N)
    assert float((out.view(T, H, N).double() - want).abs().max()) <= 2e-5      # float sums of up to 128 products of unit size
