"""The products of few rows where their ring of weight batches can go wrong: every depth (by the CTAs an SM gets), rows and columns left
over, fewer steps of K than warps, units that follow one another in a CTA, every group of activation rows.  Bounds: sums of K
bfloat16 products in float, K 2^-24 of the sum of magnitudes at most; one rounding to bfloat16 where the result is stored so."""
import pytest
import torch

from herbert_rs_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 8, 9, 16, 29, 64])
@pytest.mark.parametrize("N,K", [(24, 8), (48, 264), (1024, 2048), (2376, 1032), (4744, 520), (8200, 264), (33032, 136), (2048, 8200)])
def test_every_depth_and_every_edge(M, N, K):
    g = torch.Generator("cuda").manual_seed(N + K + M)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.1).to(torch.bfloat16)
    ref = a.double() @ w.double().T
    bound = K * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T) + 1e-30
    for _ in range(2):
        c = torch.full((M, N), float("nan"), device="cuda")
        ops.gemm_skinny(a, w, c, ops.EPI_STORE_F32)
        assert ((c.double() - ref).abs() <= bound).all()
    half = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_skinny(a, w, half)
    assert ((half.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + bound).all()
    # a NaN in a row of the weights or of the activations stays in its column or row
    w[N - 1, K - 1] = float("nan")
    a[0, 0] = float("nan")
    ops.gemm_skinny(a, w, c, ops.EPI_STORE_F32)
    assert torch.isnan(c[0]).all() and torch.isnan(c[:, N - 1]).all()
    assert M == 1 or ((c[1:, :N - 1].double() - ref[1:, :N - 1]).abs() <= bound[1:, :N - 1]).all()


@pytest.mark.parametrize("M", [17, 32, 33, 40, 57])
@pytest.mark.parametrize("N,K", [(24, 8), (48, 264), (2376, 1032), (4744, 520), (8200, 264)])
def test_the_edges_of_the_ring_and_of_the_products_without_it(M, N, K):
    """17 to 32 rows with the ring, 33 to 64 with a batch in registers: one unit a CTA and several."""
    test_every_depth_and_every_edge(M, N, K)
