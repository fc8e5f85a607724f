"""The 32-bit products and the any-shape attention at the edges of their tiles, row counts and ranges of K."""
import pytest
import torch

from herbert_rs_b200 import ops
from test_gpu_kernels import _attention_case, close, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 3, 4, 5, 8, 9, 16, 17, 63, 65, 130])
@pytest.mark.parametrize("N,K", [(1, 4), (7, 132), (129, 1028), (1024, 2048), (3001, 124), (130, 4096)])
def test_gemm_f32_rows_and_tiles(M, N, K):
    g = torch.Generator().manual_seed(M * 131 + N + K)
    a, w, r = torch.randn(M, K + 4, generator=g), torch.randn(N, K, generator=g), torch.randn(M, N + 1, generator=g)
    ref = a[:, :K].double() @ w.double().T
    # rounding of a sum of K products of unit size: sqrt(K) * 2^-24 of sqrt(K) each way, six times that at most over all outputs
    tol = 6 * K * 2.0 ** -24 + 1e-6
    out = torch.full((M, N + 1), 7.0, device="cuda")
    ops.gemm_simt(dev(a)[:, :K], dev(w), out[:, :N], ops.EPI_STORE)
    assert float((out[:, :N].cpu().double() - ref).abs().max()) <= tol
    assert (out[:, N] == 7.0).all()
    res = dev(r.clone())
    ops.gemm_simt(dev(a)[:, :K], dev(w), res[:, :N], ops.EPI_RESIDUAL)
    assert float((res[:, :N].cpu().double() - ref - r[:, :N].double()).abs().max()) <= tol + 1e-6
    assert torch.equal(res[:, N].cpu(), r[:, N])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd", [(2, 1, 33), (4, 2, 128), (2, 2, 132), (2, 1, 500)])
@pytest.mark.parametrize("window", [None, 257])
def test_attention_simt_runs_of_keys(dtype, nh, nkv, hd, window):
    few = ([1, 32, 33, 256, 257, 600], [1, 2, 1, 1, 3, 1])
    for lens, qlens in (few, ([620, 9], [600, 9])):          # eight warps a unit, and two
        _runs(dtype, nh, nkv, hd, window, lens, [min(n, q) for n, q in zip(lens, qlens)])


def _runs(dtype, nh, nkv, hd, window, lens, qlens):
    c = _attention_case(dtype, nh, nkv, hd, lens, qlens, window)
    out = torch.empty(c["q"].shape, device="cuda", dtype=dtype)
    ops.attention_simt(dev(c["q"]), c["q"].shape[1], out, dev(c["k"]), dev(c["v"]), dev(c["tok_seq"]), dev(c["tok_pos"]),
                       dev(c["table"]), nh, nkv, hd, 16, c["scale"], window)
    close(out, c["ref"], dtype, rowwise=True)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hd", [1, 126, 127, 130, 254, 257, 511])
def test_attention_simt_heads_of_no_multiple_of_four(dtype, hd):
    """The instances for up to 128, 256 and 512 channels, a channel at a time."""
    test_attention_simt_runs_of_keys(dtype, 2, 1, hd, None)
