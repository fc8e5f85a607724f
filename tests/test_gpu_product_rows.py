"""The epilogues of the tcgen05 products that turn blocks of 32 x 32 round: rows and columns left over, outputs whose rows are not on
16 bytes (those go a row a lane), and the norm begun beside columns of both kinds.  Bounds: sums of K bfloat16 products in float,
K 2^-24 of the sum of magnitudes at most; one rounding to bfloat16 (2^-8) where the result is stored as such."""
import numpy as np
import pytest
import torch

from herbert_rs_b200 import ops

pytestmark = pytest.mark.gpu
K = 136


def _operands(M, N, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.1).to(torch.bfloat16)
    ref = a.double() @ w.double().T
    return a, w, ref, K * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T) + 1e-30


@pytest.mark.parametrize("M", [129, 512, 513, 799])
@pytest.mark.parametrize("N", [256, 296, 1001])
@pytest.mark.parametrize("extra", [0, 1, 4])
def test_every_row_stride_gives_the_same_numbers(M, N, extra):
    a, w, ref, bound = _operands(M, N, 5)
    wide = torch.full((M, N + extra), 7.0, device="cuda")
    ops.gemm_tcgen05(a, w, wide[:, :N], ops.EPI_STORE_F32)
    assert ((wide[:, :N].double() - ref).abs() <= bound).all() and (wide[:, N:] == 7.0).all()
    ops.gemm_tcgen05(a, w, wide[:, :N], ops.EPI_RESIDUAL)
    assert ((wide[:, :N].double() - 2 * ref).abs() <= 2 * bound + 2.0 ** -23 * ref.abs()).all() and (wide[:, N:] == 7.0).all()
    half = torch.full((M, N + extra), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.gemm_tcgen05(a, w, half[:, :N], ops.EPI_STORE)
    assert ((half[:, :N].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + bound).all() and (half[:, N:] == 7.0).all()
    ops.check_kernel_errors()


@pytest.mark.parametrize("M,N", [(512, 296), (517, 1000), (1025, 2048)])
def test_the_begun_norm_counts_every_column_once(M, N):
    a, w, ref, bound = _operands(M, N, 6)
    x = torch.randn(M, N, device="cuda")
    want = x.double() + ref
    nw = 1.0 + 0.1 * torch.randn(N, device="cuda")
    pend = ops.gemm_tcgen05_norm(a, w, x, ops.EPI_RESIDUAL, (nw, 1e-6), lambda shape, dtype: torch.full(shape, float("nan"), device="cuda", dtype=dtype))
    assert ((x.double() - want).abs() <= bound + 2.0 ** -23 * want.abs()).all()
    sums, exact = pend.sumsq[:, :M].double().sum(0), (x.double() ** 2).sum(1)
    assert ((sums - exact).abs() <= N * 2.0 ** -24 * exact).all()                       # float sums of N squares
    y = x.double() * nw.double()
    assert ((pend.xw.double() - y).abs() <= (2.0 ** -8 + 2.0 ** -20) * y.abs()).all()   # one rounding to bfloat16
    ops.check_kernel_errors()


@pytest.mark.parametrize("M,N", [(512, 296), (517, 1000), (1025, 2048)])
def test_a_rows_squares_are_added_column_by_column(M, N):
    """The same bits for whole blocks of 32 columns and for those left over: one multiply-add a column, in order (x86's 64-bit
    mantissa holds each exactly enough to be rounded once to float)."""
    a, w, _, _ = _operands(M, N, 7)
    x = torch.randn(M, N, device="cuda")
    pend = ops.gemm_tcgen05_norm(a, w, x, ops.EPI_RESIDUAL, (torch.ones(N, device="cuda"), 1e-6), lambda shape, dtype: torch.zeros(shape, device="cuda", dtype=dtype))
    parts, xs = pend.parts, x.cpu().numpy().astype(np.longdouble)
    half = next(h for h in (128, 64) if 2 * -(-N // (2 * h)) == parts)
    for i in range(parts):
        s = np.zeros(M, dtype=np.float32)
        for c in range(i * half, min(N, (i + 1) * half)):
            s = (s.astype(np.longdouble) + xs[:, c] * xs[:, c]).astype(np.float32)
        assert np.array_equal(pend.sumsq[i, :M].cpu().numpy(), s), i
    ops.check_kernel_errors()
