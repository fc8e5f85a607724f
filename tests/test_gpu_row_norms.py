"""The kernels that keep a row in registers, at the widths where their shapes change, against float64 (and the widths beside them,
which the general kernels take)."""
import pytest
import torch

from herbert_rs_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"
WIDTHS = [128, 132, 1024, 2048, 2176, 4096, 8192, 8320]
DT = [torch.float32, torch.bfloat16]


def _near(got, ref, dtype):
    # float sums of up to 8,320 numbers, six roundings deep; bfloat16 results are rounded once more
    rel = 3e-6 if dtype == torch.float32 else 2.0 ** -8
    assert float((got.double() - ref).abs().max()) <= rel * max(1.0, float(ref.abs().max()))


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("D", WIDTHS)
@pytest.mark.parametrize("rows", [1, 5])
def test_row_norms(D, rows, dtype):
    g = torch.Generator(device=DEV).manual_seed(D + rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    y, z, x0 = rnd(rows, D) + 0.3, rnd(rows, D), rnd(rows, D)
    w, w2, bias, scale = rnd(D), rnd(D), rnd(D), rnd(D)
    eps = 1e-5
    yd, zd, xd = y.double(), z.double(), x0.double()
    rms = lambda v, groups=1: (v.view(rows, groups, -1) / (v.view(rows, groups, -1).pow(2).mean(-1, keepdim=True) + eps).sqrt()).view(rows, D)

    for gate, next_norm, want_h in ((True, True, True), (False, False, True), (True, False, False)):
        x, h = x0.clone(), torch.empty(rows, D, dtype=dtype, device=DEV)
        ops.gated_norm_residual(y, w, eps, x, dtype, gate=z if gate else None, gate_bias=bias if gate else None,
                                next_norm=(w2, eps) if next_norm else None, h=h if want_h else None)
        v = yd * torch.sigmoid(zd + bias.double()) if gate else yd
        ref = xd + rms(v) * w.double()
        _near(x, ref, torch.float32)
        if want_h:
            _near(h, rms(ref) * w2.double() if next_norm else ref, dtype)

    for groups in [n for n in (1, 2, 4) if D % n == 0]:
        x, h = x0.clone(), torch.empty(rows, D, dtype=dtype, device=DEV)
        ops.group_rmsnorm_residual(y, w, x, h, eps, groups, dtype, bias=bias, second=(z, 0.75, -0.5))
        ref = xd + rms(0.75 * yd - 0.5 * zd + bias.double(), groups) * w.double()
        _near(x, ref, torch.float32); _near(h, ref, dtype)
        picked = torch.tensor(list(range(rows))[::-1], dtype=torch.int32, device=DEV)
        ops.group_rmsnorm(y, w, h, eps, groups, rows=picked)
        _near(h, (rms(yd, groups) * w.double()).flip(0), dtype)

    ln = (yd - yd.mean(-1, keepdim=True)) / (yd.var(-1, unbiased=False, keepdim=True) + eps).sqrt() * w.double()
    for s in (scale, None):
        x, h = x0.clone(), torch.empty(rows, D, dtype=dtype, device=DEV)
        ops.layernorm_residual(y, w, s, x, h, eps, dtype)
        ref = xd + (ln * s.double() if s is not None else ln)
        _near(x, ref, torch.float32); _near(h, ref, dtype)
    h = torch.empty(rows, D, dtype=dtype, device=DEV)
    ops.layernorm(y, w, h, eps, bias=bias)
    _near(h, ln + bias.double(), dtype)

    x, h = x0.clone(), torch.empty(rows, D, dtype=dtype, device=DEV)
    ops.scaled_residual_norm(y, 0.5, x, w, h, eps)
    ref = xd + 0.5 * yd
    _near(x, ref, torch.float32); _near(h, rms(ref) * w.double(), dtype)

    table, pos = rnd(9, D).to(dtype), rnd(4, D).to(dtype)
    ids, at = torch.tensor([8, 0, -1, 9, 3][:rows], dtype=torch.int32, device=DEV), torch.tensor([0, 3, 1, 2, 4][:rows], dtype=torch.int32, device=DEV)
    out = torch.full((rows, 2, D), 7.0, device=DEV)
    ops.embed(table, ids, out, 1.5, pos, at)
    for t in range(rows):
        i, p = int(ids[t]), int(at[t])
        ref = table[i].float() * 1.5 + (pos[p].float() if p < 4 else 0.0) if 0 <= i < 9 else torch.zeros(D, device=DEV)
        _near(out[t], ref.double().expand(2, D), torch.float32)


@pytest.mark.parametrize("n,D", [(1, 128), (1, 2688), (2, 256), (2, 3200), (3, 384), (3, 2560), (4, 2048), (4, 2176), (4, 4096), (4, 132), (5, 256)])
@pytest.mark.parametrize("rows", [1, 148, 149, 300])
@pytest.mark.parametrize("rms", [False, True])
def test_copies_of_the_stream(n, D, rows, rms):
    """One to four copies a row in registers and beside it: the narrowest and widest rows, and the rows an SM where wide ones change."""
    g = torch.Generator(device=DEV).manual_seed(n * D + rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x0, y, mix, ow, iw, w, bias = rnd(rows, n, D), rnd(rows, D), rnd(n, n) * 0.5, rnd(n), rnd(n), rnd(D), rnd(D)
    x, h = x0.clone(), torch.empty(rows, D, device=DEV)
    ops.streams_join(x, y, mix, ow, iw, norm=(w, bias, 1e-5, rms), h=h)
    ref = torch.einsum("st,rsd->rtd", mix.double(), x0.double()) + ow.double()[:, None] * y.double()[:, None]
    _near(x, ref, torch.float32)
    u = torch.einsum("t,rtd->rd", iw.double(), ref)
    mean = 0.0 if rms else u.mean(-1, keepdim=True)
    want = (u - mean) / ((u - mean).pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w.double() + bias.double()
    # the norm divides by the spread of u: its float error is that of u over it, a few roundings of the largest of n + 1 terms
    assert float((h.double() - want).abs().max()) <= 2e-5 * max(1.0, float(want.abs().max()))
