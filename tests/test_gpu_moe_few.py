"""The routed feed-forward of few tokens against a float64 restatement, at the edges of its tiles, ranges and token groups."""
import pytest
import torch

from herbert_rs_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T,top,E", [(1, 1, 1), (1, 4, 32), (2, 3, 40), (8, 4, 32), (9, 2, 5), (16, 4, 33), (31, 2, 2), (32, 4, 100)])
@pytest.mark.parametrize("D,F", [(8, 8), (72, 40), (2048, 1408), (520, 264)])
@pytest.mark.parametrize("gated,weigh_input,accumulate,twice", [(0, False, True, False), (2, False, False, True), (2, True, True, False)])
def test_moe_few(T, top, E, D, F, gated, weigh_input, accumulate, twice):
    g = torch.Generator().manual_seed(T * 1000 + D + gated)
    h = torch.randn(T, D, generator=g).bfloat16()
    N = 2 * F if gated else F
    up = (torch.randn(E, N, D, generator=g) / D ** 0.5).bfloat16()
    down = (torch.randn(E, D, F, generator=g) / F ** 0.5).bfloat16()
    ids = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).int()
    if twice:
        ids[:, -1] = ids[:, 0]                      # an expert named twice by one token counts twice
    wts = torch.rand(T, top, generator=g) + 0.1
    y0 = torch.randn(T, D, generator=g)
    mid = torch.empty(T * top, F, dtype=torch.bfloat16, device=DEV)
    y = y0.to(DEV)
    upd, downd = up.to(DEV), down.to(DEV)
    ops.moe_experts(h.to(DEV), upd, downd, ids.to(DEV), wts.to(DEV), mid, y, ops.ACT_SILU if gated else ops.ACT_GELU, accumulate=accumulate,
                    gated=gated, weigh_input=weigh_input)
    hd, ref, size = h.to(DEV).double(), torch.zeros(T, D, dtype=torch.float64, device=DEV), torch.zeros(T, D, dtype=torch.float64, device=DEV)
    for t in range(T):
        for r in range(top):
            e, w = int(ids[t, r]), float(wts[t, r])
            z = upd[e].double() @ hd[t]
            if gated:
                rows = z.view(F // 8, 2, 8)
                a, b = rows[:, 0].reshape(-1), rows[:, 1].reshape(-1)
                if weigh_input:
                    a, b = a * w, b * w
                m = torch.nn.functional.silu(a) * b
            else:
                m = torch.nn.functional.gelu(z)
            ref[t] += (1.0 if weigh_input else w) * (downd[e].double() @ m)
            size[t] += (1.0 if weigh_input else w) * (downd[e].double().abs() @ m.abs())
    # the hidden values are rounded to bfloat16 once (2^-9 each); float sums add far less
    want = ref + (y0.to(DEV).double() if accumulate else 0.0)
    assert ((y.double() - want).abs() <= size * 2.0 ** -8 + 1e-5).all()
