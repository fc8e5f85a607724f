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
    # the hidden values are rounded to bfloat16 once (2^-8 each); float sums add far less
    want = ref + (y0.to(DEV).double() if accumulate else 0.0)
    assert ((y.double() - want).abs() <= size * 2.0 ** -8 + 1e-5).all()


@pytest.mark.parametrize("T,top,E", [(1, 1, 1), (1, 4, 32), (2, 3, 40), (8, 4, 32), (9, 2, 5), (16, 4, 33), (31, 2, 2), (32, 4, 100)])
@pytest.mark.parametrize("D,F", [(8, 8), (72, 40), (2048, 1408), (520, 264)])
@pytest.mark.parametrize("gated,weigh_input,accumulate,twice", [(0, False, True, False), (2, False, False, True), (2, True, True, False)])
@pytest.mark.parametrize("few", ["always", "never"])
def test_moe_few_by_choice(T, top, E, D, F, gated, weigh_input, accumulate, twice, few):
    """The same at every size with the experts read once for all tokens, and with a warp per output number."""
    saved, ops.options.moe_few = ops.options.moe_few, few
    try:
        test_moe_few(T, top, E, D, F, gated, weigh_input, accumulate, twice)
    finally:
        ops.options.moe_few = saved


@pytest.mark.parametrize("act", [ops.ACT_GELU, ops.ACT_SILU, ops.ACT_GELU_TANH])
@pytest.mark.parametrize("T,top,E,D,F", [(300, 2, 5, 136, 72), (130, 4, 16, 264, 392), (700, 1, 3, 512, 128)])
def test_moe_tc_plain_experts(act, T, top, E, D, F):
    g = torch.Generator(device=DEV).manual_seed(T + D)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    h, up, down = rnd(T, D).bfloat16(), (rnd(E, F, D) / D ** 0.5).bfloat16(), (rnd(E, D, F) / F ** 0.5).bfloat16()
    ids = torch.stack([torch.randperm(E, generator=g, device=DEV)[:top] for _ in range(T)]).int()
    wts = torch.rand(T, top, generator=g, device=DEV)
    y0 = rnd(T, D)
    assert ops.moe_tc_ok(h, up, top, 0, act) == (T * top >= ops.MOE_TC_MIN_PAIRS)
    assert not ops.moe_tc_ok(h, up, top, 0, ops.ACT_RELU)
    fn = {ops.ACT_GELU: torch.nn.functional.gelu, ops.ACT_SILU: torch.nn.functional.silu,
          ops.ACT_GELU_TANH: lambda z: torch.nn.functional.gelu(z, approximate="tanh")}[act]
    for accumulate in (True, False):
        y = y0.clone()
        ops.moe_experts_tc(h, up, down, ids, wts, y, accumulate, lambda s, dt: torch.empty(s, dtype=dt, device=DEV), gated=0, act=act)
        mid = fn(torch.einsum("td,efd->tef", h.double(), up.double()))
        chosen = torch.zeros(T, E, dtype=torch.float64, device=DEV).scatter_add_(1, ids.long(), wts.double())
        ref = torch.einsum("te,tef,edf->td", chosen, mid, down.double())
        size = torch.einsum("te,tef,edf->td", chosen, mid.abs(), down.double().abs())
        # the hidden values are rounded to bfloat16 once; float sums and the fast exponential add far less
        assert ((y.double() - ref - (y0.double() if accumulate else 0.0)).abs() <= size * 2.0 ** -8 + 1e-5).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [1, 7, 600, 1189])
@pytest.mark.parametrize("E,top,groups,keep", [(1, 1, 1, 1), (15, 3, 3, 2), (32, 4, 8, 4), (70, 6, 1, 1)])
@pytest.mark.parametrize("D", [8, 20, 264, 2048])
def test_moe_route_tiles(dtype, T, E, top, groups, keep, D):
    g = torch.Generator(device=DEV).manual_seed(T + E + D)
    h, r = torch.randn(T, D, generator=g, device=DEV).to(dtype), (torch.randn(E, D, generator=g, device=DEV) / D ** 0.5).to(dtype)
    ids = torch.full((T, top), -1, dtype=torch.int32, device=DEV)
    wts = torch.zeros(T, top, device=DEV)
    ops.moe_route(h, r, ids, wts, top, renorm=True, score=1, groups=groups, keep=keep, weight_scale=1.5)
    s = torch.sigmoid(h.double() @ r.double().T)
    if groups > 1:
        best = s.view(T, groups, -1).topk(2, -1).values.sum(-1)
        kept = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(keep, -1).indices, True)
        clear = best.sort(-1, descending=True).values
        sure = clear[:, keep - 1] - clear[:, keep] > 1e-5 if keep < groups else torch.ones(T, dtype=torch.bool, device=DEV)
        masked = s.masked_fill(~kept.repeat_interleave(E // groups, 1), -1.0)
    else:
        sure, masked = torch.ones(T, dtype=torch.bool, device=DEV), s
    ranked = masked.sort(-1, descending=True).values
    if top < E:
        sure &= ranked[:, top - 1] - ranked[:, top] > 1e-5
    assert (ids >= 0).all() and (ids < E).all()
    # where the last choice is no tie within float rounding, the choices are the largest scores; the weights are theirs
    want = masked.topk(top, -1)
    assert torch.equal(ids.long().sort(-1).values[sure], want.indices.sort(-1).values[sure])
    got = torch.gather(s, 1, ids.long())
    assert float((wts.double() - 1.5 * got / got.sum(-1, keepdim=True)).abs().max()) < 2e-5


@pytest.mark.parametrize("dtype,D", [(torch.float32, 20), (torch.bfloat16, 264), (torch.float32, 4096), (torch.bfloat16, 8192)])
@pytest.mark.parametrize("T", [148, 149, 591, 592, 741])
@pytest.mark.parametrize("E,top,groups,keep", [(8, 2, 1, 1), (9, 3, 3, 2), (16, 4, 4, 2), (17, 2, 1, 1)])
def test_moe_route_tokens_a_block(dtype, D, T, E, top, groups, keep):
    """One, two, four and eight tokens a block, at the token and expert counts where they change."""
    test_moe_route_tiles(dtype, T, E, top, groups, keep, D)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [3, 1201])
@pytest.mark.parametrize("E,top,groups,keep,score", [(32, 4, 8, 4, 1), (32, 4, 1, 1, 0), (15, 15, 3, 3, 0), (16, 2, 4, 1, 1), (6, 2, 1, 1, 1)])
@pytest.mark.parametrize("D", [20, 264])
def test_moe_route_scores_that_are_not_numbers(dtype, T, E, top, groups, keep, score, D):
    """A token whose scores are not numbers gets experts that exist, each once, and weights that are not numbers; no other token
    notices it.  An expert whose scores are not numbers is taken when nothing else is left."""
    g = torch.Generator(device=DEV).manual_seed(T + E + D)
    h, r = torch.randn(T, D, generator=g, device=DEV).to(dtype), (torch.randn(E, D, generator=g, device=DEV) / D ** 0.5).to(dtype)

    def route(h, r, top, keep):
        ids = torch.full((len(h), top), -7, dtype=torch.int32, device=DEV)
        wts = torch.zeros(len(h), top, device=DEV)
        ops.moe_route(h, r, ids, wts, top, renorm=True, score=score, groups=groups, keep=keep)
        return ids, wts
    ids0, wts0 = route(h, r, top, keep)
    bad = torch.tensor([t for t in (1, 7, 8, 600, T - 1) if t < T], device=DEV).unique()
    good = torch.ones(T, dtype=torch.bool, device=DEV)
    good[bad] = False
    broken = h.clone()
    broken[bad[0]] = float("nan")
    broken[bad[1:], 3] = float("nan")
    ids, wts = route(broken, r, top, keep)
    assert torch.equal(ids[good], ids0[good]) and torch.equal(wts[good], wts0[good])
    assert torch.equal(ids[bad], torch.arange(top, dtype=torch.int32, device=DEV).expand(len(bad), top))
    assert wts[bad].isnan().all()
    if score == 1:                                # a softmax over a score that is no number has none that is
        r2 = r.clone()
        r2[E // 2] = float("nan")
        ids, wts = route(h, r2, E if groups == 1 else keep * (E // groups), keep)
        assert (ids >= 0).all() and (ids < E).all() and (ids.sort(-1).values.diff(dim=-1) > 0).all()
        assert ((ids == E // 2) == (torch.arange(ids.shape[1], device=DEV) == ids.shape[1] - 1))[(ids == E // 2).any(-1)].all()
        assert groups > 1 or (ids[:, -1] == E // 2).all()


@pytest.mark.parametrize("path,dtype,T", [("experts", torch.float32, 9), ("experts", torch.bfloat16, 9), ("experts", torch.bfloat16, 40),
                                          ("grouped", torch.bfloat16, 300), ("tc", torch.bfloat16, 300)])
@pytest.mark.parametrize("gated", [0, 2])
def test_pairs_without_an_expert_contribute_nothing(path, dtype, T, gated):
    """Indices outside the experts: left out by every kernel, and nothing is written beside the scratch arrays."""
    E, top, D, F = 7, 3, 136, 72
    g = torch.Generator(device=DEV).manual_seed(T + gated)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    h, up, down = rnd(T, D).to(dtype), (rnd(E, 2 * F if gated else F, D) / D ** 0.5).to(dtype), (rnd(E, D, F) / F ** 0.5).to(dtype)
    ids = torch.stack([torch.randperm(E, generator=g, device=DEV)[:top] for _ in range(T)]).int()
    wts = torch.rand(T, top, generator=g, device=DEV)
    missing = torch.rand(T, top, generator=g, device=DEV) < 0.3
    missing[2] = True                               # a token with no expert at all
    broken = torch.where(missing, torch.tensor([E, -1, 2 ** 30], dtype=torch.int32, device=DEV).expand(T, top), ids)
    torch.cuda.synchronize()

    def call(ids, wts):
        y, guards = torch.zeros(T, D, device=DEV), []

        def scratch(shape, dt):
            n = 1
            for k in shape:
                n *= k
            whole = torch.full((n + 4096,), 77, dtype=dt, device=DEV)
            whole[2048:2048 + n] = 0
            guards.append((whole, n))
            return whole[2048:2048 + n].view(shape)
        if path == "experts":
            ops.moe_experts(h, up, down, ids, wts, scratch((T * top, F), dtype), y, ops.ACT_SILU, gated=gated)
        elif path == "grouped":
            ops.moe_experts_grouped(h, up, down, ids, wts, y, ops.ACT_SILU, False, scratch, gated=gated)
        else:
            ops.moe_experts_tc(h, up, down, ids, wts, y, False, scratch, gated=gated)
        for whole, n in guards:
            assert (whole[:2048] == 77).all() and (whole[2048 + n:] == 77).all()
        return y
    got, want = call(broken, wts), call(ids, wts.masked_fill(missing, 0.0))
    # the same products; a weight of 0 adds 0, so only the order of the kept pairs' sums may differ
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())
    assert (got[2] == 0).all()
