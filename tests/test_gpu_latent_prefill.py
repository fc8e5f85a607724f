"""Prompts' attention over a cached latent on tcgen05 against float64: both halves of the latent, blocks beyond its width, windows,
sinks, starts behind cached keys, shuffled pages, rows that do not fill a tile."""
from types import SimpleNamespace

import pytest
import torch

from herbert_rs_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("H,rank,rot", [(16, 512, 64), (16, 256, 32), (5, 320, 16), (8, 64, 0), (3, 512, 0), (40, 128, 64)])
@pytest.mark.parametrize("window,sunk,page", [(None, False, 64), (100, True, 128), (None, True, 64)])
def test_latent_prefill(H, rank, rot, window, sunk, page):
    need = -(-150 * 128 // (H * -(-rank // 256)))
    qlens = [need, 1, 67, 130]
    pos0 = [0, 200, 63, 0]
    lens = [p + n for p, n in zip(pos0, qlens)]
    g = torch.Generator(device=DEV).manual_seed(H + rank + rot)
    W = rank + rot
    total = sum(-(-n // page) for n in lens)
    order = torch.randperm(total + 2, generator=g, device=DEV)
    cache = torch.zeros(total + 2, 1, page, W, dtype=torch.bfloat16, device=DEV)
    stride = max(-(-n // page) for n in lens) + 1
    pages = torch.zeros(len(lens), stride, dtype=torch.int32, device=DEV)
    keys, at = [], 0
    for b, n in enumerate(lens):
        k = torch.randn(n, W, generator=g, device=DEV).bfloat16()
        keys.append(k)
        for i in range(-(-n // page)):
            pages[b, i] = order[at]
            part = k[i * page:(i + 1) * page]
            cache[order[at], 0, :len(part)] = part
            at += 1
    T = sum(qlens)
    q = torch.randn(T, H * W, generator=g, device=DEV) * (2.0 / W ** 0.5)
    sink = torch.randn(H, generator=g, device=DEV) if sunk else None
    start = [sum(qlens[:i]) for i in range(len(qlens) + 1)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(n_seqs=len(lens), n_tokens=T, max_q_len=max(qlens), seq_start=i32(start), seq_pos0=i32(pos0))
    out = torch.full((T, H * rank), 9.0, device=DEV)
    assert ops.latent_prefill_tc_ok(q, out, cache, H, rank, rot, page, batch)
    tok_seq = i32(sum(([b] * n for b, n in enumerate(qlens)), []))
    tok_pos = i32(sum((list(range(p, p + n)) for p, n in zip(pos0, qlens)), []))
    ops.latent_attention(q, out, cache, sink, tok_seq, tok_pos, pages, H, rank, rot, page, window, batch=batch)
    ops.check_kernel_errors()
    for b, n in enumerate(qlens):
        k = keys[b].double()
        qb = q[start[b]:start[b + 1]].bfloat16().double().view(n, H, W)
        s = torch.einsum("thw,jw->thj", qb, k)
        pos = torch.arange(pos0[b], pos0[b] + n, device=DEV)[:, None]
        j = torch.arange(lens[b], device=DEV)[None]
        seen = (j <= pos) & (j > pos - window if window else torch.ones_like(j, dtype=torch.bool))
        s = s.masked_fill(~seen[:, None], float("-inf"))
        if sunk:
            s = torch.cat([s, sink.double()[None, :, None].expand(n, H, 1)], -1)
        p = torch.softmax(s, -1)[..., :lens[b]]
        ref = torch.einsum("thj,jr->thr", p, k[:, :rank])
        got = out[start[b]:start[b + 1]].view(n, H, rank).double()
        # weights are rounded to bfloat16 (2^-8 of each) before their product with the values, and so in their sum
        bound = torch.einsum("thj,jr->thr", p, k[:, :rank].abs()) * 2.0 ** -7 + 1e-5
        assert ((got - ref).abs() <= bound).all(), (b, float((got - ref).abs().max()))


def test_small_steps_and_odd_pages_keep_their_kernels():
    b = SimpleNamespace(n_seqs=1, max_q_len=600)
    for page, n, want in ((64, 600, True), (64, 590, False), (48, 600, False), (32, 600, False)):
        cache = torch.zeros(4, 1, page, 576, dtype=torch.bfloat16, device=DEV)
        q, out = torch.zeros(n, 16 * 576, device=DEV), torch.zeros(n, 16 * 512, device=DEV)
        assert ops.latent_prefill_tc_ok(q, out, cache, 16, 512, 64, page, b) == want
    assert not ops.latent_prefill_tc_ok(q, out, cache.float(), 16, 512, 64, 64, b)


def test_many_short_sequences_keep_the_kernel_of_short_tiles():
    for H, rank, n, per, want in ((16, 512, 1200, 1, False), (16, 512, 600, 2, False), (16, 512, 400, 3, True), (16, 256, 1200, 1, True),
                                  (40, 320, 300, 1, True)):
        cache = torch.zeros(4, 1, 64, rank + 64, dtype=torch.bfloat16, device=DEV)
        q, out = torch.empty(n * per, H * (rank + 64), device=DEV), torch.empty(n * per, H * rank, device=DEV)
        b = SimpleNamespace(n_seqs=n, max_q_len=per)
        assert ops.latent_prefill_tc_ok(q, out, cache, H, rank, 64, 64, b) == want


@pytest.mark.parametrize("H,rank,rot", [(16, 512, 64), (16, 256, 32)])
def test_pages_that_held_something_before(H, rank, rot):
    """Rows of a sequence's last page behind its last key hold another sequence's numbers: they do not count, whatever they are."""
    page, W, n = 64, rank + rot, 1300
    g = torch.Generator(device=DEV).manual_seed(H + rank)
    cache = torch.randn(24, 1, page, W, generator=g, device=DEV).bfloat16()
    q = torch.randn(n, H * W, generator=g, device=DEV) * (2.0 / W ** 0.5)
    pages = torch.randperm(24, generator=g, device=DEV)[:21].int().view(1, 21).contiguous()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(n_seqs=1, n_tokens=n, max_q_len=n, seq_start=i32([0, n]), seq_pos0=i32([0]))
    tok_seq, tok_pos = torch.zeros(n, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV)
    outs = []
    for behind in (None, 0.0, 3.0e38, -3.0e38):
        c = cache.clone()
        if behind is not None:
            c[pages[0, 20].long(), 0, n - 20 * page:] = behind
        out = torch.full((n, H * rank), 9.0, device=DEV)
        assert ops.latent_prefill_tc_ok(q, out, c, H, rank, rot, page, batch)
        ops.latent_attention(q, out, c, None, tok_seq, tok_pos, pages, H, rank, rot, page, None, batch=batch)
        outs.append(out)
    ops.check_kernel_errors()
    assert all(torch.equal(outs[0], o) for o in outs[1:])


@pytest.mark.parametrize("H,rank,rot,below,above", [(16, 512, 64, 591, 592), (16, 256, 32, 1183, 1184)])
def test_a_prompt_on_both_sides_of_the_rule(H, rank, rot, below, above):
    """One token less than gives every SM a tile, and that many: the other kernel, the same numbers up to rounding."""
    page, W = 64, rank + rot
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the token counts are those of 148 SMs")
    g = torch.Generator(device=DEV).manual_seed(H + rank)
    per = -(-above // page)
    cache = torch.randn(per, 1, page, W, generator=g, device=DEV).bfloat16()
    pages = torch.arange(per, dtype=torch.int32, device=DEV).view(1, per)
    q = torch.randn(above, H * W, generator=g, device=DEV) * (2.0 / W ** 0.5)
    outs = []
    for n in (below, above):
        batch = SimpleNamespace(n_seqs=1, n_tokens=n, max_q_len=n, seq_start=torch.tensor([0, n], dtype=torch.int32, device=DEV),
                                seq_pos0=torch.zeros(1, dtype=torch.int32, device=DEV))
        out = torch.full((n, H * rank), 9.0, device=DEV)
        assert ops.latent_prefill_tc_ok(q[:n], out, cache, H, rank, rot, page, batch) == (n == above)
        ops.latent_attention(q[:n], out, cache, None, torch.zeros(n, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV),
                             pages, H, rank, rot, page, None, batch=batch, scratch=lambda s, dt: torch.empty(s, dtype=dt, device=DEV))
        outs.append(out[:below].view(below, H, rank).double())
    ops.check_kernel_errors()
    p = torch.softmax(torch.einsum("thw,jw->thj", q[:below].bfloat16().double().view(below, H, W), cache.view(-1, W)[:below].double())
                      .masked_fill(torch.ones(below, below, dtype=torch.bool, device=DEV).triu(1)[:, None], float("-inf")), -1)
    # both round the softmax weights to bfloat16 (2^-8 of each), each at its own scale
    bound = torch.einsum("thj,jr->thr", p, cache.view(-1, W)[:below, :rank].double().abs()) * 2.0 ** -7 + 1e-5
    assert ((outs[0] - outs[1]).abs() <= bound).all()


@pytest.mark.parametrize("halves", [True, False])
@pytest.mark.parametrize("rank,rot", [(512, 64), (40, 6), (64, 80)])
def test_the_rotated_key_rounds_its_second_product_first(rank, rot, halves):
    """u c - v s and v c + u s with the product of s rounded and the other one taken exactly (a multiply-add): the same bits however the
    kernel around is written.  float64 holds the exact product and the sum closely enough to be rounded once to float, but for ties
    at its 53rd bit: none in these numbers."""
    T, page, P = 500, 64, 8
    g = torch.Generator(DEV).manual_seed(rot)
    kv = torch.randn(T, rank + rot, device=DEV, generator=g)
    freq = (10000.0 ** (-torch.arange(rot // 2, dtype=torch.float64) * 2 / rot)).float().to(DEV)
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    cache = torch.zeros(P, 1, page, rank + rot, device=DEV)
    mscale = 1.25
    ops.latent_kv_store(kv, torch.ones(rank, device=DEV), 1e-6, freq, mscale, rank, rot, torch.zeros_like(pos), pos,
                        torch.arange(P, dtype=torch.int32, device=DEV).view(1, P), cache, page, halves=halves)
    ang = pos.float()[:, None] * freq
    s, c = torch.sin(ang) * mscale, torch.cos(ang) * mscale
    r = kv[:, rank:]
    u, v = (r[:, :rot // 2], r[:, rot // 2:]) if halves else (r[:, 0::2], r[:, 1::2])
    got = cache.view(-1, rank + rot)[:T, rank:]
    a, b = (got[:, :rot // 2], got[:, rot // 2:]) if halves else (got[:, 0::2], got[:, 1::2])
    assert torch.equal(a, (u.double() * c.double() - (v * s).double()).float())
    assert torch.equal(b, (v.double() * c.double() + (u * s).double()).float())
