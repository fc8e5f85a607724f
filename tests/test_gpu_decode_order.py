"""Decode attention of many sequences with one key range each: the longest are taken first.  The order must change nothing: the same
bits as the same sequences in batches too small to be ordered."""
import pytest
import torch

from herbert_rs_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [17, 64, 128, 129])
@pytest.mark.parametrize("nh,nkv", [(4, 2), (18, 2)])
def test_the_order_changes_nothing(n, nh, nkv):
    g = torch.Generator().manual_seed(n)
    page, hd = 64, 128
    lens = torch.randint(1, 400, (n,), generator=g)
    lens[1::5] = lens[0]                                    # equal lengths too
    P = 7
    table = torch.randperm(n * P, generator=g).view(n, P).int().cuda()
    kc, vc = (torch.randn(n * P, nkv, page, hd, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    q = torch.randn(n, nh * hd, generator=g).to(torch.bfloat16).cuda()
    seq_len = lens.int().cuda()

    def run(a, b):
        out = torch.full((b - a, nh * hd), float("nan"), device="cuda", dtype=torch.bfloat16)
        scratch = torch.empty(ops.attention_decode_scratch_floats(b - a, nh, hd, 1), device="cuda")
        ops.attention_decode(q[a:b], q.stride(0), out, kc, vc, seq_len[a:b].contiguous(), table[a:b], scratch, nh, nkv, hd, page, 1, hd ** -0.5, None)
        return out

    whole = run(0, n)
    assert torch.equal(whole, torch.cat([run(a, min(a + 16, n)) for a in range(0, n, 16)]))
    assert torch.isfinite(whole).all()


@pytest.mark.parametrize("n", [5, 16, 17, 128])
@pytest.mark.parametrize("nh,nkv", [(32, 32), (288, 32)])
@pytest.mark.parametrize("longest", [200, 1500])
def test_few_sequences_of_many_heads_and_short_ones(n, nh, nkv, longest):
    """More CTAs than SMs at few sequences too; with `longest` 200 nothing is ranked.  Four sequences at a time stay in their order."""
    g = torch.Generator().manual_seed(n)
    page, hd, P = 64, 128, 24
    lens = torch.randint(1, longest + 1, (n,), generator=g)
    lens[1::5] = lens[0]
    table = torch.randint(0, 300, (n, P), generator=g).int().cuda()
    kc, vc = (torch.randn(300, nkv, page, hd, device="cuda").to(torch.bfloat16) for _ in range(2))
    q = torch.randn(n, nh * hd, device="cuda").to(torch.bfloat16)
    seq_len = lens.int().cuda()

    def run(a, b):
        out = torch.full((b - a, nh * hd), float("nan"), device="cuda", dtype=torch.bfloat16)
        scratch = torch.empty(ops.attention_decode_scratch_floats(b - a, nh, hd, 1), device="cuda")
        ops.attention_decode(q[a:b], q.stride(0), out, kc, vc, seq_len[a:b].contiguous(), table[a:b], scratch, nh, nkv, hd, page, 1, hd ** -0.5, None)
        return out

    whole = run(0, n)
    assert torch.equal(whole, torch.cat([run(a, min(a + 4, n)) for a in range(0, n, 4)])) and torch.isfinite(whole).all()
