"""The recurrences over a state per head against a float64 restatement, at the sizes of their register tiles, chunks and columns."""
from types import SimpleNamespace

import pytest
import torch

from herbert_rs_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _batch(lens):
    start = [0]
    for n in lens:
        start.append(start[-1] + n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    return SimpleNamespace(seq_slot=i32([len(lens) - i for i in range(len(lens))]), seq_start=i32(start), n_seqs=len(lens), max_q_len=max(lens),
                           n_tokens=start[-1])


def _check(kind, lens, H, G, dk, dv):
    g = torch.Generator(device=DEV).manual_seed(dk + dv + H + len(lens))
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    uni = lambda *s: torch.rand(*s, generator=g, device=DEV)
    b = _batch(lens)
    T = b.n_tokens
    unit = lambda x: torch.nn.functional.normalize(x, dim=-1)
    q, k, v = rnd(T, G, dk) / dk ** 0.5, unit(rnd(T, G, dk)), rnd(T, H, dv)
    state = rnd(len(lens) + 1, H, dk, dv) * 0.3
    start = state.clone()
    out = torch.full((T, H * dv), 9.0, device=DEV)
    rep = lambda x: x.double().repeat_interleave(H // G, 1)
    a = d = gates = w = u = p = None
    if kind == "gla":
        a = uni(T, H, dk) * 0.3 + 0.7
        pad = (-H * dv) % 4
        proj = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1), torch.zeros(T, pad, device=DEV)], 1).contiguous()
        ops.gla_scan(proj, 0, H * dk, 2 * H * dk, a.reshape(T, -1).contiguous(), state, b.seq_slot, b.seq_start, out, b.n_seqs, H, dk, dv, 0.5)
    elif kind == "general":
        w, u = uni(T, H, dk) * 0.3 + 0.7, k
        p = u * uni(T, H, dk)
        k = rnd(T, H, dk) / dk ** 0.5
        prep = torch.stack([q, k, w, u, p], 2).contiguous()
        ops.general_delta_scan(prep, v.reshape(T, -1), state, b, out, H, dk, dv)
    else:
        d = uni(H) * 0.2 + 0.8
        gates = uni(T, 2, H) * 0.5 + 0.5
        ops.linear_scan(q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1), state, b, out, H, G, dk, dv,
                        gates=gates.reshape(T, -1).contiguous() if kind == "delta" else None, decay=d if kind == "decay" else None)
    qd, kd, vd = rep(q), rep(k), v.double()
    ref = torch.empty(T, H, dv, dtype=torch.float64, device=DEV)
    t = 0
    for i, n in enumerate(lens):
        slot = len(lens) - i
        S = start[slot].double()
        for _ in range(n):
            if kind == "gla":
                S = S * a[t].double()[:, :, None] + kd[t][:, :, None] * vd[t][:, None]
            elif kind == "decay":
                S = S * d.double()[:, None, None] + kd[t][:, :, None] * vd[t][:, None]
            elif kind == "delta":
                S = S * gates[t, 0].double()[:, None, None]
                S = S + kd[t][:, :, None] * (gates[t, 1].double()[:, None] * (vd[t] - torch.einsum("hkv,hk->hv", S, kd[t])))[:, None]
            else:
                seen = torch.einsum("hkv,hk->hv", S, u[t].double())
                S = S * w[t].double()[:, :, None] - p[t].double()[:, :, None] * seen[:, None] + kd[t][:, :, None] * vd[t][:, None]
            ref[t] = torch.einsum("hkv,hk->hv", S, qd[t]) * (0.5 if kind == "gla" else 1.0)
            t += 1
        # float rounding of a decaying recurrence of unit-sized numbers: a few 2^-24 of them per step of the memory's length
        assert float((state[slot].double() - S).abs().max()) <= 1e-5 * max(1.0, float(S.abs().max()))
    assert float((out.view(T, H, dv).double() - ref).abs().max()) <= 1e-5 * max(1.0, float(ref.abs().max()))
    assert torch.equal(state[0], start[0])


@pytest.mark.parametrize("kind", ["gla", "decay", "delta", "general"])
@pytest.mark.parametrize("dk", [64, 128, 256, 60])
@pytest.mark.parametrize("lens,H,G,dv", [([1, 1], 2, 1, 36), ([7, 8, 9, 1], 3, 3, 4), ([17], 16, 8, 128), ([33, 1, 16], 8, 4, 260), ([5] * 40, 4, 4, 132), ([3], 2, 2, 33)])
def test_scan_rows(kind, dk, lens, H, G, dv):
    _check(kind, lens, H, H if kind in ("gla", "general") else G, dk, dv)


@pytest.mark.parametrize("kind", ["gla", "decay", "delta", "general"])
@pytest.mark.parametrize("dk", [64, 128, 256])
@pytest.mark.parametrize("shape", ["many", "few"])
def test_scan_rows_over_several_chunks(kind, dk, shape):
    """Sequences of several chunks and a rest, four columns a thread (many CTAs) and two (about one an SM)."""
    if shape == "many":
        _check(kind, [33, 80, 97, 64, 65] * 5, 4, 4, dk, 260)
    else:
        _check(kind, [70, 65, 64], 16, 16 if kind in ("gla", "general") else 8, dk, (8448 // dk + 3) // 4 * 4)


@pytest.mark.parametrize("dk", [64, 128, 256])
@pytest.mark.parametrize("less", [0, 1])
def test_gla_scan_around_the_length_where_its_kernel_changes(dk, less):
    """As many tokens a sequence on average as the rule asks for, and one token less."""
    n = 64 if dk > 128 else 16
    _check("gla", [n + 3, n - 3, n, n - less, 2 * n - 1, 1] * 2, 8, 8, dk, 132)
