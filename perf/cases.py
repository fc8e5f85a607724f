"""Measured workloads of the engine: prompts, decode steps and whole turns through `Engine.step`.

A case names a model (the dense decoder or one of the other designs, at the layer sizes that bench.py
uses), a storage type, a batch of sequences of unequal length, and what one pass does with them:

  prompt   the whole prompts of new sequences in one step, logits at every last token
  decode   `steps` steps of one token per sequence on top of contexts that are already cached;
           the sequences are cut back to their contexts afterwards (`Engine.truncate`)
  turn     the prompts and then `steps` decode steps, as one answer of a chat does it (models with
           recurrent state cannot be cut back, so they are measured by whole turns)

The tokens of every step are given (teacher forcing), so a pass's logits do not hang on near ties of the
ones before it.  Weights and tokens are random and come from the seed.  `exact` restates every design in
64 bits with plain torch operations: whole sequences, no cache, no batching.
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

import herbert_rs_b200 as hb
from herbert_rs_b200.sampling import device_choose
from herbert_rs_b200.weights.loader import build_model, fill_model
from herbert_rs_b200.weights.random_init import random_tensor

DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
#: the command line's defaults
SAMPLING = hb.SamplingParams(temperature=0.4, top_k=40, top_p=0.9)


# ---- models ---------------------------------------------------------------------------------------
def config_of(case: dict) -> dict:
    """The model's config.json.  `size` "0.6b" and "8b" are the dense decoder's published layer sizes;
    "1k" and "2k" the other designs' sizes of that width with four layers."""
    model, size = case["model"], case["size"]
    if model == "qwen3":
        c = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=151936, hidden_size=4096, num_hidden_layers=36,
                 num_attention_heads=32, num_key_value_heads=8, head_dim=128, intermediate_size=12288, rope_theta=1000000.0,
                 rms_norm_eps=1e-6, max_position_embeddings=40960, tie_word_embeddings=False, eos_token_id=151645)
        if size == "0.6b":
            c.update(hidden_size=1024, num_hidden_layers=28, num_attention_heads=16, intermediate_size=3072, tie_word_embeddings=True)
        if case.get("layers"):
            c["num_hidden_layers"] = case["layers"]
        return c
    big = size == "2k"
    width, ff, vocab = (2048, 8192, 32000) if big else (1024, 3072, 32000)
    heads, kv, eps = (16, 8, 1e-6) if big else (8, 4, 1e-6)
    experts, top, expert_ff, shared_ff = (32, 4, 1408, 2560) if big else (16, 2, 768, 1536)
    groups = {"count": 8, "keep": 4} if big else {"count": 4, "keep": 2}
    norm, dense = {"eps": eps}, {"kind": "dense", "ff": ff}
    moe = {"kind": "moe", "expert": {"ff": expert_ff}, "router": {"experts": experts, "top": top}}

    def layers(*kinds):
        return [{"type": t, "mixer": m, "mlp": f} for t, m, f in kinds]
    if model == "kebisun":
        dim, rot, rank, q_rank, dk, dv = (128, 64, 512, 768, 256, 512) if big else (64, 32, 256, 384, 128, 256)
        latent = {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": dim, "kv_rank": rank, "q_rank": q_rank, "scale": (dim + rot) ** -0.5,
                  "mask": {"size": 4096},
                  "rot": {"base": 10000.0, "dims": rot, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
        gla = {"heads": 4, "dim": dk, "vdim": dv, "tau": 16.0, "decay_rank": 32}
        return {"architecture": "Kebisun", "vocab": vocab, "width": width, "embedding": {"scale": 1.0}, "norm": norm,
                "layers": layers(("latent_attention", latent, dense), ("gla", gla, moe), ("latent_attention", latent, moe), ("gla", gla, dense))}
    if model == "votapel":
        h, g, dim = (16, 8, 128) if big else (16, 8, 64)
        att = {"heads": h, "kv_heads": g, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 30.0, "q_temp": {"coef": 0.1, "every": 1024}}
        f = dict(moe, shared={"ff": shared_ff}, router=dict(moe["router"], scale=1.0, groups=groups))
        return {"architecture": "Votapel", "vocab": vocab, "width": width, "max_positions": 8192, "norm": norm, "residual_mult": 0.5,
                "layers": layers(*[("attention", att, f)] * 4)}
    if model == "begupel":
        lightning = {"heads": heads, "dim": 128, "vdim": 128,
                     "decay": [round(1.0 - 2.0 ** -(5 + 3 * i / (heads - 1)), 6) for i in range(heads)]}
        left = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 4096},
                "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 4.0}}}
        right = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "conv": 4}
        side = {"left": left, "right": right, "left_scale": 0.5, "right_scale": 0.5}
        return {"architecture": "Begupel", "vocab": vocab, "width": width, "norm": {"eps": eps, "groups": 4}, "canon": {"taps": 4},
                "logit_softcap": 30.0, "embedding": {"bigram": {"buckets": 65536, "mul_prev": 1000003, "mul_cur": 31}},
                "layers": layers(*[("lightning", lightning, dense), ("parallel", side, dense)] * 2)}
    if model == "nefivik":
        att = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 4096}, "conv": 4,
               "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
        delta = {"heads": heads, "dim": 128}
        f = dict(moe, expert={"ff": expert_ff, "limit": 7.0}, router=dict(moe["router"], groups=groups))
        return {"architecture": "Nefivik", "vocab": vocab, "width": width, "norm": norm, "token_side": {"dim": 128 if big else 64},
                "layers": layers(("attention", att, f), ("general_delta", delta, f), ("attention", dict(att, kv_from=0), f),
                                 ("general_delta", delta, f))}
    if model == "putazen":
        dim, rot, rank = (128, 64, 512) if big else (64, 32, 256)
        att = {"heads": heads, "kv_heads": kv, "dim": 64, "vdim": 128, "scale": 0.125, "diff": 0.35,
               "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
        latent = {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": dim, "kv_rank": rank, "scale": (dim + rot) ** -0.5,
                  "rot": {"base": 10000.0, "dims": rot}}
        scan = {"heads": 4 * heads, "vdim": 64, "state": 128, "groups": 4 if big else 2, "norm_groups": 4 if big else 2, "conv": 4}
        f = dict(dense, limit=7.0)
        return {"architecture": "Putazen", "vocab": vocab, "width": width, "embedding": {"scale": 1.0}, "norm": norm, "streams": 4,
                "layers": layers(("attention", att, f), ("mamba2", scan, f), ("latent_attention", latent, f), ("mamba2", scan, f))}
    if model == "muzasun":
        att = {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "v_mix": True, "rot": {"base": 10000.0, "dims": 128}}
        memory = {"heads": heads, "dim": 128, "vdim": 256, "gate_cap": 20.0}
        delta = {"heads": heads, "kv_heads": heads, "dim": 128, "vdim": 128, "conv": 4, "low_rank": 128 if big else 64}
        f = dict(moe, shared={"ff": shared_ff})
        return {"architecture": "Muzasun", "vocab": vocab, "width": width, "norm": norm, "residual_mult": 0.5, "logit_scale": 1.0,
                "layers": layers(("mlstm", memory, dense), ("attention", att, f), ("channel_delta", delta, dense), ("attention", att, f))}
    raise ValueError(model)


#: How strongly a token's embedding points at its experts, beside what the layers add to the stream.
DECIDED = {"kebisun": 24.0, "nefivik": 32.0, "votapel": 10.0, "muzasun": 8.0}


def tensor_of(case: dict, name: str, ps, seed: int) -> torch.Tensor:
    """A tensor of the model: random, but for the mixtures.  A trained router's choices hang on the token and are
    clear; with a random one the last expert chosen and the first left out are often so close that the rounding of
    an activation swaps them, and outputs then differ by a whole expert.  So here every token has its experts (as
    many as are chosen, at random): its embedding holds their router rows, and all layers share the rows."""
    if name.endswith((".hc1.mix", ".hc2.mix")):
        # every copy of the stream mostly keeps itself: random mixing alone would make copies that nearly cancel
        return random_tensor(name, ps, seed, "cuda") + torch.eye(ps.shape[0], dtype=torch.bfloat16, device="cuda")
    if name.endswith("mix.i.b"):
        # the matrix memory's input gates start nearly closed, as trained ones do: wide open ones leave read-outs
        # whose denominator passes near zero, which no 16-bit input can decide
        return random_tensor(name, ps, seed, "cuda") - 3.0
    if not name.endswith("mlp.router") and not (name == "embed" and case["model"] in DECIDED):
        return random_tensor(name, ps, seed, "cuda")
    r = next(layer["mlp"]["router"] for layer in config_of(case)["layers"] if "router" in layer["mlp"])
    width = ps.shape[1]
    router = random_tensor("router", type(ps)((r["experts"], width), "matrix", "normal"), seed, "cuda")
    if name != "embed":
        return router
    gen = torch.Generator("cuda").manual_seed(seed)
    # neighbours two by two, so that their groups, rated by their two best or their best, are clear as well
    pairs = torch.rand(ps.shape[0], r["experts"] // 2, generator=gen, device="cuda").topk(r["top"] // 2, -1).indices
    theirs = torch.cat([2 * pairs, 2 * pairs + 1], -1)
    pull = torch.zeros(ps.shape[0], r["experts"], device="cuda").scatter_(
        1, theirs, torch.linspace(1.0, 0.7, r["top"], device="cuda").expand(ps.shape[0], -1))
    rows = torch.nn.functional.normalize(router.float(), dim=-1)
    return (random_tensor(name, ps, seed, "cuda").float() + DECIDED[case["model"]] * (pull @ rows)).to(torch.bfloat16)


def lengths_of(case: dict) -> list:
    """Tokens of each sequence's prompt or context: `longest` once, the others spread over [shortest, longest]."""
    lo, hi, n = case["shortest"], case["longest"], case["batch"]
    r = random.Random(f"{lo} {hi} {n}")
    return [hi] + [int(round(math.exp(r.uniform(math.log(lo), math.log(hi))))) for _ in range(n - 1)]


def tokens_of(case: dict, seed: int):
    """(prompts, one list of `steps` tokens per sequence, uniforms [passes, batch] for sampling)."""
    rng = np.random.default_rng([seed, 1])
    vocab = config_of(case).get("vocab_size") or config_of(case)["vocab"]
    prompts = [rng.integers(0, vocab, n).tolist() for n in lengths_of(case)]
    after = [rng.integers(0, vocab, case["steps"]).tolist() for _ in prompts]
    return prompts, after, rng.random((case["steps"] + 1, len(prompts)), dtype=np.float32)


# ---- the cases ------------------------------------------------------------------------------------
def _case(name, model, size, what, batch, shortest, longest, steps=0, dtype="bfloat16", layers=0, sampled=False):
    return dict(name=name, model=model, size=size, what=what, batch=batch, shortest=shortest, longest=longest, steps=steps,
                dtype=dtype, layers=layers, sampled=sampled)


#: Layers of the 8B-sized dense decoder here: each has the full sizes and the vocabulary is whole; fewer of
#: them than the 36, so that the 64-bit restatement of a batch ends in seconds and bfloat16's own error, which
#: grows with depth on random weights, stays well inside what can be told from a mistake.
LAYERS_8B = 8


def listed() -> list:
    return [
        # one user's chat at the smallest published size: every launch and every host microsecond counts
        _case("0.6b decode b1", "qwen3", "0.6b", "decode", 1, 1283, 1283, steps=2),
        # a server's admission step: sixteen waiting prompts of 32 to 1,024 tokens together
        _case("0.6b prompts b16", "qwen3", "0.6b", "prompt", 16, 32, 1024),
        # the true 32-bit path: a few short prompts, answered with the command line's default sampling
        _case("0.6b float32 turn b3", "qwen3", "0.6b", "turn", 3, 20, 150, steps=3, dtype="float32", sampled=True),
        # the headline benchmark's decode: eight sequences behind prompts of 2,048 tokens
        _case("8b decode b8", "qwen3", "8b", "decode", 8, 2048, 2048, steps=4, layers=LAYERS_8B),
        # a loaded server: 64 sequences at unequal contexts
        _case("8b decode b64", "qwen3", "8b", "decode", 64, 200, 2000, steps=2, layers=LAYERS_8B),
        # the headline benchmark's prefill: one long prompt
        _case("8b prompt 2048", "qwen3", "8b", "prompt", 1, 2048, 2048, layers=LAYERS_8B),
        # one turn of each other design: unequal prompts, then an answer's first tokens.  A single long prompt,
        # small batches and larger ones take turns over the designs
        _case("kebisun turn b4", "kebisun", "2k", "turn", 4, 300, 1500, steps=8),
        _case("votapel turn b8", "votapel", "2k", "turn", 8, 100, 1000, steps=8),
        _case("begupel turn b1", "begupel", "2k", "turn", 1, 2048, 2048, steps=16),
        _case("nefivik turn b2", "nefivik", "2k", "turn", 2, 700, 1301, steps=12),
        _case("putazen turn b4", "putazen", "2k", "turn", 4, 200, 2000, steps=8),
        _case("muzasun turn b16", "muzasun", "2k", "turn", 16, 37, 600, steps=8),
    ]


def _log_uniform(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """Another case of the same ranges: batches of 1 to 64, sequences of 16 to 2,048 tokens, every design at
    both sizes, prompts, decode steps and turns."""
    model = rng.choice(["qwen3", "qwen3", "qwen3", "qwen3", "kebisun", "votapel", "begupel", "nefivik", "putazen", "muzasun"])
    layers, dtype, sampled = 0, "bfloat16", False
    if model == "qwen3":
        size = rng.choice(["0.6b", "8b"])
        layers = LAYERS_8B if size == "8b" else 0
        what = rng.choice(["decode", "decode", "prompt", "turn"])
        if size == "0.6b" and rng.random() < 0.2:
            what, dtype, sampled = "turn", "float32", True
    else:
        size, what = rng.choice(["1k", "2k"]), "turn"
    # tokens in all sequences together, so that no drawn case costs more than the largest listed one
    most = 450 if dtype == "float32" else 49152 if what == "decode" else 2048 if size == "8b" else 6144
    batch = _log_uniform(rng, 1, 3 if dtype == "float32" else 64 if what == "decode" else 16)
    longest = _log_uniform(rng, 16, min(2048, 150 if dtype == "float32" else max(16, most // batch)))
    shortest = max(1, int(longest * rng.choice([1.0, 0.5, 0.1])))
    steps = 0 if what == "prompt" else rng.randint(1, 4 if what == "decode" or dtype == "float32" else 12)
    c = _case("", model, size, what, batch, shortest, longest, steps, dtype, layers, sampled)
    del c["name"]
    return c


# ---- a pass ---------------------------------------------------------------------------------------
def prepare(case: dict, seed: int) -> dict:
    """An engine over a model with random weights, the step's tokens, and for `decode` the contexts in the cache."""
    prompts, after, uniforms = tokens_of(case, seed)
    rt = hb.Runtime("cuda", DTYPES[case["dtype"]])
    room = sum(hb.Engine.pages_for(len(p) + case["steps"] + 1) for p in prompts) * rt.page_size
    model = build_model(config_of(case), rt)
    specs = model.param_specs()
    fill_model(model, lambda name: tensor_of(case, name, specs[name], seed), rt)
    engine = hb.Engine(model, max_tokens=room, max_slots=len(prompts))
    state = {"what": case["what"], "engine": engine, "prompts": prompts, "steps": [list(t) for t in zip(*after)], "slots": None, "uniforms": None}
    if case["sampled"]:
        state["uniforms"] = torch.from_numpy(uniforms).cuda()
    if case["what"] == "decode":
        state["slots"] = [engine.alloc_slot() for _ in prompts]
        at = 0
        while at < len(prompts):        # a few sequences at a time: up to 8,192 tokens a step, or one sequence
            stop, n = at + 1, len(prompts[at])
            while stop < len(prompts) and n + len(prompts[stop]) <= 8192:
                n += len(prompts[stop])
                stop += 1
            engine.step(list(zip(state["slots"][at:stop], prompts[at:stop])), None)
            at = stop
    return state


def run(state: dict) -> dict:
    """One pass: the logits of every step in order, and where the case samples the chosen tokens."""
    engine, prompts, slots = state["engine"], state["prompts"], state["slots"]
    logits, tokens = [], []

    def step(entries):
        z = engine.step(entries, "last")
        if state["uniforms"] is not None:
            out = torch.empty(len(entries), dtype=torch.int32, device=z.device)
            device_choose(z, SAMPLING, state["uniforms"][len(tokens)], out)
            tokens.append(out)
        # the engine's own buffer: the next step overwrites it
        logits.append(z.clone() if state["steps"] else z)

    new = slots is None
    if new:
        slots = [engine.alloc_slot() for _ in prompts]
        step(list(zip(slots, prompts)))
    for given in state["steps"]:
        step([(s, [t]) for s, t in zip(slots, given)])
    for s, p in zip(slots, prompts):
        if new:
            engine.free_slot(s)
        else:
            engine.truncate(s, len(p))
    return {"logits": logits, "tokens": tokens}


def tolerance(case: dict) -> dict:
    """Against `exact` the bfloat16 cases measure 0.004 to 0.009, the 8B-sized ones 0.016 (their streams grow with
    depth), and the 32-bit ones 2.2e-6; two correct ways to the same logits differ by about as much as one does."""
    return {"rel": 0.03, "max": 0.4} if case["dtype"] == "bfloat16" else {"rel": 1e-5, "max": 2e-4, "differ": 0.01}


# ---- what a pass cannot do without ------------------------------------------------------------------
def _specs(case: dict) -> dict:
    return build_model(config_of(case), hb.Runtime("cpu", torch.bfloat16)).param_specs()


def _mixers(cfg: dict) -> list:
    """Per layer: (attention or None, state or None): attention = (heads, key channels, value channels, cached
    numbers per token, window), state = (entries, operations per entry and token)."""
    if "hidden_size" in cfg:
        h, g, d = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
        return [((h, d, d, 2 * g * d, None), None)] * cfg["num_hidden_layers"]
    out = []
    for layer in cfg["layers"]:
        m, t = layer["mixer"], layer["type"]
        att, state = None, None
        if t == "parallel":
            r = m["right"]
            state = (r["heads"] * r["dim"] * r["vdim"], 7)
            m, t = m["left"], "attention"
        if t == "attention":
            maps = 2 if "diff" in m else 1
            planes = m["kv_heads"] * (maps * m["dim"] + (0 if cfg["architecture"] == "Votapel" else m["vdim"]))
            att = (m["heads"] * maps, m["dim"], m["vdim"], 0 if "kv_from" in m else planes, (m.get("mask") or {}).get("size"))
        elif t == "latent_attention":
            att = (m["heads"], m["kv_rank"] + m["rot_dim"], m["kv_rank"], m["kv_rank"] + m["rot_dim"], (m.get("mask") or {}).get("size"))
        elif t == "mamba2":
            state = (m["heads"] * m["state"] * m["vdim"], 5)
        else:
            ops = {"gla": 5, "lightning": 5, "general_delta": 9, "mlstm": 6, "channel_delta": 7}[t]
            state = (m["heads"] * m["dim"] * m.get("vdim", m["dim"]), ops)
        out.append((att, state))
    return out


_TABLES = ("embed", "pos", "bigram", "side.embed", "model.embed_tokens.weight")


def work(case: dict) -> dict:
    """Bytes: every step reads the weights it multiplies with (of a mixture the experts that its tokens are
    expected to choose), the cached keys and values and the recurrent state once, and writes its logits.
    Operations: two per weight and token, the scores and sums of attention, the state updates."""
    cfg, specs = config_of(case), _specs(case)
    es = 2 if case["dtype"] == "bfloat16" else 4
    lens, vocab = lengths_of(case), cfg.get("vocab_size") or cfg["vocab"]
    width = cfg.get("hidden_size") or cfg["width"]
    passes = ([[(0, n) for n in lens]] if case["what"] != "decode" else []) + [[(n + i, 1) for n in lens] for i in range(case["steps"])]
    experts = [layer["mlp"]["router"] for layer in cfg.get("layers", []) if (layer.get("mlp") or {}).get("kind") == "moe"]
    share, spared = (experts[0]["top"] / experts[0]["experts"], 1 - experts[0]["top"] / experts[0]["experts"]) if experts else (1.0, 0.0)
    dense = routed = 0
    for name, ps in specs.items():
        n = math.prod(ps.shape)
        if name in _TABLES or name in ("head", "lm_head.weight"):
            continue
        if ".mlp.e" in name:
            routed += n
        else:
            dense += n
    total_bytes = total_flops = 0.0
    for entries in passes:
        tokens, rows = sum(n for _, n in entries), len(entries)
        total_bytes += es * (dense + routed * (1 - spared ** tokens) + vocab * width + 2 * tokens * width) + 4 * rows * vocab
        total_flops += 2.0 * (tokens * (dense + routed * share) + rows * vocab * width)
        for att, state in _mixers(cfg):
            if att:
                h, dk, dv, cached, window = att
                for past, n in entries:
                    pairs = n * past + n * (n + 1) / 2
                    if window and past + n > window:
                        pairs = min(pairs, n * window)
                    total_flops += 2.0 * pairs * h * (dk + dv)
                    total_bytes += es * cached * (min(past, window or past) + n)
            if state:
                total_flops += float(state[0]) * state[1] * tokens
                total_bytes += 4 * state[0] * sum(2 if past else 1 for past, _ in entries)
    return {"bytes": total_bytes, "flops": total_flops}


# ---- the designs in 64 bits -------------------------------------------------------------------------
class _Weights:
    """The model's random tensors by name, made when asked for, in 64 bits; `at(prefix)` shortens the names."""

    def __init__(self, case, specs, seed, prefix=""):
        self.case, self.specs, self.seed, self.prefix = case, specs, seed, prefix

    def at(self, prefix):
        return _Weights(self.case, self.specs, self.seed, self.prefix + prefix)

    def stored(self, name):
        return tensor_of(self.case, self.prefix + name, self.specs[self.prefix + name], self.seed)

    def __getitem__(self, name):
        return self.stored(name).double()

    def __contains__(self, name):
        return self.prefix + name in self.specs

    def mul(self, h, name):
        y = h @ self[name].T
        return y + self[name + ".b"] if name + ".b" in self else y


def _unit(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _glu(g, u, limit):
    """The clamped gated activation."""
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1)


def _silu(x):
    return x * torch.sigmoid(x)


def _conv(x, w, bias=None):
    """Causal convolution per channel: x [T, C], w [C, taps]."""
    taps = w.shape[1]
    y = torch.nn.functional.pad(x, (0, 0, taps - 1, 0)).unfold(0, taps, 1)
    y = (y * w).sum(-1)
    return y if bias is None else y + bias


def _frequencies(dims, base, scaling=None):
    """Angles per position and the factor on cosine and sine, under the three kinds of stretching in use."""
    i = torch.arange(dims // 2, dtype=torch.float64, device="cuda")
    f = float(base) ** (-2.0 * i / dims)
    if not scaling:
        return f, 1.0
    factor = float(scaling["factor"])
    if "fast" in scaling:
        def place(turns):
            return dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
        lo, hi = max(math.floor(place(scaling["fast"])), 0), min(math.ceil(place(scaling["slow"])), dims - 1)
        r = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        return f / factor * r + f * (1 - r), 0.1 * math.log(factor) + 1.0
    if "low" in scaling:
        low, high = float(scaling["low"]), float(scaling["high"])
        r = ((scaling["original"] * f / (2 * math.pi) - low) / (high - low)).clamp(0, 1)
        return f / factor * (1 - r) + f * r, 1.0
    return f / factor, 1.0


def _rotate(x, f, m=1.0, neighbours=False, back=False):
    """x [T, heads, dim]: the pairs of the first 2 len(f) channels, halves or neighbours, turned by position * f."""
    n = f.shape[0]
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None, None] * f
    c, s = torch.cos(a) * m, torch.sin(-a if back else a) * m
    head, rest = x[..., :2 * n], x[..., 2 * n:]
    u, v = (head[..., 0::2], head[..., 1::2]) if neighbours else (head[..., :n], head[..., n:])
    p, q = u * c - v * s, v * c + u * s
    head = torch.stack([p, q], -1).flatten(-2) if neighbours else torch.cat([p, q], -1)
    return torch.cat([head, rest], -1)


def _attend(q, k, v, scale, window=None, cap=None, sink=None, sigmoid_bias=None):
    """q [T, H, d], k [T, G, d], v [T, G, e] -> [T, H, e], causal."""
    T, H = q.shape[:2]
    G = k.shape[1]
    i = torch.arange(T, device=q.device)
    hidden = i[None, :] > i[:, None]
    if window:
        hidden |= i[:, None] - i[None, :] >= window
    out = []
    for h in range(H):
        g = h * G // H
        s = (q[:, h] @ k[:, g].T) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if sigmoid_bias is not None:
            p = torch.sigmoid(s + sigmoid_bias[h]).masked_fill(hidden, 0.0)
        else:
            s = s.masked_fill(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(T, 1)], 1)
            p = torch.softmax(s, -1)[:, :T]
        out.append(p @ v[:, g])
    return torch.stack(out, 1)


def _scan(q, k, v, decay, beta=None, remove=None):
    """S <- decay S + k v^T and o = S^T q per head, a token at a time; q, k [T, H, d], v [T, H, e], decay [T, H, d]
    or [T, H, 1].  beta: the delta rule (what the decayed state says of k is taken from v first); remove: (unit key,
    rate) of the part that is taken out of the state before."""
    T, H, d = k.shape
    S = torch.zeros(H, d, v.shape[2], dtype=torch.float64, device=q.device)
    out = torch.empty(T, H, v.shape[2], dtype=torch.float64, device=q.device)
    k, q, a = k[..., None], q[:, :, None, :], decay[..., None]
    for t in range(T):
        u = v[t][:, None, :]
        if remove is not None:
            unit, rate = remove[0][t][..., None], remove[1][t][..., None]
            S = a[t] * S - (rate * unit) * (unit.transpose(1, 2) @ S) + k[t] * u
        else:
            S = a[t] * S
            if beta is not None:
                u = beta[t][:, None, None] * (u - k[t].transpose(1, 2) @ S)
            S = S + k[t] * u
        out[t] = (q[t] @ S)[:, 0]
    return out


def _heads(x, n):
    return x.reshape(x.shape[0], n, -1)


def _latent(h, W, m, eps, neighbours):
    """Attention over a cached latent; with `g` also a sink and an output gate."""
    H, dn, dr, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
    q = W.mul(_unit(W.mul(h, "dq"), eps) * W["dq.norm"], "uq") if "dq" in W else W.mul(h, "q")
    q, kv = _heads(q, H), W.mul(h, "dkv")
    c = _unit(kv[:, :rank], eps) * W["dkv.norm"]
    f, ms = _frequencies(dr, m["rot"]["base"], m["rot"].get("scaling"))
    kr = _rotate(_heads(kv[:, rank:], 1), f, ms, neighbours).expand(-1, H, -1)
    q = torch.cat([q[..., :dn], _rotate(q[..., dn:], f, ms, neighbours)], -1)
    k = torch.cat([_heads(c @ W["uk"].T, H), kr], -1)
    o = _attend(q, k, _heads(c @ W["uv"].T, H), m["scale"], (m.get("mask") or {}).get("size"), sink=W["sink"] if "sink" in W else None)
    o = o.flatten(1)
    return (o * torch.sigmoid(W.mul(h, "g")) if "g" in W else o) @ W["o"].T


def _gla(h, W, m, eps):
    H = m["heads"]
    decay = torch.exp(torch.nn.functional.logsigmoid((h @ W["a1"].T) @ W["a2"].T + W["a2.b"]) / m["tau"])
    o = _scan(_heads(W.mul(h, "q"), H) * m["dim"] ** -0.5, _heads(W.mul(h, "k"), H), _heads(W.mul(h, "v"), H), _heads(decay, H))
    return ((_unit(o, eps) * W["norm"]).flatten(1) * _silu(W.mul(h, "g"))) @ W["o"].T


def _lightning(h, W, m, eps):
    H = m["heads"]
    q, k, v = (_heads(_silu(W.mul(h, n)), H) for n in "qkv")
    decay = torch.tensor(m["decay"], dtype=torch.float64, device=h.device)[None, :, None].expand(h.shape[0], H, 1)
    return (_unit(_scan(q, k, v, decay).flatten(1), eps) * W["norm"] * torch.sigmoid(W.mul(h, "g"))) @ W["o"].T


def _delta_qkv(h, W, m):
    """Projections through their convolutions; q and k of unit length, each group's given to its heads."""
    H, G = m["heads"], m["kv_heads"]
    q, k, v = (_silu(_conv(W.mul(h, n), W[n + ".conv"])) for n in "qkv")
    q, k = (_heads(x, G).repeat_interleave(H // G, 1) for x in (q, k))
    q, k = (x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    return q * m["dim"] ** -0.5, k, _heads(v, H)


def _parallel(h, W, m, eps):
    L, R, wl, wr = m["left"], m["right"], W.at("left."), W.at("right.")
    f, _ = _frequencies(L["rot"]["dims"], L["rot"]["base"], L["rot"]["scaling"])
    q, k = (_rotate(_heads(_unit(wl.mul(h, n), eps) * wl[n + ".norm"], n_h), f, neighbours=True) for n, n_h in (("q", L["heads"]), ("k", L["kv_heads"])))
    fv, _ = _frequencies(L["vdim"], L["rot"]["base"])
    v = _rotate(_heads(wl.mul(h, "v"), L["kv_heads"]), fv, neighbours=True)
    left = _rotate(_attend(q, k, v, L["scale"], L["mask"]["size"]), fv, neighbours=True, back=True).flatten(1) @ wl["o"].T
    q, k, v = _delta_qkv(h, wr, R)
    decay = torch.exp(-torch.exp(wr["A_log"]) * torch.nn.functional.softplus(h @ wr["a"].T + wr["dt_bias"]))
    o = _scan(q, k, v, decay[..., None], beta=torch.sigmoid(wr.mul(h, "b")))
    right = ((_unit(o, eps) * wr["norm"]).flatten(1) * _silu(wr.mul(h, "g"))) @ wr["o"].T
    return m["left_scale"] * left + m["right_scale"] * right


def _general_delta(h, W, m, eps):
    H = m["heads"]
    r, k, v = (_heads(W.mul(h, n), H) for n in "rkv")
    decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ W["w1"].T) @ W["w2"].T + W["w0"]))
    rate = torch.sigmoid(W.mul(h, "a"))
    unit = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    o = _unit(_scan(r, k, v, _heads(decay, H), remove=(unit, _heads(rate, H))), eps)
    return (o.flatten(1) * W["norm"] * torch.sigmoid(W.mul(h, "g"))) @ W["o"].T


def _mamba2(h, W, m, eps):
    H, N, G, inner = m["heads"], m["state"], m["groups"], m["heads"] * m["vdim"]
    z, xbc, dt = (h @ W["in"].T).split([inner, inner + 2 * G * N, H], -1)
    xbc = _silu(_conv(xbc, W["conv"], W["conv.b"]))
    x, B, C = xbc.split([inner, G * N, G * N], -1)
    x, B, C = _heads(x, H), _heads(B, G).repeat_interleave(H // G, 1), _heads(C, G).repeat_interleave(H // G, 1)
    dt = torch.nn.functional.softplus(dt + W["dt_bias"])[..., None]
    y = _scan(C, dt * B, x, torch.exp(-torch.exp(W["A_log"])[:, None] * dt)) + W["D"][:, None] * x
    y = _unit(_heads(y.flatten(1) * _silu(z), m["norm_groups"]), eps).flatten(1) * W["norm"]
    return y @ W["o"].T


def _difference(h, W, m, eps):
    H, G, dk = m["heads"], m["kv_heads"], m["dim"]
    f, ms = _frequencies(m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"])
    q, k = _rotate(_heads(W.mul(h, "q"), 2 * H), f, ms), _rotate(_heads(W.mul(h, "k"), 2 * G), f, ms)
    v = _heads(W.mul(h, "v"), G)
    one, two = (_attend(q[:, i::2], k[:, i::2], v, m["scale"]) for i in (0, 1))
    lam = torch.exp((W["lq1"] * W["lk1"]).sum()) - torch.exp((W["lq2"] * W["lk2"]).sum()) + m["diff"]
    return (_unit(one - lam * two, eps) * (1 - m["diff"])).flatten(1) @ W["o"].T


def _mlstm(h, W, m, eps):
    H, cap, T = m["heads"], m["gate_cap"], h.shape[0]
    q, k, v = (_heads(h @ W[n].T, H) for n in "qkv")
    i = cap * torch.tanh((h @ W["i"].T + W["i.b"]) / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ W["f"].T + W["f.b"]) / cap))
    # the largest of the additions to come so far, each weakened by the gates after it; 0 before the first
    total = f.cumsum(0)
    top = total + torch.cummax(torch.cat([torch.zeros_like(i[:1]), i - total]), 0).values[1:]
    before = torch.cat([torch.zeros_like(top[:1]), top[:-1]])
    keep, add = torch.exp(f + before - top)[..., None], torch.exp(i - top)[..., None]
    both = _scan(q * m["dim"] ** -0.5, add * k, torch.cat([v, torch.ones(T, H, 1, dtype=v.dtype, device=v.device)], -1), keep)
    bottom = torch.maximum(both[..., -1:].abs(), torch.exp(-top)[..., None]) + 1e-6
    o = _unit(both[..., :-1] / bottom, eps).flatten(1)
    return (o * W["norm"] * torch.sigmoid(h @ W["g"].T)) @ W["o"].T


def _channel_delta(h, W, m, eps):
    H = m["heads"]
    q, k, v = _delta_qkv(h, W, m)
    soft = torch.nn.functional.softplus((h @ W["a1"].T) @ W["a2"].T + W["dt_bias"])
    decay = torch.exp(-torch.exp(W["A_log"])[:, None] * _heads(soft, H))
    o = _scan(q, k, v, decay, beta=torch.sigmoid(h @ W["b"].T))
    gate = torch.sigmoid((h @ W["g1"].T) @ W["g2"].T)
    return ((_unit(o, eps) * W["norm"]).flatten(1) * gate) @ W["o"].T


def _mixture(h, W, f, scores, group_score, expert, weigh_inputs=False):
    """The routed feed-forward: scores [T, E], the best groups stay open, the best `top` of theirs are used."""
    r = f["router"]
    gr, E = r.get("groups"), r["experts"]
    pick = scores
    if gr:
        parts = scores.reshape(len(h), gr["count"], -1)
        keep = group_score(parts).topk(gr["keep"], -1).indices
        closed = torch.ones(len(h), gr["count"], dtype=torch.bool, device=h.device).scatter(1, keep, False)
        pick = parts.masked_fill(closed[..., None], -math.inf).flatten(1)
    idx = pick.topk(r["top"], -1).indices
    weight = scores.gather(1, idx) * r.get("scale", 1.0)
    out = torch.zeros_like(h)
    for e in range(E):
        rows, place = (idx == e).nonzero(as_tuple=True)
        if len(rows):
            w = weight[rows, place][:, None]
            we = W.at(f"e{e}.")
            out[rows] += expert(h[rows] * w, we) if weigh_inputs else w * expert(h[rows], we)
    return out


def _swiglu(h, W):
    return (_silu(h @ W["gate"].T) * (h @ W["up"].T)) @ W["down"].T


def _hidden(ids, cfg, W):
    """The residual stream before the final norm, normed: [T, width]."""
    kind = cfg.get("architecture", "Qwen3")
    ids_t = torch.tensor(ids, device="cuda")
    eps = cfg["rms_norm_eps"] if kind == "Qwen3" else cfg["norm"]["eps"]
    gelu = torch.nn.functional.gelu
    if kind == "Qwen3":
        x = W.stored("model.embed_tokens.weight")[ids_t].double()
        H, G = cfg["num_attention_heads"], cfg["num_key_value_heads"]
        f, _ = _frequencies(cfg["head_dim"], cfg["rope_theta"])
        for i in range(cfg["num_hidden_layers"]):
            w = W.at(f"model.layers.{i}.")
            a = w.at("self_attn.")
            h = _unit(x, eps) * w["input_layernorm.weight"]
            q, k = (_rotate(_unit(_heads(h @ a[n + "_proj.weight"].T, g), eps) * a[n + "_norm.weight"], f) for n, g in (("q", H), ("k", G)))
            x = x + _attend(q, k, _heads(h @ a["v_proj.weight"].T, G), cfg["head_dim"] ** -0.5).flatten(1) @ a["o_proj.weight"].T
            h, a = _unit(x, eps) * w["post_attention_layernorm.weight"], w.at("mlp.")
            x = x + (_silu(h @ a["gate_proj.weight"].T) * (h @ a["up_proj.weight"].T)) @ a["down_proj.weight"].T
        return _unit(x, eps) * W["model.norm.weight"]
    x = W.stored("embed")[ids_t].double()
    if kind == "Votapel":
        x = x + W["pos"][:len(ids)]
    if kind == "Begupel":
        b = cfg["embedding"]["bigram"]
        x = x + W["bigram"][[b["buckets"]] + [(p * b["mul_prev"] + c * b["mul_cur"]) % b["buckets"] for p, c in zip(ids, ids[1:])]]
        groups = cfg["norm"]["groups"]
        norm = lambda y, w: _unit(_heads(y, groups), eps).flatten(1) * w  # noqa: E731
    elif kind == "Kebisun":
        norm = lambda y, w: torch.nn.functional.layer_norm(y, y.shape[-1:], w, None, eps)  # noqa: E731
    elif kind == "Putazen":
        X = torch.stack([x] * cfg["streams"])
    squash = lambda y, w, n: torch.tanh(w[n + ".alpha"] * y) * w[n] + w[n + ".b"]  # noqa: E731
    kvs, first = {}, None
    for i, layer in enumerate(cfg["layers"]):
        w = W.at(f"l{i}.")
        mix, mlp, m, f, t = w.at("mix."), w.at("mlp."), layer["mixer"], layer["mlp"], layer["type"]
        if kind == "Kebisun":
            y = _latent(x, mix, m, eps, False) if t == "latent_attention" else _gla(x, mix, m, eps)
            x = x + norm(y, w["norm1"]) * w["ls1"]
            if f["kind"] == "dense":
                y = (gelu(x @ mlp["gate"].T, approximate="tanh") * (x @ mlp["up"].T)) @ mlp["down"].T
            else:
                y = _mixture(x, mlp, f, torch.softmax(x @ mlp["router"].T, -1), None, lambda z, e: gelu(z @ e["up"].T) @ e["down"].T)
            x = x + norm(y, w["norm2"]) * w["ls2"]
        elif kind == "Votapel":
            h = _unit(x, eps) * (1 + w["norm1"])
            p = torch.arange(len(ids), device="cuda")
            warm = 1 + m["q_temp"]["coef"] * torch.log(torch.div(p + 1, m["q_temp"]["every"], rounding_mode="floor").double() + 1)
            q, k = _heads(mix.mul(h, "q") * warm[:, None], m["heads"]), _heads(mix.mul(h, "k"), m["kv_heads"])
            y = _attend(q, k, k, m["scale"], cap=m["softcap"], sink=mix["sink"] if "sink" in mix else None).flatten(1) @ mix["o"].T
            y = y + _mixture(h, mlp, f, torch.sigmoid(h @ mlp["router"].T), lambda s: s.topk(2, -1).values.sum(-1), _swiglu)
            x = x + cfg["residual_mult"] * (y + _swiglu(h, mlp.at("shared.")))
        elif kind == "Begupel":
            h = x + _conv(x, w["canon1"])
            x = x + norm((_lightning if t == "lightning" else _parallel)(h, mix, m, eps), w["norm1"])
            y = mlp.mul(torch.relu(mlp.mul(x, "gate")) * mlp.mul(x, "up"), "down")
            x = x + norm(y, w["norm2"])
        elif kind == "Nefivik":
            h = _unit(x, eps) * w["norm1"]
            if t == "attention":
                fr, _ = _frequencies(m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"])
                if "kv_from" not in m:
                    k, v = (_heads(_conv(h @ mix[n].T, mix[n + ".conv"]), m["kv_heads"]) for n in "kv")
                    kvs[i] = (_rotate(k, fr), v)
                k, v = kvs[m.get("kv_from", i)]
                q = _rotate(_heads(_conv(h @ mix["q"].T, mix["q.conv"]), m["heads"]), fr)
                o = _attend(q, k, v, m["scale"], m["mask"]["size"], sigmoid_bias=mix["pb"]) * torch.sigmoid(h @ mix["g"].T)[..., None]
                y = o.flatten(1) @ mix["o"].T
            else:
                y = _general_delta(h, mix, m, eps)
            x = x + _unit(y * torch.sigmoid(w.mul(h, "rg1")), eps) * w["norm1b"]
            h, limit = _unit(x, eps) * w["norm2"], f["expert"]["limit"]
            y = _mixture(h, mlp, f, torch.softmax(h @ mlp["router"].T, -1), lambda s: s.amax(-1),
                         lambda z, e: _glu(z @ e["gate"].T, z @ e["up"].T, limit) @ e["down"].T)
            x = x + _unit(y * torch.sigmoid(w.mul(h, "rg2")), eps) * w["norm2b"]
            n, s = cfg["token_side"]["dim"], w.at("side.")
            e = W.stored("side.embed")[ids_t, i * n:(i + 1) * n].double()
            x = x + _unit((gelu(x @ s["gate"].T, approximate="tanh") * e) @ s["proj"].T, eps) * s["norm"]
        elif kind == "Putazen":
            run_mixer = {"attention": lambda h: _difference(h, mix, m, eps), "latent_attention": lambda h: _latent(h, mix, m, eps, True),
                         "mamba2": lambda h: _mamba2(h, mix, m, eps)}[t]
            for q, sub in ((1, run_mixer), (2, lambda h: _glu(h @ mlp["gate"].T, h @ mlp["up"].T, f["limit"]) @ mlp["down"].T)):
                u = torch.einsum("s,std->td", w[f"hc{q}.in"], X)
                y = sub(torch.nn.functional.layer_norm(u, u.shape[-1:], w[f"norm{q}"], w[f"norm{q}.b"], eps))
                X = torch.einsum("st,snd->tnd", w[f"hc{q}.mix"], X) + w[f"hc{q}.out"][:, None, None] * y
        else:
            h = squash(x, w, "norm1")
            if t == "attention":
                q, k = (_rotate(_unit(_heads(mix.mul(h, n), g), eps) * mix[n + ".norm"].reshape(-1, m["dim"]),
                                _frequencies(m["rot"]["dims"], m["rot"]["base"])[0])
                        for n, g in (("q", m["heads"]), ("k", m["kv_heads"])))
                v = mix.mul(h, "v")
                if first is None:
                    first = v
                else:
                    v = (1 - mix["vmix"]) * v + mix["vmix"] * first
                y = mix.mul(_attend(q, k, _heads(v, m["kv_heads"]), m["scale"]).flatten(1), "o")
            else:
                y = (_mlstm if t == "mlstm" else _channel_delta)(h, mix, m, eps)
            h = squash(x, w, "norm2")
            if f["kind"] == "dense":
                y = y + _swiglu(h, mlp)
            else:
                y = y + _mixture(h, mlp, f, torch.sigmoid(h @ mlp["router"].T), None, _swiglu, weigh_inputs=True) + _swiglu(h, mlp.at("shared."))
            x = x + cfg["residual_mult"] * y
    if kind == "Votapel":
        return _unit(x, eps) * (1 + W["final.norm"])
    if kind == "Putazen":
        x = X.sum(0)
        return torch.nn.functional.layer_norm(x, x.shape[-1:], W["final.norm"], W["final.norm.b"], eps)
    if kind == "Nefivik":
        return _unit(x, eps) * W["final.norm"]
    return squash(x, W, "final.norm") if kind == "Muzasun" else norm(x, W["final.norm"])


@torch.no_grad()
def exact(case: dict, seed: int):
    if work(dict(case, what="prompt", steps=0))["flops"] > 2.5e14:      # over about 20 seconds in 64 bits
        return None
    cfg = config_of(case)
    W = _Weights(case, _specs(case), seed)
    prompts, after, _ = tokens_of(case, seed)
    first = 0 if case["what"] == "decode" else 1
    rows = [_hidden(p + a, cfg, W)[len(p) - first:len(p) + len(a)] for p, a in zip(prompts, after)]
    head = W["model.embed_tokens.weight" if cfg.get("tie_word_embeddings") else "lm_head.weight" if "hidden_size" in cfg else "head"]
    logits = torch.stack(rows, 1) @ head.T * cfg.get("logit_scale", 1.0)
    if cfg.get("logit_softcap"):
        logits = cfg["logit_softcap"] * torch.tanh(logits / cfg["logit_softcap"])
    return {"logits": list(logits), "tokens": [None] * len(logits) if case["sampled"] else []}
