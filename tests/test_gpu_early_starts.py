"""Kernels started beside their predecessors (programmatic dependent launch) must change nothing: every design's prompts and decode steps,
recorded and eager, have the bits of the plain stream order."""
import numpy as np
import pytest
import torch

import bench
import herbert_rs_b200 as hb
from gpu_util import engine_for, random_ids
from herbert_rs_b200 import ops

pytestmark = pytest.mark.gpu

DENSE = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=32000, hidden_size=1024, num_hidden_layers=3,
             num_attention_heads=16, num_key_value_heads=8, head_dim=128, intermediate_size=3072, rope_theta=1000000.0, rms_norm_eps=1e-6,
             max_position_embeddings=4096, tie_word_embeddings=True, eos_token_id=3)
CONFIGS = {
    **{f"kebisun {s}": lambda s=s: bench._kebisun_config(**bench.DESIGN_SIZES[s][0]) for s in ("1k", "2k")},
    **{f"votapel {s}": lambda s=s: bench._votapel_config(**bench.VOTAPEL_SIZES[s][0]) for s in ("1k", "2k")},
    **{f"begupel {s}": lambda s=s: bench._begupel_config(**bench.BEGUPEL_SIZES[s][0]) for s in ("1k", "2k")},
    **{f"nefivik {s}": lambda s=s: bench._nefivik_config(**bench.NEFIVIK_SIZES[s][0]) for s in ("1k", "2k")},
    **{f"putazen {s}": lambda s=s: bench._putazen_config(**bench.PUTAZEN_SIZES[s][0]) for s in ("1k", "2k")},
    **{f"muzasun {s}": lambda s=s: bench._muzasun_config(**bench.MUZASUN_SIZES[s][0]) for s in ("1k", "2k")},
    "dense 1k": lambda: DENSE,
    "dense 4k": lambda: dict(DENSE, hidden_size=4096, num_attention_heads=32, intermediate_size=12288, num_hidden_layers=2, tie_word_embeddings=False),
}


@pytest.fixture
def pdl():
    """Sets (recorded steps' mode, eager steps' mode); the options are put back afterwards."""
    saved = ops.options.pdl_graph, ops.options.pdl_eager

    def put(graph, eager):
        ops.options.pdl_graph, ops.options.pdl_eager = graph, eager

    yield put
    put(*saved)
    ops.set_pdl(0)


@pytest.mark.parametrize("name", sorted(CONFIGS))
def test_the_bits_of_the_plain_stream_order(name, pdl):
    cfg = CONFIGS[name]()
    model = hb.random_model(cfg, 5, hb.Runtime("cuda", torch.bfloat16))
    for batch, longest in ((1, 700), (3, 90), (12, 150), (17, 20)) + (((64, 40),) if name.startswith("dense") else ()):
        rng = np.random.default_rng(batch)
        lens = [longest] + [int(n) for n in rng.integers(1, longest + 1, batch - 1)]
        reqs = [random_ids(rng, 32000, n + 4) for n in lens]

        def run(graphs):
            eng = hb.Engine(model, max_tokens=batch * (longest + 68), max_slots=batch, use_graphs=graphs)
            slots = [eng.alloc_slot() for _ in reqs]
            out = [eng.step([(s, r[:n]) for s, r, n in zip(slots, reqs, lens)], "last").clone()]
            for t in range(4):
                out.append(eng.step([(s, [r[n + t]]) for s, r, n in zip(slots, reqs, lens)], "last").clone())
            return torch.stack(out)

        pdl(0, False)
        base = run(True)
        assert torch.isfinite(base).all()
        for graph, eager, graphs in ((1, True, True), (2, True, True), (0, True, False)):
            pdl(graph, eager)
            assert torch.equal(run(graphs), base), (batch, graph, eager, graphs)
    ops.check_kernel_errors()


def test_a_recorded_step_is_recorded_again_when_the_option_changes(model_dirs, pdl):
    eng = engine_for(model_dirs["D"], "bfloat16")
    s = eng.alloc_slot()
    eng.step([(s, [1, 2, 3])], "last")
    for graph, recorded in ((1, 1), (0, 2), (1, 2), (2, 3)):
        pdl(graph, True)
        eng.step([(s, [4])], "last")
        assert len(eng._graphs) == recorded
