"""The work that bench.py counts for a launcher: launchers that take the same operation at other sizes count alike."""
import collections

import pytest

import bench
from herbert_rs_b200 import ops


@pytest.mark.parametrize("kind,names", [
    (kind, names) for kind in ("kebisun", "votapel", "nefivik", "muzasun")
    for names in ([n for n in ops._SIGS if n.startswith("hb_moe_experts") and not n.endswith(("_ok", "_rows"))],)] + [
    (kind, ["hb_latent_attention", "hb_latent_attention_mma_bf16", "hb_latent_prefill_tc_bf16"]) for kind in ("kebisun", "putazen")])
def test_every_launcher_of_an_operation_is_counted(kind, names):
    ctx = collections.defaultdict(lambda: 8, kind=kind)
    work = {n: bench._launcher_work(n, 2, ctx) for n in names}
    assert len(work) >= 3 and len(set(work.values())) == 1 and None not in work.values(), work
