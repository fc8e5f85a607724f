"""Kernels started beside their predecessors (programmatic dependent launch) must change nothing."""
import pytest

from gpu_util import engine_for
from herbert_rs_b200 import ops

pytestmark = pytest.mark.gpu

@pytest.fixture
def pdl():
    """Sets (recorded steps' mode, eager steps' mode); the options are put back afterwards."""
    saved = ops.options.pdl_graph, ops.options.pdl_eager

    def put(graph, eager):
        ops.options.pdl_graph, ops.options.pdl_eager = graph, eager

    yield put
    put(*saved)
    ops.set_pdl(0)


def test_a_recorded_step_is_recorded_again_when_the_option_changes(model_dirs, pdl):
    eng = engine_for(model_dirs["D"], "bfloat16")
    s = eng.alloc_slot()
    eng.step([(s, [1, 2, 3])], "last")
    for graph, recorded in ((1, 1), (0, 2), (1, 2), (2, 3)):
        pdl(graph, True)
        eng.step([(s, [4])], "last")
        assert len(eng._graphs) == recorded
