"""What the kernels' sources must keep to so that a kernel may start beside its predecessor (programmatic dependent launch)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "herbert_rs_b200", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))

# Weights and tables, and what the host copied before the step: no kernel of a step writes them.
CONSTANT = {"W", "w", "w2", "wr", "up", "down", "nw", "bias", "sink", "scale", "add", "yb", "a_log", "dt_bias", "table", "pos_table", "pair_table",
            "freq", "fv", "tok_seq", "tok_pos", "positions", "seq_slot", "seq_start", "seq_pos0", "seq_len", "seq_pages", "rows"}
# Outputs that their kernel never reads.
WRITTEN = {"out", "h", "C", "mid", "gates", "ids", "wts", "pair_off", "tile_off", "list", "slot", "tile_expert", "rows_used", "row_scale", "sorted",
           "pv", "pi", "overflow", "cache"}
WRITTEN_IN = {"a": {"gla_decay_kernel"}, "y": {"gla_output_kernel", "gated_rmsnorm_kernel", "gated_rmsnorm_warp_kernel", "rotate_heads_back_kernel",
                                             "head_gate_kernel", "difference_heads_kernel"}}


def code_of(path):
    text = open(path).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def kernels_of(path):
    """(name, parameter list, body) of every kernel in a file."""
    text, out = code_of(path), []

    def closing(at, a, b):
        depth = 0
        for i in range(at, len(text)):
            depth += (text[i] == a) - (text[i] == b)
            if depth == 0:
                return i
        raise AssertionError(path)

    for m in re.finditer(r"__global__", text):
        for call in re.compile(r"(\w+)\s*\(").finditer(text, m.end()):
            if call.group(1) not in ("__launch_bounds__", "__cluster_dims__"):
                break
        end = closing(call.end() - 1, "(", ")")
        brace = text.index("{", end)
        out.append((call.group(1), text[call.end():end], text[brace:closing(brace, "{", "}")]))
    return out


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_what_a_predecessor_writes_is_read_with_ordinary_loads(path):
    """A kernel that starts early is alive while its predecessor writes.  Neither `__ldg` (data that is read-only for the kernel's whole life)
    nor `__restrict__` (which lets a load pass the wait, and turn into one) may stand at what another kernel of the step writes."""
    text = code_of(path)
    assert "__ldg" not in text
    for const, name in re.findall(r"(const )?\w+\* __restrict__ (\w+)", text):
        assert name in CONSTANT if const else name in WRITTEN or name in WRITTEN_IN, name
    for kernel, params, _ in kernels_of(path):
        for const, name in re.findall(r"(const )?\w+\* __restrict__ (\w+)", params):
            if not const and name in WRITTEN_IN:
                assert kernel in WRITTEN_IN[name], (kernel, name)
