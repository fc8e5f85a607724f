"""What the kernels' sources must keep to so that a kernel may start beside its predecessor (programmatic dependent launch)."""
import glob
import os
import re
import subprocess

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


def test_what_a_launcher_keeps_it_keeps_per_device(tmp_path):
    """A number is asked for once on each device, again after a failure, and always beyond the table."""
    src = tmp_path / "per_device.cpp"
    src.write_text("""
#include "per_device.h"
#include <cstdio>
static HbPerDevice kept;
int main() {
  int asked = 0;
  auto get = [&](int dev, int answer) { return hb_per_device(kept, dev, [&]() { ++asked; return answer; }); };
  if (get(0, 148) != 148 || get(0, 7) != 148 || asked != 1) return 1;
  if (get(1, -1) != -1 || get(1, 132) != 132 || get(1, 5) != 132 || asked != 3) return 2;
  if (get(HB_KEPT_DEVICES, 3) != 3 || get(HB_KEPT_DEVICES, 4) != 4 || asked != 5) return 3;
  return get(0, 1) == 148 ? 0 : 4;
}
""")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0


def test_the_products_of_few_rows_set_their_shared_memory_up_on_every_device():
    code = code_of(os.path.join(CSRC, "gemm_skinny.cu"))
    assert "static HbPerDevice" in code and not re.search(r"\n +static (int|bool)\b", code)


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_every_kernel_waits_for_its_predecessor_and_takes_tensor_memory_before_it_lets_the_next_one_start(path):
    """A kernel that does not wait lets its successor pass while older ones still run; tensor memory that an early CTA of the next kernel
    could take first would never come free."""
    for kernel, _, body in kernels_of(path):
        assert "pdl_wait();" in body, kernel
        depth = body[:body.index("pdl_wait();")].count("{") - body[:body.index("pdl_wait();")].count("}")
        assert depth == 1, f"{kernel}: every thread waits"
        if "tcgen05.alloc" in body and "pdl_launch();" in body:
            assert body.index("tcgen05.alloc") < body.index("pdl_launch();"), kernel
