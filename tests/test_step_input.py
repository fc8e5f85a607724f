"""What a step's input goes through on the host, and the launch that zeroes a new sequence's state."""
import numpy as np
import pytest
import torch

from herbert_rs_b200.cache import CacheNeed, SequenceCache, StateNeed
from herbert_rs_b200.engine.batch import StepBatch
from herbert_rs_b200.engine.engine import _token_array

V = 10


@pytest.mark.parametrize("tokens", [[0], [9, 0, 3], [True, 2], [np.int32(3), np.uint8(4), 5], [np.int64(9)]])
def test_ids_that_are_inside_become_the_same_numbers(tokens):
    assert _token_array(tokens, V).tolist() == [int(t) for t in tokens]


@pytest.mark.parametrize("tokens", [[10], [-1], [1, 2.0], [1, "a"], [None], [2 ** 70, 1], [np.uint64(2 ** 63), 1], [np.True_, 1], [[1], 2], [np.float32(1)]])
def test_anything_else_is_left_to_the_check_that_names_it(tokens):
    assert _token_array(tokens, V) is None


def test_the_step_buffer_is_the_same_either_way():
    seqs = [[1, 2, 3], [9], [4, 5]]
    bufs = []
    for ids in (None, [np.array(s, dtype=np.int64) for s in seqs]):
        batch = StepBatch([2, 0, 1], seqs, [0, 7, 64], [[2], [0], [1]], 1, ids=ids)
        buf = np.full(batch.layout.total, -1, dtype=np.int32)
        batch.fill_host(buf, [np.arange(3 * batch.pages_width, dtype=np.int32)])
        bufs.append(buf)
    assert np.array_equal(*bufs)


@pytest.mark.gpu
@pytest.mark.parametrize("groups", [1, 3, 17, 35])
def test_a_new_slots_state_is_zero_and_nobody_elses(groups):
    shapes = [((1,), torch.int32), ((3, 5), torch.float32), ((4, 16, 7), torch.float32), ((7,), torch.bfloat16), ((2, 128, 128), torch.float32)]
    needs = [CacheNeed(state=StateNeed((*shapes[i % 5][0], 1 + i // 5), shapes[i % 5][1])) for i in range(groups)] + [CacheNeed(state=StateNeed((1, 1), torch.int32))]
    cache = SequenceCache(needs, [None] * len(needs), 2, 3, device="cuda")
    for st in cache.state:
        st.fill_(3)
    slot = cache.alloc_slot()
    for st in cache.state:
        assert not st[:, slot].any()
        rest = [s for s in range(3) if s != slot]
        assert (st[:, rest] == 3).all()
