"""What preparing a step costs and refuses on the host, and the clearing of state planes at the edges of its range."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from herbert_rs_b200 import ops
from herbert_rs_b200.engine import engine
from herbert_rs_b200.errors import RequestError


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [[(5, 3, 0)], [(5, 3, 0), (2, 3, 4)], [(70000, 2, 3)], [(1, 2, 1), (65536, 2, 1)]])
def test_planes_of_any_extent_are_cleared(shapes):
    """Planes without a number, and planes of more entries than a grid is deep."""
    planes = [torch.ones(s, device="cuda") for s in shapes]
    ops.RowClearer(planes).clear(1)
    for p in planes:
        assert not p[:, 1].any() and (p[:, 0] == 1).all() and (p[:, 2:] == 1).all()


class _Cache:
    num_kv_groups, max_pages_per_seq, lengths = 1, 32, [0] * 64

    def reserve(self, pairs):
        pass

    def page_rows(self, group, slots, width):
        return np.zeros((len(slots), width), dtype=np.int32)


def _engine():
    """As much of an engine as a step is prepared with, without a device."""
    e = engine.Engine.__new__(engine.Engine)
    e.model = SimpleNamespace(spec=SimpleNamespace(vocab_size=1000, position_components=1))
    e.rt, e.cache, e.use_graphs = SimpleNamespace(page_size=64), _Cache(), True
    e._host, e._dev = torch.empty(1 << 14, dtype=torch.int32), torch.empty(1 << 14, dtype=torch.int32)
    e._copied = SimpleNamespace(synchronize=lambda: None, record=lambda: None)
    return e


def test_ids_are_checked_once_a_step(monkeypatch):
    """Not once a sequence: 64 sequences of one token each spent 0.2 ms a step on it."""
    calls, check = [], engine._token_array
    monkeypatch.setattr(engine, "_token_array", lambda tokens, vocab: calls.append(len(tokens)) or check(tokens, vocab))
    batch = _engine()._prepare([(i, [7 * i]) for i in range(64)], "last")
    assert calls == [64] and batch.token_ids.tolist() == [7 * i for i in range(64)]


@pytest.mark.parametrize("entries,message", [
    ([(3, [1, 2]), (5, [7, 1000])], "slot 5: token id 1000 is outside"), ([(3, [1, -1, 2000]), (5, [])], "slot 3: token id -1 is outside"),
    ([(3, []), (5, [1000])], "slot 3: a sequence must bring"), ([(3, [1]), (5, [])], "slot 5: a sequence must bring"),
    ([(3, [1.0])], "slot 3: token id 1.0 is outside")])
def test_what_is_refused_is_named_in_order(entries, message):
    with pytest.raises(RequestError, match=message):
        _engine()._prepare(entries, "last")
