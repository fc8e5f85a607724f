"""What preparing a step costs and refuses on the host, and the clearing of state planes at the edges of its range."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from herbert_rs_b200 import ops


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [[(5, 3, 0)], [(5, 3, 0), (2, 3, 4)], [(70000, 2, 3)], [(1, 2, 1), (65536, 2, 1)]])
def test_planes_of_any_extent_are_cleared(shapes):
    """Planes without a number, and planes of more entries than a grid is deep."""
    planes = [torch.ones(s, device="cuda") for s in shapes]
    ops.RowClearer(planes).clear(1)
    for p in planes:
        assert not p[:, 1].any() and (p[:, 0] == 1).all() and (p[:, 2:] == 1).all()
