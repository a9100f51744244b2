"""Super elements hold the two-pass product's element outputs only where level 0
takes two passes, and for the right-hand sides that run in a precision."""
import gc

import numpy as np
import pytest
import torch

from tests.test_gpu_super_passes import _solver

pytestmark = pytest.mark.gpu
LOADS = 24


def _memory(shape, mixed):
    gc.collect()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    s = _solver(shape, mixed, LOADS)
    used = free - torch.cuda.mem_get_info()[0]
    U, its, res = s.pcg_all()
    assert max(res) < 1e-8
    y = s.matvec(0, U[:s.numDOFs], fp32=True)
    assert torch.isfinite(y).all()
    del s, U, y
    return used


def test_element_outputs_where_they_are_used(monkeypatch):
    """The outputs of a right-hand side are 24 values an element slot: for 10x48x10
    (19 thousand slots) 3.7 MB in double and 1.8 in single, 10x60x10 (25 thousand) 4.9
    and 2.4.  FP64 takes one pass on the first; on the second it needs them in
    double for every load case, in single for one."""
    _memory((10, 48, 10), False)               # what a first solver leaves to the process
    one = _memory((10, 48, 10), False)
    two = _memory((10, 60, 10), False)
    both = _memory((10, 60, 10), True)
    monkeypatch.setenv("TOPGPU_COARSE_TWOPASS_MIN", "0")
    forced = _memory((10, 48, 10), False)
    assert forced - one > 0.7 * LOADS * 3.7e6
    assert both - two > 0.7 * LOADS * 2.4e6
