"""Device memory of the 4-wide nodes: their packed form exists once it is selected."""
import numpy as np
import pytest
import torch

from rustracer_b200 import abi
from rustracer_b200.renderer import GpuScene
from tests.test_gpu_packed_nodes import _hard_rays, _soup

pytestmark = pytest.mark.gpu

N = 200_000
LEAVES = 80 * N                                  # record and box of every primitive


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_packed_on_the_first_selection():
    sb, r = _soup(N, 3), _hard_rays(3)
    g = GpuScene(sb)
    ref = g.trace_closest(r)
    before = _free()
    g.set_tuning(node_format=abi.RT_NODES_WIDE4)
    first = before - _free()
    # its leaves are new; its nodes take the place of the build's
    assert 0.75 * LEAVES < first < 1.5 * LEAVES
    for fmt in (abi.RT_NODES_WIDE4, abi.RT_NODES_FULL, abi.RT_NODES_WIDE4):
        g.set_tuning(node_format=fmt)
        got = g.trace_closest(r)
        assert all(np.array_equal(got[k].view(np.uint32), ref[k].view(np.uint32)) for k in ref.dtype.names)
    assert before - _free() <= first + (1 << 21)


def test_released_with_the_scene():
    sb = _soup(N, 4)
    left = []
    for k in range(4):
        g = GpuScene(sb)
        if k % 2:
            g.set_tuning(node_format=abi.RT_NODES_WIDE4)
        g.close()
        left.append(_free())
    assert max(left[1:]) - min(left[1:]) <= 1 << 22
