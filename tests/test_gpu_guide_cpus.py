"""Downloads and sample preparation with fewer CPUs than threads they would like."""
import os

import numpy as np
import pytest

from tests.test_gpu_guide import _params, _samples, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cpus", [1, 3, 4])
def test_few_cpus(cpus):
    mine = sorted(os.sched_getaffinity(0))
    if len(mine) < cpus:
        pytest.skip("fewer CPUs than that")
    gs, p = _scene(), _params(71)
    s = _samples(4096, 12)
    gs.guide_set_params(p)
    loss, grad = gs.guide_loss_grad(s)
    try:
        os.sched_setaffinity(0, set(mine[:cpus]))
        assert np.array_equal(gs.guide_get_params(), p)
        loss2, grad2 = gs.guide_loss_grad(s)
    finally:
        os.sched_setaffinity(0, set(mine))
    assert loss2 == loss
    # the gradient's atomics are unordered: up to 4096 terms, each pair of sums within
    # their roundings of one another in norm
    assert np.linalg.norm(grad2 - grad) <= 4096 * 2.0 ** -24 * np.linalg.norm(grad)
