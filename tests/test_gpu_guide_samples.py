"""Explicit training samples at the edges of a warp's rows and of the batch
padding: loss and gradient against the CPU restatement."""
import numpy as np
import pytest

from oracle import guide as OG
from tests.test_gpu_guide import INV, LO, RES, _params, _rel, _samples, _scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    gs, p = _scene(), _params(61)
    gs.guide_set_params(p)
    return gs, p


@pytest.mark.parametrize("n", [1, 15, 16, 17, 33, 1023, 1025])
def test_loss_and_gradient(scene, n):
    gs, p = scene
    s = _samples(n, 20 + n)
    loss, g = gs.guide_loss_grad(s)
    lref, gref = OG.loss_and_grad(p, RES, LO, INV, s)
    assert abs(loss - lref) < 1e-3 * max(abs(lref), 1e-2)
    # about eight bf16 roundings (2^-9 each) from the features to a gradient:
    # 1.6e-2 for one row, less over many
    assert _rel(g, gref) < (5e-2 if n < 100 else 2e-2)
