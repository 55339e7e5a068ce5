"""The loss of explicit training samples: one value per input, and the sum of its
rows' losses to the last bit of a float."""
import ctypes as C
import math

import numpy as np
import pytest

from rustracer_b200.renderer import lib
from tests.test_gpu_guide import _params, _samples, _scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    gs = _scene()
    gs.guide_set_params(_params(67))
    return gs


def _loss(gs, s):
    loss = C.c_float()
    assert lib().rt_guide_loss_grad(gs.h, C.c_void_p(s.ctypes.data), len(s), C.byref(loss), None) == 0
    return loss.value


@pytest.mark.parametrize("n", [1, 16, 17, 1024, 1500])
def test_loss_is_the_sum_of_its_rows(scene, n):
    s = np.ascontiguousarray(_samples(n, 40 + n), np.float32)
    rows = math.fsum(_loss(scene, s[i:i + 1]) for i in range(n))
    # half a unit in the last place of a float; the sum itself is in doubles
    assert abs(_loss(scene, s) - rows) <= 2.0 ** -24 * (1 + 1e-6) * abs(rows)


def test_same_bits_every_call(scene):
    s = np.ascontiguousarray(_samples(65536, 7), np.float32)
    assert len({_loss(scene, s) for _ in range(20)}) == 1


def test_training_reports_the_same_loss(scene):
    s = np.ascontiguousarray(_samples(2000, 9), np.float32)
    ref = _loss(scene, s)
    assert scene.guide_train(s, 1) == ref
    scene.guide_set_params(_params(67))
