"""Parameters and gradients come back whole: into pageable and pinned memory,
from two threads of two scenes at once."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from rustracer_b200 import abi
from rustracer_b200.renderer import lib
from tests.test_gpu_guide import _scene

pytestmark = pytest.mark.gpu


def _pattern(k):
    return (np.arange(abi.RT_GUIDE_PARAMS, dtype=np.float32) * np.float32(1.0 + k) + np.float32(k))


def test_pageable_and_pinned():
    gs, p = _scene(), _pattern(0)
    gs.guide_set_params(p)
    assert np.array_equal(gs.guide_get_params(), p)
    pinned = torch.zeros(abi.RT_GUIDE_PARAMS).pin_memory()
    assert lib().rt_guide_params(gs.h, C.c_void_p(pinned.data_ptr()), 0) == 0
    assert np.array_equal(pinned.numpy(), p)


def test_unaligned_destination():
    gs, p = _scene(), _pattern(1)
    gs.guide_set_params(p)
    buf = np.zeros(abi.RT_GUIDE_PARAMS * 4 + 64, np.uint8)
    assert lib().rt_guide_params(gs.h, C.c_void_p(buf.ctypes.data + 4), 0) == 0
    assert np.array_equal(buf[4:4 + p.nbytes].view(np.float32), p)
    assert not buf[:4].any() and not buf[4 + p.nbytes:].any()


def test_two_threads():
    sc = [_scene(), _scene()]
    for k, gs in enumerate(sc):
        gs.guide_set_params(_pattern(k))
    out = [None, None]

    def run(k):
        for _ in range(3):
            out[k] = sc[k].guide_get_params()

    th = [threading.Thread(target=run, args=(k,)) for k in (0, 1)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for k in (0, 1):
        assert np.array_equal(out[k], _pattern(k))
