"""A CUDA call that fails without harm to the context (no such device, no memory)
is reported once, by the call that made it; what runs afterwards is not
touched by it."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from merle_b200 import abi, lib
from merle_b200.planner import MLP

pytestmark = pytest.mark.gpu


def test_failed_call_leaves_no_error_behind(mb, cuda):
    m = MLP(8, 16, 4, seed=1)
    x = np.random.default_rng(0).random((5, 8), np.float32)
    want = m.forward(x)
    cfg = abi.mb_mlp_config(8, 16, 4, 1)
    other = C.c_void_p()
    assert lib().mb_mlp_create(1 << 20, C.byref(cfg), C.byref(other)) == abi.MB_ERR_CUDA
    np.testing.assert_array_equal(m.forward(x), want)
    m.close()
