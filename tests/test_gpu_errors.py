"""A CUDA call that fails without harm to the context (no such device, no memory)
is reported once, by the call that made it; what runs afterwards is not
touched by it."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from merle_b200 import abi, lib, workload as WL
from merle_b200.engine import Engine
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


def test_network_after_a_batch_that_does_not_fit(mb, cuda):
    """34M rows of 4,096 activations (550 GB) are refused; the buffers of the
    smaller batch before are gone then, and the next call makes its own."""
    m = MLP(1, 4096, 1, seed=1)
    x = np.linspace(-1, 1, 7, dtype=np.float32).reshape(7, 1)
    want = m.forward(x)
    y = np.zeros(7, np.float32)
    assert lib().mb_mlp_forward(m.handle, x.ctypes.data_as(C.POINTER(C.c_float)), 1 << 25, 0,
                                y.ctypes.data_as(C.POINTER(C.c_float))) == abi.MB_ERR_OOM
    np.testing.assert_array_equal(m.forward(x[:3]), want[:3])
    np.testing.assert_array_equal(m.forward(x), want)
    m.close()


def test_batch_after_a_batch_that_does_not_fit(mb, cuda):
    """Eight queries of 4.2G groups each (269 GB of sums) are refused before
    anything runs; the next batch allocates its own results."""
    e = Engine(0)
    e.gen_star(1, 1, 100_003)
    e.build_index()
    qs = [abi.query(t, *p) for t, p in map(WL.as_tuple, WL.ssb13())]
    want = e.query_batch(qs)
    big = (abi.mb_query * 8)(*[abi.query(2, 0, 600_000_000, 0, 10)] * 8)
    out = np.zeros(8, np.int64)
    assert lib().mb_engine_query_batch(e.handle, big, 8, None, out.ctypes.data, None) == abi.MB_ERR_OOM
    for n in (2, len(qs)):
        got = e.query_batch(qs[:n])
        np.testing.assert_array_equal(got[0], want[0][:len(got[0])])
        np.testing.assert_array_equal(got[1], want[1][:n])
    e.close()
