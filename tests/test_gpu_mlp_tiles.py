"""The network's tiled kernels (csrc/mlp.cu) at sizes around their tiles (16 rows
x 64 outputs forward, 32 x 32 weights and 128-row splits backward) against the
float64 oracle: forward within the FP32 rounding of a sum of `in` products,
gradients within that of a sum over the rows."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp as OM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 17, 128, 129, 1000])
@pytest.mark.parametrize("nin,hidden,nout", [(32, 64, 16), (1, 1, 1), (33, 65, 31), (64, 130, 96)])
def test_gradients_and_forward(cuda, mb, n, nin, hidden, nout):
    from merle_b200 import planner as P
    r = np.random.default_rng(n + nin)
    x = r.random((n, nin)).astype(np.float32)
    t = r.normal(0, 1, (n, nout)).astype(np.float32)
    mask = (r.random((n, nout)) < 0.8).astype(np.float32)
    mask[0, 0] = 1
    m = P.MLP(nin, hidden, nout, seed=5)
    try:
        p = m.get_params()
        want, _ = OM.forward(p, x, nin, hidden, nout)
        np.testing.assert_allclose(m.forward(x), want, rtol=1e-4, atol=1e-5)
        _, g = m.gradients(x, t, mask)
        _, wg = OM.loss_and_grad(p, x, t, mask, nin, hidden, nout)
        np.testing.assert_allclose(g, wg, rtol=1e-3, atol=1e-5 * np.max(np.abs(wg)))
    finally:
        m.close()


def test_gradients_of_more_rows_than_a_grid_has_splits(cuda, mb):
    """65,536 splits of 128 rows and one row more, the only one with a target: a network
    this small would take a split per 128 rows, one more than a grid has in z."""
    from merle_b200 import planner as P
    n = 65536 * 128 + 1
    x = np.zeros((n, 1), np.float32)
    t = np.zeros((n, 1), np.float32)
    t[-1, 0] = 2
    m = P.MLP(1, 1, 1, seed=5)
    try:
        p = m.get_params()
        _, g = m.gradients(x, t, np.ones((n, 1), np.float32))
        _, wg = OM.loss_and_grad(p, x, t, np.ones((n, 1), np.float32), 1, 1, 1)
        np.testing.assert_allclose(g, wg, rtol=1e-3, atol=1e-5 * np.max(np.abs(wg)))
    finally:
        m.close()
