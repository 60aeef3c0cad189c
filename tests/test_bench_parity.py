"""The bench's parity check where the reference's CPU code is not built: every answer
against the repository's own oracle, and a wrong one is named."""
from __future__ import annotations

import numpy as np
import pytest

import bench
from merle_b200 import abi, workload as WL
from merle_b200.engine import Engine
from tests import helpers as H


@pytest.mark.parametrize("n", [1, 40_003])
def test_oracle_parity(orc, mb, n):
    star = orc.StarHost(bench.SEED_DATA, 1, n)
    qs = [abi.query(t, *p) for t, p in map(WL.as_tuple, WL.ssb13() + WL.span_mix(1, 8))]
    want = [orc.join_grpby(n, H.ssb_op(star, WL.TEMPLATE_NAME[int(q.tmpl)], WL.as_tuple(q)[1]).to_c(),
                           Engine.ngroups(q)) for q in qs]
    answers = bench.oracle_pass(star, n, qs, 4)
    for (a, r), (b, s) in zip(answers, want):
        np.testing.assert_array_equal(a, b)
        assert r == s
    offs = np.cumsum([0] + [len(a) for a, _ in answers])[:-1].tolist()
    out, nq = np.concatenate([a for a, _ in answers]), np.array([r for _, r in answers], np.uint64)
    p = bench.oracle_check(qs, answers, out, offs, nq, n)
    assert p["oracle_equal"] is True and p["reference_equal"] is None and p["mismatched"] == []
    assert p["queries"] == len(qs) and p["groups_compared"] == len(out)
    answers[3][0][-1] += 1 << 32            # the oracle's sum off past 32 bits
    answers[5] = (answers[5][0], answers[5][1] + 1)  # its row count
    p = bench.oracle_check(qs, answers, out, offs, nq, n)
    assert p["oracle_equal"] is False and p["mismatched"] == [3, 5]
