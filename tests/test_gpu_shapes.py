"""Compiled op forms of the fused kernel (csrc/shape.cuh) on a GPU: the four
query templates at table sizes around the tile edges, in both column layouts,
at every tile width and group strategy, with and without candidate checks,
against the CPU oracle's no-index answer.  Integer work: bit-exact."""
from __future__ import annotations

import numpy as np
import pytest

from merle_b200 import abi, workload as WL
from tests import helpers as H

pytestmark = pytest.mark.gpu

# a warp tile is 1,024 words_per_lane rows; 64-row drain batches; 1,024-row chunks
ROWS = [1, 63, 1023, 1025, 4097, 40_003, 300_001]


@pytest.fixture(scope="module")
def oracle_answers(orc):
    """(rows, query) -> the oracle's sums and row count."""
    memo, hosts = {}, {}

    def get(n, t, a):
        if (n, t, a) not in memo:
            if n not in hosts:
                hosts[n] = orc.StarHost(5, 1, n)
            ng = int(_ngroups(abi.query(t, *a)))
            memo[n, t, a] = orc.join_grpby(n, H.ssb_op(hosts[n], WL.TEMPLATE_NAME[t], a).to_c(), ng)
        return memo[n, t, a]
    return get


def _ngroups(q):
    from merle_b200.engine import Engine
    return Engine.ngroups(q)


def _queries():
    """Exact covers, candidate-checked edges, dense (every 1,024-row chunk
    fills several drain batches) and empty results."""
    qs = [WL.as_tuple(q) for q in WL.ssb13()]
    qs += [(1, (67, 1769, 2, 11, 3, 48)), (2, (26, 995, 1, 249)), (3, (3, 243, 6, 246, 17, 2103)),
           (4, (4, 214, 110, 220, 280, 720, 14, 2518)), (2, (40, 80, 13, 14)), (1, (1, 2, 0, 1, 1, 2)),
           (3, (10, 11, 20, 21, 0, 2557)), (4, (3, 249, 0, 250, 40, 1000, 5, 2550))]
    return qs


@pytest.mark.parametrize("width4", [False, True])
@pytest.mark.parametrize("n", ROWS)
def test_templates_match_oracle(oracle_answers, cuda, n, width4):
    from merle_b200.engine import Engine
    e = Engine(0)
    try:
        e.gen_star(5, 1, n, width4=width4)
        e.build_index()
        for t, a in _queries():
            q = abi.query(t, *a)
            want, wn = oracle_answers(n, t, a)
            for v in (0, 1, 2, 4):
                for gs in (abi.GRP_AUTO, abi.GRP_SHARED, abi.GRP_GLOBAL):
                    p = abi.mb_plan()
                    p.launch.words_per_lane, p.launch.grp_strategy = v, gs
                    got, gn, _ = e.query(q, p)
                    np.testing.assert_array_equal(got, want, err_msg=f"{t}{a} V={v} gs={gs}")
                    assert gn == wn
    finally:
        e.close()


@pytest.mark.parametrize("cover", [abi.COVER_RULE, abi.COVER_NOEDGE, abi.COVER_NOCOMPL, abi.COVER_FINE])
def test_covers_agree(oracle_answers, cuda, cover):
    """Which clauses an uncertain row is checked against depends on the
    predicates' covers: every cover gives the oracle's answer."""
    from merle_b200.engine import Engine
    n = 40_003
    e = Engine(0)
    try:
        e.gen_star(5, 1, n)
        e.build_index()
        for t, a in _queries():
            want, wn = oracle_answers(n, t, a)
            p = abi.mb_plan()
            p.cover = cover
            got, gn, _ = e.query(abi.query(t, *a), p)
            np.testing.assert_array_equal(got, want, err_msg=f"{t}{a} cover {cover}")
            assert gn == wn
    finally:
        e.close()
