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


PROGRAMS = {  # general programs (not a conjunctive chain), with and without edge bins
    "or_and": ([abi.ORM, 0, 0, 0], [abi.ORM, 0, 1, 0], [abi.ANDM, 0, 2, 0]),
    "not_or": ([abi.ORM, 1, 0, 0], [abi.NOT, 0, 1, 0], [abi.ORM, 0, 1, 0]),
    "regs": ([abi.ORM, 0, 0, 0], [abi.ORM, 1, 1, 0], [abi.ORM, 2, 2, 0], [abi.AND, 0, 1, 0], [abi.OR, 0, 2, 0]),
}


@pytest.mark.parametrize("chk", [False, True])
@pytest.mark.parametrize("n", [1, 1023, 2049, 40_003])
def test_general_programs_match_oracle(orc, cuda, n, chk):
    """Programs outside the conjunctive form in the warp-independent kernel, at
    every tile width and group strategy, against the oracle's interpreter."""
    from merle_b200 import device as D, ops
    f, fd = orc.gen_flat(11, n), D.DevFlat(11, n)
    s = abi.mb_src()
    bm_h, bm_d = [], []
    for col, lo, hi in (("a", [0, 300, 600], [300, 600, 700]), ("b", [0, 2, 9], [2, 9, 30]), ("c", [1, 20, 30], [20, 30, 51])):
        s.col, s.width = orc.ptr(f[col]), 4
        h, _ = orc.bitmap_create(s, n, lo, hi)
        d, _ = D.bitmap_create(D.src_of(fd[col]), n, lo, hi)
        bm_h.append(h)
        bm_d.append(d)
    args = (200, 650, list(range(1, 20)), 0, 40)  # a filter, an OR clause, group-less SUM

    def prog(b, ins):
        return ops.Vprg(n, [ops.Col(middle=[x[0], x[1]], rightmost=x[2] if chk else None) for x in b],
                        [tuple(i) for i in ins]).to_c()

    def op(c):
        o = ops.flat_op(c["a"], c["b"], c["c"], c["d"], c["e"], args[0], args[1], [3, 7, 11], args[3], args[4])
        o.keys = [(3, abi.X_ID, 1, 0, 1)]
        return o.to_c()
    for name, ins in PROGRAMS.items():
        want, wn = orc.vprg_grpby(prog(bm_h, ins), op(f), 11)
        pd, od = prog(bm_d, ins), op(fd)
        for v in (0, 1, 2, 4):
            for gs in (abi.GRP_AUTO, abi.GRP_GLOBAL, abi.GRP_HASH):
                la = abi.mb_launch()
                la.words_per_lane, la.grp_strategy = v, gs
                out, nq = D.vprg_grpby(pd, od, 11, la)
                np.testing.assert_array_equal(D.to_host(out, np.int64), want, err_msg=f"{name} V={v} gs={gs}")
                assert int(D.to_host(nq, np.uint64)[0]) == wn
