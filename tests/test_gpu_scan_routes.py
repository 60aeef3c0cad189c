"""Ops that are no compiled template through the plans without an index (csrc/scan.cu): which
kernel takes them depends on their clauses, their widths and the rows.  Sums against
numpy at table sizes on both sides of each line; times against the same op on a list
of all rows."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from merle_b200 import abi, check, device as D, ops

pytestmark = pytest.mark.gpu

TILES = 148 * 32 * 1024  # a 1,024-row tile for every warp of a B200
DIM = 5000
CLAUSES = {  # name: [[(source, lo, hi), ...], ...]; sources: a (4 bytes), b (1), w (8), dimension attribute
    "none": [], "range": [[(0, 100, 600)]], "two": [[(0, 100, 600)], [(1, 20, 90)]], "wide": [[(2, 5, 1 << 40)]],
    "dim": [[(3, 10, 120)]], "range_dim": [[(0, 0, 500)], [(3, 0, 100)]], "or": [[(0, 0, 200), (1, 0, 30)]],
    "or_dim": [[(0, 0, 200), (3, 0, 30)]], "empty": [[(0, 5, 5)]], "past_the_type": [[(1, 250, 1000)]],
}
KEYS = {"one": ([], 1), "shared": ([(1, abi.X_ID, 1, 0, 1)], 200), "global": ([(0, abi.X_ID, 1, 0, 9), (1, abi.X_DIV, 25, 0, 1)], 9000)}


def table(n, seed):
    r = np.random.default_rng(seed)
    t = {"a": r.integers(0, 1000, n).astype(np.uint32), "b": r.integers(0, 225, n).astype(np.uint8),
         "w": r.integers(0, 1 << 41, n).astype(np.uint64), "fk": r.integers(0, DIM + 50, n).astype(np.uint32),
         "d": r.integers(0, 250, DIM).astype(np.uint16)}
    return t


def host_sum(t, n, clauses, keys, ng, va):
    inside = t["fk"][:n] < DIM
    cols = [t["a"][:n], t["b"][:n], t["w"][:n], t["d"][np.minimum(t["fk"][:n], DIM - 1)]]
    ok = np.ones(n, bool)
    for cl in clauses:
        any_ = np.zeros(n, bool)
        for s, lo, hi in cl:
            v = cols[s].astype(np.uint64)
            any_ |= (v >= np.uint64(lo)) & (v < np.uint64(hi)) & (inside if s == 3 else True)
        ok &= any_
    g = np.zeros(n, np.int64)
    for s, xf, div, base, mul in keys:
        v = cols[s].astype(np.int64)
        g += mul * ((v // div if xf == abi.X_DIV else v) - base)
    ok &= g < ng
    out = np.zeros(ng, np.int64)
    np.add.at(out, g[ok], cols[va][ok].astype(np.int64))
    return out, int(ok.sum())


@pytest.fixture(scope="module")
def data():
    t = table(TILES + 1000, 3)
    return t, {k: D.from_host(v) for k, v in t.items()}


def make_op(dev, off, clauses, keys, va):
    c = {k: (v if k == "d" else v[off:]) for k, v in dev.items()}
    return ops.Op(srcs=[ops.Src(c["a"]), ops.Src(c["b"]), ops.Src(c["w"]), ops.Src(c["d"], c["fk"])],
                  clauses=clauses, keys=keys, vkind=abi.V_COL, va=va).to_c()


@pytest.mark.parametrize("n", [1, 33, 100_003, TILES - 1, TILES + 777])
@pytest.mark.parametrize("clause", list(CLAUSES))
def test_sums(mb, cuda, data, clause, n):
    t, dev = data
    L = D.lib()
    for (keys, ng), va in ((KEYS["one"], 0), (KEYS["shared"], 0), (KEYS["shared"], 2), (KEYS["global"], 1)):
        want, rows = host_sum(t, n, CLAUSES[clause], keys, ng, va)
        op = make_op(dev, 0, CLAUSES[clause], keys, va)
        for f in (L.mb_join_grpby, L.mb_hash_join_grpby):
            if f is L.mb_hash_join_grpby and "dim" not in clause:
                continue
            out, nq = D.empty(ng, 8), D.empty(1, 8)
            check(f(n, C.byref(op), ng, out.data_ptr(), nq.data_ptr(), D.stream_ptr()))
            np.testing.assert_array_equal(D.to_host(out, np.int64), want)
            assert int(D.to_host(nq, np.uint64)[0]) == rows


@pytest.mark.parametrize("clause", ["none", "range", "two", "or", "range_dim"])
def test_unaligned_columns(mb, cuda, data, clause):
    t, dev = data
    n = TILES + 500
    keys, ng = KEYS["shared"]
    shifted = {k: (v if k == "d" else v[1:]) for k, v in t.items()}
    want, rows = host_sum(shifted, n, CLAUSES[clause], keys, ng, 0)
    out, nq = D.empty(ng, 8), D.empty(1, 8)
    op = make_op(dev, 1, CLAUSES[clause], keys, 0)
    check(D.lib().mb_join_grpby(n, C.byref(op), ng, out.data_ptr(), nq.data_ptr(), D.stream_ptr()))
    np.testing.assert_array_equal(D.to_host(out, np.int64), want)
    assert int(D.to_host(nq, np.uint64)[0]) == rows


@pytest.mark.parametrize("n", [300_000, TILES])
@pytest.mark.parametrize("clause", ["none", "dim", "or", "or_dim"])
def test_no_slower_than_a_list_of_all_rows(mb, cuda, data, clause, n):
    """Through the screens these took 2 to 5 times as long as row by row, the way
    mb_rows_grpby takes a list of rows to be checked."""
    _, dev = data
    L = D.lib()
    keys, ng = KEYS["shared"]
    op = make_op(dev, 0, CLAUSES[clause], keys, 0)
    rows = cuda.arange(n, dtype=cuda.int64, device="cuda").add_(1 << 31).to(cuda.int32)  # bit 31: check the row
    count = cuda.tensor([n], dtype=cuda.int64, device="cuda")
    bufs = {k: (D.empty(ng, 8), D.empty(1, 8)) for k in ("scan", "list")}
    calls = {"scan": lambda o, q: L.mb_join_grpby(n, C.byref(op), ng, o.data_ptr(), q.data_ptr(), D.stream_ptr()),
             "list": lambda o, q: L.mb_rows_grpby(rows.data_ptr(), count.data_ptr(), n, C.byref(op), ng, o.data_ptr(),
                                                  q.data_ptr(), D.stream_ptr())}
    best = {}
    for rep in range(15):
        for k, f in calls.items():
            a, b = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                check(f(*bufs[k]))
            b.record()
            cuda.cuda.synchronize()
            best[k] = min(best.get(k, 1e9), a.elapsed_time(b) * 100)
    for x, y in zip(bufs["scan"], bufs["list"]):
        assert cuda.equal(x, y)
    assert best["scan"] <= 1.3 * best["list"], best
