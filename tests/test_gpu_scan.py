"""GPU parity tests of the scan kernel (mb_join_grpby, mb_hash_join_grpby) at the edges of its
1,024-row tiles and 64-row batches: every
column width and alignment of the range screens, ranges no value or every value meets,
clauses that stay with the op (several terms, foreign keys, 8-byte values), key bits staged
in shared memory and too many for it, a dimension without a passing row, keys outside their
dimension, and the group strategies.  Integer work: bit-exact against the oracle."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from merle_b200 import abi, check, device as D, ops

pytestmark = pytest.mark.gpu

DT = {1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}


def run(fn, n, op, ng):
    out, nq = D.empty(ng, 8), D.empty(1, 8)
    check(getattr(D.lib(), fn)(n, C.byref(op), ng, out.data_ptr(), nq.data_ptr(), D.stream_ptr()))
    return D.to_host(out, np.int64), int(D.to_host(nq, np.uint64)[0])


def same(got, want, what):
    np.testing.assert_array_equal(got[0], want[0], err_msg=str(what))
    assert got[1] == want[1], what


@pytest.mark.parametrize("n", [1, 31, 127, 128, 1023, 1024, 1025, 148 * 1024, 148 * 1024 * 32 + 5, 2_000_003])
def test_scan_sizes_and_clauses(orc, cuda, n):
    """Row counts around the tile, one tile a block and one a warp; per size: two
    screens, one of several terms, one through a key, all rows, no row."""
    rng = np.random.default_rng(n)
    a = rng.integers(0, 256, n).astype(np.uint8)
    b = rng.integers(0, 1000, n).astype(np.uint16)
    v = rng.integers(0, 1 << 31, n).astype(np.uint32)
    dim = rng.integers(0, 25, 300).astype(np.uint8)
    fk = rng.integers(0, 310, n).astype(np.uint32)  # some keys outside the dimension
    dev = [D.from_host(x) for x in (a, b, v, dim, fk)]
    for clauses in ([[(0, 40, 140)], [(1, 0, 500)]], [[(1, 10, 20), (0, 3, 4)]], [[(3, 5, 20)], [(0, 0, 200)]], [],
                    [[(0, 256, 300)]], [[(0, 9, 9)]], [[(0, 0, 1 << 40)], [(1, 0, 65536)]], [[(0, 0, 256)], [(3, 30, 40)]]):
        def op(c):
            return ops.Op(srcs=[ops.Src(c[0]), ops.Src(c[1]), ops.Src(c[2]), ops.Src(c[3], c[4])], clauses=clauses,
                          keys=[(3, abi.X_ID, 1, 0, 1)], vkind=abi.V_COL, va=2).to_c()
        want = orc.join_grpby(n, op((a, b, v, dim, fk)), 25)
        for fn in ("mb_join_grpby", "mb_hash_join_grpby"):
            same(run(fn, n, op(dev), 25), want, (fn, clauses))


@pytest.mark.parametrize("width", [1, 2, 4, 8])
@pytest.mark.parametrize("offset", [0, 1, 3])
def test_scan_screen_widths_and_alignment(orc, cuda, width, offset):
    """A screen of each width on an aligned column and on ones that no vector
    load may read; the values reach the width's largest."""
    n = 1024 * 9 + 77
    rng = np.random.default_rng(width * 10 + offset)
    top = (1 << (8 * width)) - 1
    a = rng.integers(0, 1 << 8, n + offset).astype(DT[width])
    a[::7] = top
    v = rng.integers(0, 1 << 20, n + offset).astype(DT[max(width, 4)])
    d = [D.from_host(x)[offset:] for x in (a, v)]
    h = [np.ascontiguousarray(x[offset:]) for x in (a, v)]
    for lo, hi in ((0, 100), (top, top + 1 if width < 8 else top), (200, 1 << 63), (1, 2)):
        def op(c):
            return ops.Op(srcs=[ops.Src(c[0]), ops.Src(c[1])], clauses=[[(0, lo, hi)]],
                          keys=[(1, abi.X_DIV, 1 << 15, 0, 1)], vkind=abi.V_COL, va=1).to_c()
        same(run("mb_join_grpby", n, op(d), 32), orc.join_grpby(n, op(h), 32), (lo, hi))


@pytest.mark.parametrize("ng,dimsz", [(1, 33), (200, 4097), (9000, 100_000), (200, 1_200_001)])
def test_hash_key_bits(orc, cuda, ng, dimsz):
    """Two dimensions: few keys and many (more key bits than a block stages at
    1.2M rows), two attributes on one key, an empty filter, unaligned keys."""
    n = 300_007
    rng = np.random.default_rng(dimsz)
    d1 = rng.integers(0, 200, 40).astype(np.uint8)
    d2 = rng.integers(0, 10_000, dimsz).astype(np.uint16)
    d3 = rng.integers(0, 1 << 30, dimsz).astype(np.uint32)
    k1 = rng.integers(0, 41, n + 1).astype(np.uint32)
    k2 = rng.integers(0, dimsz + 5, n + 1).astype(np.uint32)
    f = rng.integers(0, 1 << 20, n + 1).astype(np.uint32)
    cols = (d1, d2, d3, k1, k2, f)
    for off in (0, 1):
        h = [np.ascontiguousarray(x[off:]) if x.size > n else x for x in cols]
        t = [D.from_host(x)[off:] if x.size > n else D.from_host(x) for x in cols]
        for c1, c2 in (((0, 100), (0, 5000)), ((250, 255), (0, 5000)), ((0, 200), (0, 1)), ((7, 8), (0, 1 << 33))):
            def op(c):
                return ops.Op(srcs=[ops.Src(c[0], c[3]), ops.Src(c[1], c[4]), ops.Src(c[2], c[4]), ops.Src(c[5])],
                              clauses=[[(1, *c2)], [(3, 1000, 1 << 19)], [(0, *c1)], [(2, 0, 1 << 29), (3, 0, 500_000)]],
                              keys=[(1, abi.X_ID, 1, 0, 1)] if ng > 1 else [], vkind=abi.V_SUB, va=2, vb=3).to_c()
            same(run("mb_hash_join_grpby", n - off, op(t), ng), orc.join_grpby(n - off, op(h), ng), (off, c1, c2))
