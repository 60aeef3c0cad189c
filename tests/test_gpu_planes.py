"""The bit-plane bitmap kernel (csrc/bitmap.cu) on a GPU against the CPU
oracle, one bin set per level: every column width, the value-to-class forms
(a byte column as its own code, lookup table, division, binary search), levels
that nest, cross or leave gaps, the most classes one pass takes and one more,
keys outside the dimension, and row counts around the 4,096-row tile.
Bit-exact, words past the table's end untouched."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from merle_b200 import abi, check, device as D

pytestmark = pytest.mark.gpu

SIZES = [1, 4095, 4096, 4097, 40_961]


def eq(lo, n, w=1):
    a = np.arange(lo, lo + n * w, w, dtype=np.uint64)
    return a, a + np.uint64(w)


def bins(pairs):
    a = np.array(pairs, np.uint64)
    return a[:, 0].copy(), a[:, 1].copy()


LEVELS = {  # name: (element bytes, value domain, levels)
    "byte_direct": (1, 256, [eq(0, 255)]),
    "byte_direct_offset": (1, 60, [eq(3, 50)]),
    "byte_all": (1, 256, [bins([(0, 1), (5, 200), (200, 256)])]),
    "byte_nested": (1, 250, [eq(0, 5, 50), eq(0, 25, 10)]),
    "short_years_months": (2, 2700, [bins([(0, 366), (366, 731), (731, 2557)]),
                                      bins([(0, 31), (31, 60), (60, 366), (366, 400), (400, 731), (731, 2557)])]),
    "gaps": (2, 1200, [bins([(10, 20), (30, 40), (1000, 1100)])]),
    "crossing": (4, 1000, [bins([(0, 300), (300, 700)]), bins([(100, 500), (600, 900)]), eq(0, 10, 100)]),
    "four_levels": (4, 1 << 13, [eq(0, 2, 4096), eq(0, 8, 1024), eq(0, 64, 128), bins([(5, 6), (8000, 8192)])]),
    "most_classes": (4, 300, [eq(7, 254)]),
    "over_one_pass": (4, 300, [eq(7, 255)]),
    "wide_equal": (4, 1 << 32, [eq(1000, 100, 40_000_000)]),
    "wide_search": (4, 1 << 32, [bins([(0, 5), (5, 1 << 20), (1 << 21, 1 << 31), (1 << 31, 1 << 33)])]),
    "wide_two_levels": (4, 1 << 32, [eq(0, 4, 1 << 30), eq(0, 64, 1 << 26)]),
    "eight_bytes": (8, 1 << 50, [eq(1 << 40, 50, 1 << 43)]),
    "eight_bytes_search": (8, 1 << 50, [bins([(3, 1 << 41), (1 << 42, 1 << 49)])]),
    "eight_bytes_table": (8, 900, [eq(100, 30, 20)]),
    "one_range": (4, 5000, [bins([(1000, 3000)])]),
}


def build(src, n, levels, pop):
    """The levels into poisoned slabs: [(words, popcounts)] on the host."""
    L = D.lib()
    W = (n + 31) // 32
    stride = int(L.mb_bitmap_stride(n))
    arr = (abi.mb_level * len(levels))()
    slabs, pops = [], []
    for i, (lo, hi) in enumerate(levels):
        slab = D.empty(len(lo) * stride, 4)
        slab.fill_(0x5A5A5A5A)
        pc = D.empty(len(lo), 8, zero=True)
        arr[i].lo, arr[i].hi = [a.ctypes.data_as(C.POINTER(C.c_uint64)) for a in (lo, hi)]
        arr[i].nbins, arr[i].out = len(lo), slab.data_ptr()
        arr[i].popcounts = pc.data_ptr() if pop else None
        slabs.append(slab.view(len(lo), stride))
        pops.append(pc)
    check(L.mb_bitmap_create_levels(C.byref(src), n, arr, len(levels), stride, D.stream_ptr()))
    out = []
    for s, p in zip(slabs, pops):
        h = D.to_host(s, np.uint32)
        assert np.all(h[:, W:] == 0x5A5A5A5A)
        out.append((h[:, :W], D.to_host(p, np.uint64)))
    return out


@pytest.mark.parametrize("case", list(LEVELS))
@pytest.mark.parametrize("n", SIZES)
def test_levels_match_oracle(orc, mb, cuda, case, n):
    w, dom, levels = LEVELS[case]
    r = np.random.default_rng(n)
    dt = {1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}[w]
    col = r.integers(0, dom, n, dtype=np.uint64).astype(dt)
    col[0] = dt(min(dom, 1 << (8 * w)) - 1)
    s = abi.mb_src()
    s.col, s.width = orc.ptr(col), w
    dev = D.from_host(col)
    for pop in (True, False):
        got = build(D.src_of(dev), n, levels, pop)
        for (lo, hi), (words, pc) in zip(levels, got):
            want, wpop = orc.bitmap_create(s, n, lo, hi)
            np.testing.assert_array_equal(words, want[:, :words.shape[1]])
            np.testing.assert_array_equal(pc, wpop if pop else np.zeros_like(wpop))


@pytest.mark.parametrize("w", [1, 2, 4, 8])
@pytest.mark.parametrize("n", [4096, 40_961])
def test_join_levels_match_oracle(orc, mb, cuda, w, n):
    """Through a foreign key, some keys outside the dimension."""
    r = np.random.default_rng(w)
    dt = {1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}[w]
    dim = r.integers(0, 250, 5000).astype(dt)
    fk = r.integers(0, 5100, n).astype(np.uint32)
    levels = [eq(0, 5, 50), eq(0, 25, 10)]
    s = abi.mb_src()
    s.col, s.width, s.fk, s.dimsz = orc.ptr(dim), w, orc.ptr(fk), len(dim)
    dd, df = D.from_host(dim), D.from_host(fk)
    got = build(D.src_of(dd, df), n, levels, True)
    for (lo, hi), (words, pc) in zip(levels, got):
        want, wpop = orc.bitmap_create(s, n, lo, hi)
        np.testing.assert_array_equal(words, want[:, :words.shape[1]])
        np.testing.assert_array_equal(pc, wpop)
