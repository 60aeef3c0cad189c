"""The bit-plane bitmap kernel at four words a lane, the form of tables of
8,000,000 rows and more: every form of its levels, columns and dimensions, at
row counts that end on and around a 4,096-row tile, a lane's four words and a
word.  Bit-exact against the same rows taken in two parts of less than
8,000,000 (one word a lane, compared with the CPU oracle in test_gpu_planes.py), and the
last rows against the oracle itself; words past the table's end untouched."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from merle_b200 import abi, check, device as D
from tests.test_gpu_planes import LEVELS, eq

pytestmark = pytest.mark.gpu

CUT = 4_194_304      # the second part starts here: whole tiles, words and 16-byte loads
TAIL = 32 * 300
POISON = 0x5A5A5A5A
# the rows of the last tile are 512 (whole words, lanes of four), 545 (a lane of two
# words, the last of one row), 639, 4,096 and 1
SIZES = [8_000_000, 8_000_033, 8_000_127, 8_003_584, 8_003_585]


def build(src, n, levels):
    """The levels into poisoned slabs on the device: [(slab, popcounts)]."""
    L = D.lib()
    stride = int(L.mb_bitmap_stride(n))
    arr = (abi.mb_level * len(levels))()
    out = []
    for i, (lo, hi) in enumerate(levels):
        slab = D.empty(len(lo) * stride, 4)
        slab.fill_(POISON)
        pc = D.empty(len(lo), 8, zero=True)
        arr[i].lo, arr[i].hi = [a.ctypes.data_as(C.POINTER(C.c_uint64)) for a in (lo, hi)]
        arr[i].nbins, arr[i].out, arr[i].popcounts = len(lo), slab.data_ptr(), pc.data_ptr()
        out.append((slab.view(len(lo), stride), pc))
    check(L.mb_bitmap_create_levels(C.byref(src), n, arr, len(levels), stride, D.stream_ptr()))
    return out


def compare(orc, torch, n, levels, dev_src, host_src):
    """dev_src / host_src(first row): the column from that row on."""
    W = (n + 31) // 32
    whole = build(dev_src(0), n, levels)
    head, rest = build(dev_src(0), CUT, levels), build(dev_src(CUT), n - CUT, levels)
    t0 = (n - TAIL) // 32 * 32
    for (lo, hi), (words, pc), (hw, hp), (rw, rp) in zip(levels, whole, head, rest):
        assert torch.equal(words[:, :CUT // 32], hw[:, :CUT // 32])
        assert torch.equal(words[:, CUT // 32:W], rw[:, :W - CUT // 32])
        assert bool((words[:, W:] == POISON).all())
        assert torch.equal(pc, hp + rp)
        want, _ = orc.bitmap_create(host_src(t0), n - t0, lo, hi)
        np.testing.assert_array_equal(D.to_host(words[:, t0 // 32:W].contiguous(), np.uint32), want[:, :W - t0 // 32])


@pytest.mark.parametrize("case", list(LEVELS))
@pytest.mark.parametrize("n", SIZES)
def test_levels_four_words_a_lane(orc, mb, cuda, case, n):
    w, dom, levels = LEVELS[case]
    r = np.random.default_rng(n)
    col = r.integers(0, dom, n, dtype=np.uint64).astype({1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}[w])
    dev = D.from_host(col)

    def host(r0):
        s = abi.mb_src()
        s.col, s.width = orc.ptr(col[r0:]), w
        return s
    compare(orc, cuda, n, levels, lambda r0: D.src_of(dev[r0:]), host)


@pytest.mark.parametrize("w", [1, 2, 4, 8])
@pytest.mark.parametrize("form", ["fine", "two", "any", "search"])
@pytest.mark.parametrize("n", SIZES[1::2])
def test_join_levels_four_words_a_lane(orc, mb, cuda, w, form, n):
    """Through a foreign key, some keys outside the dimension."""
    levels = {"fine": [eq(3, 200)], "two": [eq(0, 5, 50), eq(0, 25, 10)], "any": [eq(0, 5, 50), eq(20, 30, 7)],
              "search": [eq(0, 5, 1 << 30)]}[form]
    r = np.random.default_rng(w)
    dim = r.integers(0, 250 if form != "search" or w < 4 else 1 << 32, 5000, dtype=np.uint64)
    dim = dim.astype({1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}[w])
    fk = r.integers(0, 5100, n).astype(np.uint32)
    dd, df = D.from_host(dim), D.from_host(fk)

    def host(r0):
        s = abi.mb_src()
        s.col, s.width, s.fk, s.dimsz = orc.ptr(dim), w, orc.ptr(fk[r0:]), len(dim)
        return s
    compare(orc, cuda, n, levels, lambda r0: D.src_of(dd, df[r0:]), host)
