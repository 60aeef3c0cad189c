"""Many bins of a small table in the plane kernel: its codes are shared out over warps that
have no tile of their own."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from merle_b200 import abi, check, device as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1023, 1025, 33_000, 150_000, 900_001])
@pytest.mark.parametrize("w,first,nb", [(1, 0, 255), (1, 3, 9), (1, 7, 248), (2, 0, 254), (4, 5, 129), (8, 1, 17)])
def test_split_codes(orc, mb, cuda, n, w, first, nb):
    """Every split from one code group a CTA row to none, first codes inside a group,
    with and without row counts."""
    r = np.random.default_rng(n + nb)
    col = r.integers(0, 256, n).astype({1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}[w])
    lo = np.arange(first, first + nb, dtype=np.uint64)
    s = abi.mb_src()
    s.col, s.width = orc.ptr(col), w
    want, wpop = orc.bitmap_create(s, n, lo, lo + np.uint64(1))
    dev = D.from_host(col)
    for pop in (True, False):
        words, pc = D.bitmap_create(D.src_of(dev), n, lo, lo + np.uint64(1), pop=pop)
        np.testing.assert_array_equal(D.to_host(words, np.uint32)[:, :(n + 31) // 32], want[:, :(n + 31) // 32])
        if pop:
            np.testing.assert_array_equal(D.to_host(pc, np.uint64), wpop)


def test_many_bins_cost_a_small_table_little(mb, cuda):
    """300K rows, 250 bins against 16, with row counts: 19 us against 13; one warp for all codes of a
    tile took 31.  The least of 15 runs; the line half way."""
    n = 300_000
    g = cuda.Generator(device="cuda")
    g.manual_seed(1)
    col = cuda.randint(0, 250, (n,), device="cuda", generator=g, dtype=cuda.int32)
    L, s, stride = D.lib(), D.src_of(col), int(D.lib().mb_bitmap_stride(n))
    u64p, best = C.POINTER(C.c_uint64), {}
    for _ in range(15):
        for nb in (16, 250):
            lo = np.arange(nb, dtype=np.uint64)
            hi = lo + np.uint64(1)
            slab, pop = D.empty(nb * stride, 4), D.empty(nb, 8, zero=True)
            a, b = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                check(L.mb_bitmap_create(C.byref(s), n, lo.ctypes.data_as(u64p), hi.ctypes.data_as(u64p), nb,
                                         slab.data_ptr(), stride, pop.data_ptr(), D.stream_ptr()))
            b.record()
            cuda.cuda.synchronize()
            best[nb] = min(best.get(nb, 1e9), a.elapsed_time(b) * 50)
    assert best[250] <= 1.95 * best[16], best
