"""The WAH kernels (csrc/wah.cu) around their block edges: blocks of 4,096 groups
(126,976 rows, 3,968 words), threads of 32 groups, 4,096 stream words a block of
the group scan; runs across many blocks, streams that are not canonical or end
early, misaligned bitmaps, and more blocks than a pass sums itself.  Against the
oracle, word for word."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from merle_b200 import abi, check, device as D
from merle_b200 import wah as W
from tests.test_gpu_wah import FILL, ONES, dev32, host32, random_bitmap

pytestmark = pytest.mark.gpu

BLOCK = 31 * 4096


@pytest.mark.parametrize("kind", ["dense", "sparse", "runs", "zero", "one"])
@pytest.mark.parametrize("nrows", [992, 993, BLOCK - 31, BLOCK, BLOCK + 1, 3 * BLOCK + 17])
def test_block_edges(orc, cuda, kind, nrows):
    rng = np.random.default_rng(nrows)
    bm = random_bitmap(rng, nrows, kind)
    for order in (abi.WAH_LSB, abi.WAH_MSB):
        want = orc.wah_encode(bm, nrows, order)
        np.testing.assert_array_equal(host32(W.wah_compress(dev32(bm), nrows, order)), want)
        back = host32(W.wah_decompress(dev32(want), nrows, order))
        np.testing.assert_array_equal(back, bm[:len(back)])


def test_long_runs_and_misaligned_bitmap(orc, cuda):
    """A few set rows among runs of hundreds of blocks; the bitmap at a 4-byte
    boundary."""
    nrows = 400 * BLOCK + 5
    words = (nrows + 31) // 32
    bm = np.zeros((words + 31) // 32 * 32, np.uint32)
    bm[5], bm[3968 * 100 - 1], bm[3968 * 350] = 1, 0x80000000, 1
    bm[3968 * 120:3968 * 300] = 0xFFFFFFFF
    want = orc.wah_encode(bm, nrows, 0)
    shifted = dev32(np.concatenate([np.zeros(1, np.uint32), bm]))[1:]
    np.testing.assert_array_equal(host32(W.wah_compress(shifted, nrows, 0)), want)
    back = host32(W.wah_decompress(dev32(want), nrows, 0))
    np.testing.assert_array_equal(back, bm[:len(back)])


def streams(rng, G):
    """A stream of literals, 0 and 1 fills, with literal 0 and all-one words and
    fills of no group among them, cut or extended against G groups."""
    out, g = [], 0
    while g < G:
        k = rng.integers(0, 7)
        n = int(rng.choice([1, 2, 31, 33, 400, 9000]))
        if k == 0:
            out.append(FILL | n)
            g += n
        elif k == 1:
            out.append(FILL | ONES | n)
            g += n
        elif k == 2:
            out += [FILL, FILL | ONES]
        elif k == 3:
            out.append(int(rng.choice([0, 0x7FFFFFFF])))
            g += 1
        else:
            m = int(rng.choice([1, 40, 5000]))
            out += list(rng.integers(1, 0x7FFFFFFF, m))
            g += m
    return np.array(out, np.uint64).astype(np.uint32)


@pytest.mark.parametrize("seed", range(6))
def test_ops_on_any_stream(orc, cuda, seed):
    rng = np.random.default_rng(seed)
    G = int(rng.integers(1, 60_000))
    a, b = streams(rng, G), streams(rng, max(1, G // 2))
    for g in (1, G // 3 + 1, G, G + 5000):
        for op in (abi.WAH_AND, abi.WAH_OR, abi.WAH_XOR):
            want = orc.wah_op(op, a, b, g)
            for method in (abi.WAH_AUTO, abi.WAH_EXPLICIT, abi.WAH_DIRECT):
                got = host32(W._op(op, dev32(a), dev32(b), g, method=method))
                np.testing.assert_array_equal(got, want, err_msg=f"op {op} groups {g} method {method}")
        nrows = 31 * g - 3
        np.testing.assert_array_equal(host32(W.wah_decompress(dev32(a), nrows, 0)),
                                      orc.wah_decode(a, nrows, 0)[:int(D.lib().mb_bitmap_stride(nrows))])


def test_small_output_and_sizes(orc, cuda):
    """An output smaller than the groups but large enough for the stream."""
    L, nrows = D.lib(), 3 * BLOCK
    bm = random_bitmap(np.random.default_rng(1), nrows, "sparse")
    want = orc.wah_encode(bm, nrows, 0)
    out, n = D.empty(len(want), 4), C.c_uint64()
    check(L.mb_wah_encode(dev32(bm).data_ptr(), nrows, 0, out.data_ptr(), len(want), C.byref(n), D.stream_ptr()))
    assert n.value == len(want)
    np.testing.assert_array_equal(host32(out), want)


def test_more_blocks_than_a_direct_sum(cuda):
    """1.1G rows: 8,664 group blocks (their counts take the scan pass)."""
    T = D.torch()
    nrows = 1_100_000_000
    words = (nrows + 31) // 32
    g = T.Generator(device="cuda")
    g.manual_seed(5)
    bm = T.randint(-2**31, 2**31 - 1, (words,), dtype=T.int32, device="cuda", generator=g)
    bm[words // 3:words // 2] = 0
    w = W.wah_compress(bm, nrows)
    back = W.wah_decompress(w, nrows)
    assert T.equal(back[:words], bm) and not back[words:].any()
    assert W.wah_ngroups(w) == W.wah_groups(nrows)
