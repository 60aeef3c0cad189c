"""Launches of mb_vprg_grpby at the limits of the fused kernels, against sums taken
on the host: shared group tables that fill a CTA's shared memory."""
from __future__ import annotations

import numpy as np
import pytest

from merle_b200 import abi, device as D, ops

pytestmark = pytest.mark.gpu


def launch(**kw):
    la = abi.mb_launch()
    for k, v in kw.items():
        setattr(la, k, v)
    return la


# A CTA has 232,448 bytes.  The general kernel takes 8 a group, 2,048 V a warp for its
# row lists (V words a lane; 8 warps) and 512; the warp-independent one 4,352 a warp
# for its queue instead.
@pytest.mark.parametrize("words,groups,offset", [
    (1, 26_000, 0),   # 208,000 + 16,384, against 208,000 + 34,816
    (2, 24_700, 0),   # 197,600 + 32,768, against 197,600 + 34,816
    (0, 26_000, 4),   # bitmaps off the 16-byte grid: one word a lane
    (0, 20_000, 0),   # both fit
])
def test_general_program_beside_a_large_shared_table(mb, cuda, words, groups, offset):
    n = 50_003
    r = np.random.default_rng(groups + words)
    key, val = r.integers(0, groups, n).astype(np.uint32), r.integers(0, 1 << 32, n).astype(np.uint32)
    sel = r.random((2, n)) < 0.3
    bits = [np.packbits(s, bitorder="little") for s in sel]
    stride = (n + 31) // 32 + 8
    bm = []
    for b in bits:
        w = np.zeros(stride * 4, np.uint8)
        w[offset:offset + len(b)] = b
        bm.append(D.from_host(w.view(np.uint32))[offset // 4:])
    dk, dv = D.from_host(key), D.from_host(val)
    prg = ops.Vprg(n, [ops.Col(middle=[b]) for b in bm], [(abi.ORM, 0, 0, 0), (abi.ORM, 0, 1, 0)]).to_c()
    op = ops.Op(srcs=[ops.Src(dk), ops.Src(dv)], keys=[(0, abi.X_ID, 1, 0, 1)], vkind=abi.V_COL, va=1).to_c()
    rows = np.nonzero(sel[0] | sel[1])[0]
    want = np.zeros(groups, np.int64)
    np.add.at(want, key[rows], val[rows].astype(np.int64))
    out, nq = D.vprg_grpby(prg, op, groups, launch(grp_strategy=abi.GRP_SHARED, words_per_lane=words))
    np.testing.assert_array_equal(D.to_host(out, np.int64), want)
    assert int(D.to_host(nq, np.uint64)[0]) == len(rows)


@pytest.mark.parametrize("chk", [False, True])
@pytest.mark.parametrize("instrs", [[(abi.ORM, 0, 0, 0)], [(abi.ORM, 0, 0, 0), (abi.ORM, 0, 1, 0)]])
def test_rows_past_2_31(mb, cuda, chk, instrs):
    """Row numbers of 32 bits, conjunctive and general programs.  Without candidate checks the
    warp-independent kernel takes them: 24,000 groups fit beside its queues (192,000 +
    34,816 bytes) and not beside the general kernel's lists of four words a lane
    (65,536); with checks the general kernel does, with a smaller table."""
    n = (1 << 31) + 100_003
    groups = 1000 if chk else 24_000
    words = (n + 31) // 32
    bm = [D.empty(words + 8, 4, zero=True) for _ in range(2)]
    r = np.random.default_rng(7)
    rows = [np.unique(np.concatenate([r.integers(0, n, 3000), np.array(x)])) for x in
            ([0, (1 << 31) - 1, 1 << 31, n - 1], [5, (1 << 31) + 77, n - 2])]
    for b, q in zip(bm, rows):
        w, at = np.unique(q // 32, return_inverse=True)
        v = np.zeros(len(w), np.uint32)
        np.bitwise_or.at(v, at, np.uint32(1) << (q % 32).astype(np.uint32))
        b[cuda.from_numpy(w).cuda()] = cuda.from_numpy(v.view(np.int32)).cuda()
    col = D.empty(n, 1, zero=True)
    sel = rows[0] if len(instrs) == 1 else np.union1d(rows[0], rows[1])
    val = (sel % 251).astype(np.uint8)
    col[cuda.from_numpy(sel).cuda()] = cuda.from_numpy(val).cuda()
    cols = [ops.Col(middle=[b]) for b in bm]
    if chk:  # the first operand's rows are candidates of 10 <= value < 200
        cols[0] = ops.Col(leftmost=bm[0])
    prg = ops.Vprg(n, cols, instrs).to_c()
    op = ops.Op(srcs=[ops.Src(col)], clauses=[[(0, 10, 200)]], keys=[(0, abi.X_ID, 1, 0, 1)], vkind=abi.V_ONE).to_c()
    sure = np.isin(sel, rows[1]) if len(instrs) == 2 else np.zeros(len(sel), bool)
    keep = (sure | ((val >= 10) & (val < 200))) if chk else np.ones(len(sel), bool)
    want = np.bincount(val[keep], minlength=groups)
    out, nq = D.vprg_grpby(prg, op, groups, launch(grp_strategy=abi.GRP_SHARED))
    np.testing.assert_array_equal(D.to_host(out, np.int64), want)
    assert int(D.to_host(nq, np.uint64)[0]) == int(keep.sum())
