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
