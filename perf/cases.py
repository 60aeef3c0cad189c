"""The work a user of this engine has it do, as cases that can be timed.

A case is a dict of plain values.  `prepare` makes what a program holds before
the call (a resident table with its index, bitmaps, streams, a network), `run`
is one pass through the public entry points, `work` the bytes and operations a
pass cannot do without and `exact` its outputs in 64 bits where they are
floating-point numbers (every other output is a whole number: bitmap words,
popcounts, int64 group sums, row counts and stream words).

Kinds of case:

- query:   queries one at a time, host results (Engine.query), on any plan;
- batch:   many queries in one batched scan, host results (Engine.query_batch);
- index:   every level of the six indexed columns into kept buffers
           (mb_bitmap_create_levels);
- flat:    the flat table: three sets of bitmaps (mb_bitmap_create), then one
           virtual bitmap program with its aggregate (mb_vprg_grpby);
- synth:   the synthetic star query, an OR of two fact ranges AND a dimension
           range, counted in 256 groups (mb_vprg_grpby on recipe bitmaps);
- wah:     compression, AND and decompression of WAH streams;
- planner: the learned planner's network, BF16 planning pass and gradients.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from merle_b200 import abi, check, lib
from merle_b200 import device as D
from merle_b200 import ops
from merle_b200 import planner as PL
from merle_b200 import wah as W
from merle_b200 import workload as WL
from merle_b200.engine import Engine

PLAN_KINDS = {"fused": abi.PLAN_FUSED, "scan": abi.PLAN_SCAN, "materialised": abi.PLAN_MATERIALISED,
              "hash": abi.PLAN_HASH}


def listed() -> list[dict]:
    return [
        # the smallest call: a dashboard query against a table that fits in
        # L2; launches and host work count
        {"name": "query_small_300k", "kind": "query", "rows": 300_000, "k": 1, "width4": False, "mix": "ssb13",
         "queries": 13, "mix_seed": 0, "plans": "fused"},
        # the 13 star-schema benchmark queries at scale 20, the reference's
        # column widths, one launch each
        {"name": "query_ssb13_120m", "kind": "query", "rows": 120_000_000, "k": 20, "width4": False, "mix": "ssb13",
         "queries": 13, "mix_seed": 0, "plans": "fused"},
        # the largest single-query load: 64 ad-hoc queries over 600M rows,
        # selectivities from 1e-6 to 0.5, 4-byte columns
        {"name": "query_span_600m", "kind": "query", "rows": 600_000_000, "k": 100, "width4": True, "mix": "span",
         "queries": 64, "mix_seed": 1, "plans": "fused"},
        # the other plan kinds side by side (no index, hash joins, row lists),
        # as a planner's training run or an unindexed table has them
        {"name": "plans_ssb_120m", "kind": "query", "rows": 120_000_000, "k": 20, "width4": False, "mix": "flight1",
         "queries": 4, "mix_seed": 0, "plans": "scan,hash,materialised"},
        # a server's batch at full load: the 64-query mix in one scan, planned
        # by the engine's batch planner network
        {"name": "batch_span_600m", "kind": "batch", "rows": 600_000_000, "k": 100, "width4": True, "mix": "span",
         "queries": 64, "mix_seed": 1, "planner": True},
        # a server's batch at moderate load: 16 mixed queries, ragged row
        # count, the engine's default launch shape
        {"name": "batch_random_24m", "kind": "batch", "rows": 24_000_019, "k": 4, "width4": False, "mix": "random",
         "queries": 16, "mix_seed": 3, "planner": False},
        # loading a table: its 242-bitmap index, two columns through their
        # foreign keys
        {"name": "index_120m", "kind": "index", "rows": 120_000_000, "k": 20, "width4": False},
        # the single-query configuration from raw columns: 214 bitmaps and one
        # program over them, int32 columns
        {"name": "flat_24m", "kind": "flat", "rows": 24_000_000},
        # the synthetic demo: a program with an OR, candidate-checked bins
        {"name": "synth_candchk_60m", "kind": "synth", "rows": 60_000_000, "bits": 16, "recipe": "candchk",
         "permille": 60},
        # the compressed-bitmap baseline on a star query's three predicates
        {"name": "wah_ssb_120m", "kind": "wah", "rows": 120_000_000, "data": "ssb", "order": abi.WAH_MSB},
        # long compressed bitmaps that are mostly runs
        {"name": "wah_sparse_600m", "kind": "wah", "rows": 600_000_000, "data": "sparse", "order": abi.WAH_LSB},
        # planning 2,000 queries at once and a training step's gradients
        {"name": "planner_2k", "kind": "planner", "rows": 2000, "hidden": 64},
    ]


def _logint(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["query", "query", "plans", "batch", "batch", "index", "flat", "synth", "wah", "planner"])
    if kind == "query":
        rows = _logint(rng, 100_000, 300_000_000)
        return {"kind": "query", "rows": rows, "k": max(1, min(50, rows // 6_000_000)),
                "width4": rng.random() < 0.5, "mix": rng.choice(["ssb13", "span", "random"]),
                "queries": rng.randint(1, 24), "mix_seed": rng.randint(1, 1 << 20), "plans": "fused"}
    if kind == "plans":
        rows = _logint(rng, 100_000, 120_000_000)
        return {"kind": "query", "rows": rows, "k": max(1, rows // 6_000_000), "width4": rng.random() < 0.5,
                "mix": rng.choice(["flight1", "random"]), "queries": rng.randint(1, 6),
                "mix_seed": rng.randint(1, 1 << 20),
                "plans": rng.choice(["scan", "hash", "materialised", "scan,hash,materialised"])}
    if kind == "batch":
        rows = _logint(rng, 1_000_000, 400_000_000)
        return {"kind": "batch", "rows": rows, "k": max(1, min(67, rows // 6_000_000)),
                "width4": rng.random() < 0.5, "mix": rng.choice(["span", "random"]),
                "queries": _logint(rng, 2, 96), "mix_seed": rng.randint(1, 1 << 20),
                "planner": rng.random() < 0.5}
    if kind == "index":
        rows = _logint(rng, 100_000, 120_000_000)
        return {"kind": "index", "rows": rows, "k": max(1, rows // 6_000_000), "width4": rng.random() < 0.5}
    if kind == "flat":
        return {"kind": "flat", "rows": _logint(rng, 30_000, 60_000_000)}
    if kind == "synth":
        return {"kind": "synth", "rows": _logint(rng, 30_000, 120_000_000), "bits": rng.choice([8, 16, 32]),
                "recipe": rng.choice(["perfect", "many_or", "candchk"]), "permille": _logint(rng, 2, 300)}
    if kind == "wah":
        return {"kind": "wah", "rows": _logint(rng, 30_000, 600_000_000),
                "data": rng.choice(["ssb", "dense", "sparse", "runs"]),
                "order": rng.choice([abi.WAH_LSB, abi.WAH_MSB])}
    return {"kind": "planner", "rows": _logint(rng, 64, 8192), "hidden": 64}


# ---------------------------------------------------------------- queries
@functools.lru_cache(maxsize=32)
def _mix_tuples(mix: str, n: int, seed: int) -> tuple:
    if mix == "ssb13":
        qs = WL.ssb13()[:n]
    elif mix == "flight1":  # the first query of each benchmark flight
        qs = [WL.ssb13()[i] for i in (0, 3, 6, 10)][:n]
    elif mix == "span":
        qs = WL.span_mix(seed, n)
    else:
        qs = WL.random_mix(seed, n)
    return tuple(WL.as_tuple(q) for q in qs)


def _queries(case: dict) -> list:
    return [abi.query(t, *p) for t, p in _mix_tuples(case["mix"], case["queries"], case["mix_seed"])]


def _engine(case: dict, seed: int) -> Engine:
    e = Engine(0)
    e.gen_star(seed + 1, case["k"], case["rows"], width4=case["width4"])
    e.build_index()
    return e


def _plan(kind: str):
    if kind == "fused":
        return None  # the rule plan
    p = abi.mb_plan()
    p.kind = PLAN_KINDS[kind]
    return p


# ------------------------------------------------------------------ index
YEARS = WL.YEAR_START
INDEX_LEVELS = [  # (column, bounds of each level, coarse to fine)
    ("orderdate", [YEARS, WL.MONTH_START]),
    ("discount", [list(range(12))]),
    ("quantity", [list(range(1, 52))]),
    ("custcity", [list(range(0, 251, 50)), list(range(0, 251, 10))]),
    ("suppcity", [list(range(0, 251, 50)), list(range(0, 251, 10))]),
    ("partmfgr", [list(range(0, 1001, 200)), list(range(0, 1001, 40))]),
]


def _prepare_index(case: dict, seed: int) -> dict:
    n = case["rows"]
    star = D.DevStar(seed + 1, case["k"], n, width4=case["width4"])
    stride = int(lib().mb_bitmap_stride(n))
    passes, slabs, pops, keep = [], [], [], []
    for name, levels in INDEX_LEVELS:
        if name == "custcity":
            src = D.src_of(star.custcity, star["custkey"])
        elif name == "partmfgr":
            src = D.src_of(star.partmfgr, star["partkey"])
        else:
            src = D.src_of(star[name])
        arr = (abi.mb_level * len(levels))()
        for i, b in enumerate(levels):
            lo = np.array(b[:-1], np.uint64)
            hi = np.array(b[1:], np.uint64)
            slab = D.empty(len(lo) * stride, 4, zero=True)
            pop = D.empty(len(lo), 8, zero=True)
            arr[i].lo = lo.ctypes.data_as(C.POINTER(C.c_uint64))
            arr[i].hi = hi.ctypes.data_as(C.POINTER(C.c_uint64))
            arr[i].nbins, arr[i].out, arr[i].popcounts = len(lo), slab.data_ptr(), pop.data_ptr()
            keep += [lo, hi]
            slabs.append(slab)
            pops.append(pop)
        passes.append((src, arr, len(levels)))
    return {"kind": "index", "n": n, "stride": stride, "passes": passes, "slabs": slabs, "pops": pops,
            "keep": (star, keep)}


def _run_index(s: dict):
    L, st = lib(), D.stream_ptr()
    for p in s["pops"]:
        p.zero_()
    for src, arr, nl in s["passes"]:
        check(L.mb_bitmap_create_levels(C.byref(src), s["n"], arr, nl, s["stride"], st))
    return {"bitmaps": s["slabs"], "popcounts": s["pops"]}


# ------------------------------------------------------------------- flat
FLAT_BINS = {"a": (range(0, 1000, 10), 10), "b": (range(64), 1), "c": (range(1, 51), 1)}


def _prepare_flat(case: dict, seed: int) -> dict:
    n = case["rows"]
    f = D.DevFlat(seed + 1, n)
    stride = int(lib().mb_bitmap_stride(n))
    sets, keep = {}, [f]
    for c, (lows, width) in FLAT_BINS.items():
        lo = np.array(list(lows), np.uint64)
        hi = lo + np.uint64(width)
        slab = D.empty(len(lo) * stride, 4, zero=True).view(len(lo), stride)
        sets[c] = (D.src_of(f[c]), lo, hi, slab, D.empty(len(lo), 8, zero=True))
    rows = {c: sets[c][3] for c in sets}
    # a in [200, 450) AND b in {3, 7, 11} AND c < 25: popcount and SUM(e * d)
    prg = ops.Vprg(n, [ops.Col(middle=[rows["a"][j] for j in range(20, 45)]),
                       ops.Col(middle=[rows["b"][j] for j in (3, 7, 11)]),
                       ops.Col(middle=[rows["c"][j] for j in range(24)])],
                   [(abi.ORM, 0, 0, 0), (abi.ANDM, 0, 1, 0), (abi.ANDM, 0, 2, 0)]).to_c()
    op = ops.flat_op(f["a"], f["b"], f["c"], f["d"], f["e"], 200, 450, [3, 7, 11], 0, 25).to_c()
    return {"kind": "flat", "n": n, "stride": stride, "sets": sets, "prg": prg, "op": op,
            "out": D.empty(1, 8), "nq": D.empty(1, 8), "keep": keep}


def _run_flat(s: dict):
    L, st = lib(), D.stream_ptr()
    u64p = C.POINTER(C.c_uint64)
    for src, lo, hi, slab, pop in s["sets"].values():
        pop.zero_()
        check(L.mb_bitmap_create(C.byref(src), s["n"], lo.ctypes.data_as(u64p), hi.ctypes.data_as(u64p), len(lo),
                                 slab.data_ptr(), s["stride"], pop.data_ptr(), st))
    out, nq = D.vprg_grpby(s["prg"], s["op"], 1, None, s["out"], s["nq"])
    return {"bitmaps": [x[3] for x in s["sets"].values()], "popcounts": [x[4] for x in s["sets"].values()],
            "sum": out, "rows": nq}


# ------------------------------------------------------------------ synth
_SYNTH_DT = {8: torch.uint8, 16: torch.int16, 32: torch.int32}
RECIPES = {"perfect": abi.RECIPE_PERFECT, "many_or": abi.RECIPE_MANY_OR, "candchk": abi.RECIPE_CANDCHK}


def _synth_domain(case: dict) -> int:
    return 250 if case["bits"] == 8 else 1000


def _prepare_synth(case: dict, seed: int) -> dict:
    n, dom = case["rows"], _synth_domain(case)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 1)
    dt = _SYNTH_DT[case["bits"]]
    dimsz = max(64, n // 100)
    rnd = lambda hi, m: torch.randint(0, hi, (m,), device="cuda", generator=g, dtype=torch.int32)  # noqa: E731
    a1, a2, fk = rnd(dom, n).to(dt), rnd(dom, n).to(dt), rnd(dimsz, n)
    d1 = torch.arange(dimsz, device="cuda", dtype=torch.int32)
    d2 = rnd(256, dimsz).to(torch.uint8)
    w = max(3, dom * case["permille"] // 1000)
    x = min(dom - w, dom // 5)
    dlo, dhi = dimsz // 10, dimsz // 10 + max(3, dimsz // 3)
    r = abi.mb_recipe()
    r.factsz = n
    preds = [(None, a1, x, x + w), (None, a2, x // 2, x // 2 + w), (fk, d1, dlo, dhi)]
    for i, (key, attr, lo, hi) in enumerate(preds):
        r.nbit[i] = attr.element_size() * 8
        r.min[i], r.max[i], r.dimsz[i] = lo, hi, 0xFFFFFFFF
        r.fk[i] = key.data_ptr() if key is not None else None
        r.attr[i] = attr.data_ptr()
    ins = (abi.mb_instr * abi.MB_MAXNINSTR)()
    for i, t in enumerate([(abi.ORM, 0, 0, 0), (abi.ORM, 0, 1, 0), (abi.ANDM, 0, 2, 0)]):
        ins[i].opcode, ins[i].dstreg, ins[i].src1, ins[i].src2 = t
    owned = _Owned()
    check(lib().mb_recipe_build(C.byref(r), RECIPES[case["recipe"]], ins, C.byref(owned.prg), D.stream_ptr()))
    op = ops.synth_op(a1, a2, fk, d1, d2, x, x + w, x // 2, x // 2 + w, dlo, dhi).to_c()
    return {"kind": "synth", "owned": owned, "op": op, "out": D.empty(256, 8), "nq": D.empty(1, 8),
            "keep": (a1, a2, fk, d1, d2)}


class _Owned:
    """A recipe's program, its bitmaps freed with it."""

    def __init__(self):
        self.prg = abi.mb_owned_vprg()

    def __del__(self):
        lib().mb_owned_vprg_release(C.byref(self.prg))


# -------------------------------------------------------------------- wah
def _wah_bitmaps(case: dict, seed: int) -> list:
    n = case["rows"]
    words = (n + 31) // 32
    if case["data"] == "ssb":  # the predicates of a star query: a year, three discounts, half the quantities
        star = D.DevStar(seed + 1, max(1, n // 6_000_000), n)
        preds = [(D.src_of(star["orderdate"]), 366, 731), (D.src_of(star["discount"]), 1, 4),
                 (D.src_of(star["quantity"]), 1, 25)]
        return [D.bitmap_create(src, n, [lo], [hi], pop=False)[0][0] for src, lo, hi in preds]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 1)
    out = []
    for _ in range(2):
        if case["data"] == "dense":
            b = torch.randint(-2**31, 2**31 - 1, (words,), dtype=torch.int32, device="cuda", generator=g)
        elif case["data"] == "sparse":  # one word in a hundred holds a row
            b = (torch.rand(words, device="cuda", generator=g) < 0.01).to(torch.int32)
        else:  # runs of about a thousand words: clear, set, a pattern
            vals = torch.tensor([0, -1, 0x5555], dtype=torch.int32, device="cuda").repeat(words // 2400 + 1)
            lens = torch.randint(600, 1400, (vals.numel(),), device="cuda", generator=g)
            b = torch.repeat_interleave(vals, lens)[:words].contiguous()
            if b.numel() < words:
                b = torch.cat([b, torch.zeros(words - b.numel(), dtype=torch.int32, device="cuda")])
        if n % 32:
            b[-1] &= (1 << (n % 32)) - 1
        out.append(b)
    return out


def _prepare_wah(case: dict, seed: int) -> dict:
    n = case["rows"]
    bitmaps, groups = _wah_bitmaps(case, seed), W.wah_groups(n)
    # a program that compresses bitmaps of one table keeps its buffers: any
    # stream over n rows has at most one word per 31-bit group
    streams = [D.empty(groups, 4, zero=True) for _ in bitmaps]
    ands = [D.empty(groups, 4, zero=True) for _ in bitmaps[1:]]
    return {"kind": "wah", "n": n, "order": case["order"], "bitmaps": bitmaps, "groups": groups, "streams": streams,
            "ands": ands, "back": D.empty(int(lib().mb_bitmap_stride(n)), 4, zero=True)}


def _run_wah(s: dict):
    L, st, n, g = lib(), D.stream_ptr(), s["n"], s["groups"]
    words = [C.c_uint64() for _ in range(2 * len(s["bitmaps"]) - 1)]
    for b, out, w in zip(s["bitmaps"], s["streams"], words):
        check(L.mb_wah_encode(b.data_ptr(), n, s["order"], out.data_ptr(), g, C.byref(w), st))
    r, rw, k = s["streams"][0], words[0], len(s["bitmaps"])
    for i, out in enumerate(s["ands"]):
        check(L.mb_wah_op(abi.WAH_AND, r.data_ptr(), rw.value, s["streams"][i + 1].data_ptr(), words[i + 1].value, g,
                          out.data_ptr(), g, C.byref(words[k + i]), st))
        r, rw = out, words[k + i]
    check(L.mb_wah_decode(r.data_ptr(), rw.value, s["order"], n, s["back"].data_ptr(), st))
    return {"streams": s["streams"], "ands": s["ands"], "bitmap": s["back"],
            "words": np.array([w.value for w in words], np.int64)}


# ---------------------------------------------------------------- planner
def _planner_arrays(case: dict, seed: int):
    r = np.random.default_rng(seed + 1)
    n, h = case["rows"], case["hidden"]
    x = r.random((n, PL.NF), np.float32)
    t = np.abs(r.normal(0, 0.3, (n, PL.NC))).astype(np.float32)
    mask = (r.random((n, PL.NC)) < 0.9).astype(np.float32)
    shapes = [(h, PL.NF), (h,), (h, h), (h,), (PL.NC, h), (PL.NC,)]
    params = np.concatenate([(r.uniform(-1, 1, s) * math.sqrt(6.0 / s[-1] if len(s) == 2 else 0.01)).ravel()
                             for s in shapes]).astype(np.float32)
    return x, t, mask, params, shapes


def _run_planner(s: dict):
    y = s["net"].forward(s["x"], bf16=True)
    _, g = s["net"].gradients(s["x"], s["t"], s["mask"])
    return {"plan": y, "gradients": g}


def _exact_planner(case: dict, seed: int) -> dict:
    x, t, mask, params, shapes = _planner_arrays(case, seed)
    p, at = [], 0
    for sh in shapes:
        m = int(np.prod(sh))
        p.append(params[at:at + m].astype(np.float64).reshape(sh))
        at += m
    W1, b1, W2, b2, W3, b3 = p
    x, t, mask = x.astype(np.float64), t.astype(np.float64), mask.astype(np.float64)
    h1 = np.maximum(x @ W1.T + b1, 0)
    h2 = np.maximum(h1 @ W2.T + b2, 0)
    y = h2 @ W3.T + b3
    dy = 2 * (y - t) * mask / mask.sum()
    d2 = (dy @ W3) * (h2 > 0)
    d1 = (d2 @ W2) * (h1 > 0)
    g = [d1.T @ x, d1.sum(0), d2.T @ h1, d2.sum(0), dy.T @ h2, dy.sum(0)]
    return {"plan": y, "gradients": np.concatenate([a.ravel() for a in g])}


# ---------------------------------------------------------- prepare and run
def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "query":
        return {"kind": kind, "engine": _engine(case, seed), "queries": _queries(case),
                "plans": [_plan(p) for p in case["plans"].split(",")]}
    if kind == "batch":
        s = {"kind": kind, "engine": _engine(case, seed), "queries": _queries(case)}
        if case["planner"]:
            net = PL.MLP(abi.MB_BATCH_FEATURES, 64, abi.MB_BATCH_CANDIDATES)
            net.set_params(np.fromfile("merle_b200/weights/batch_planner.f32", np.float32))
            check(lib().mb_engine_set_batch_planner(s["engine"].handle, net.handle))
            s["net"] = net
        return s
    if kind == "index":
        return _prepare_index(case, seed)
    if kind == "flat":
        return _prepare_flat(case, seed)
    if kind == "synth":
        return _prepare_synth(case, seed)
    if kind == "wah":
        return _prepare_wah(case, seed)
    x, t, mask, params, _ = _planner_arrays(case, seed)
    net = PL.MLP(PL.NF, case["hidden"], PL.NC)
    net.set_params(params)
    return {"kind": kind, "net": net, "x": x, "t": t, "mask": mask}


def run(s: dict):
    kind = s["kind"]
    if kind == "query":
        sums, rows = [], []
        for plan in s["plans"]:
            for q in s["queries"]:
                out, nq, _ = s["engine"].query(q, plan)
                sums.append(out)
                rows.append(nq)
        return {"sums": np.concatenate(sums), "rows": np.array(rows, np.int64)}
    if kind == "batch":
        out, nq = s["engine"].query_batch(s["queries"])
        return {"sums": out, "rows": nq.astype(np.int64)}
    if kind == "index":
        return _run_index(s)
    if kind == "flat":
        return _run_flat(s)
    if kind == "synth":
        out, nq = D.vprg_grpby(s["owned"].prg.prg, s["op"], 256, None, s["out"], s["nq"])
        return {"counts": out, "rows": nq}
    if kind == "wah":
        return _run_wah(s)
    return _run_planner(s)


def exact(case: dict, seed: int):
    """Only the network computes floating-point numbers; sums are int64."""
    return _exact_planner(case, seed) if case["kind"] == "planner" else None


# ------------------------------------------------------------------- work
_BOUNDS = {"date": (YEARS, WL.MONTH_START), "disc": (range(12),), "qty": (range(1, 52),),
           "ccity": (range(0, 251, 50), range(0, 251, 10)), "scity": (range(0, 251, 50), range(0, 251, 10)),
           "mfgr": (range(0, 1001, 200), range(0, 1001, 40))}


def _cover(col: str, lo: int, hi: int) -> set:
    """The fewest bins (level, bin) that hold [lo, hi) or its complement, the
    finest bins that hold part of it included."""
    levels = [list(b) for b in _BOUNDS[col]]
    dlo, dhi = levels[0][0], levels[0][-1]
    lo, hi = max(lo, dlo), min(hi, dhi)

    def walk(a: int, b: int) -> set:
        got, x = set(), a
        while x < b:
            for li, bs in enumerate(levels):
                j = next((i for i in range(len(bs) - 1) if bs[i] <= x < bs[i + 1]))
                if (bs[j] == x and bs[j + 1] <= b) or li == len(levels) - 1:
                    got.add((col, li, j))
                    x = bs[j + 1]
                    break
        return got

    if lo >= hi or (lo == dlo and hi == dhi):
        return set()
    out = walk(dlo, lo) | walk(hi, dhi)
    inside = walk(lo, hi)
    return inside if len(inside) <= len(out) else out


def _preds(t: int, p: tuple) -> list:
    if t == 1:
        return [("date", p[0], p[1]), ("disc", p[2], p[3]), ("qty", p[4], p[5])]
    if t == 2:
        return [("mfgr", p[0], p[1]), ("scity", p[2], p[3])]
    if t == 3:
        return [("ccity", p[0], p[1]), ("scity", p[2], p[3]), ("date", p[4], p[5])]
    return [("ccity", p[0], p[1]), ("scity", p[2], p[3]), ("mfgr", p[4], p[5]), ("date", p[6], p[7])]


# what a selected row's op reads: the value's columns and the group key's
_PAYLOAD = {1: ("eprice", "disc"), 2: ("mfgr", "date", "revenue"), 3: ("scity", "date", "ccity", "revenue"),
            4: ("scity", "date", "mfgr", "revenue", "scost")}
_GROUPED = {"ccity": 1, "mfgr": 2}  # denormalised per-row attributes: bytes
_NARROW = {"date": 2, "disc": 1, "qty": 1, "scity": 1}
_DOM = {"date": 2556, "disc": 11, "qty": 50, "ccity": 250, "scity": 250, "mfgr": 1000}


def _width(col: str, width4: bool) -> int:
    if col in _GROUPED:
        return _GROUPED[col]
    return 4 if width4 else _NARROW.get(col, 4)


def _sectors(n: int, width: int, frac: float) -> float:
    """Bytes of the 32-byte sectors that hold a selected row."""
    return n * width * (1.0 - (1.0 - min(1.0, frac)) ** (32 // width))


def _index_query_bytes(n: int, width4: bool, qs: list) -> float:
    """Queries answered together: each bitmap word and payload sector once."""
    bins, untouched = set(), {}
    for t, p in qs:
        s = WL.est_selectivity(abi.query(t, *p))
        for col, lo, hi in _preds(t, p):
            bins |= _cover(col, lo, hi)
        for col in _PAYLOAD[t]:
            untouched[col] = untouched.get(col, 1.0) * (1.0 - min(1.0, s))
    return len(bins) * ((n + 31) // 32) * 4 + sum(_sectors(n, _width(c, width4), 1.0 - u)
                                                 for c, u in untouched.items())


def _scan_query_bytes(n: int, width4: bool, t: int, p: tuple) -> float:
    """No index: each predicate's column where the predicates before it
    leave a row, most selective first, then the payload."""
    fr = sorted((max(1e-9, (min(hi, dom + (col == "qty")) - lo) / dom), col) for col, lo, hi in _preds(t, p)
                for dom in (_DOM[col],))
    total, left = 0.0, 1.0
    for f, col in fr:
        w = 4 if col in _GROUPED else _width(col, width4)  # a dimension attribute: its foreign key
        total += _sectors(n, w, left)
        left *= min(1.0, f)
    return total + sum(_sectors(n, _width(c, width4), left) for c in _PAYLOAD[t])


def work(case: dict) -> dict:
    kind = case["kind"]
    n = case["rows"]
    bm = (n + 31) // 32 * 4
    if kind in ("query", "batch"):
        qs = list(_mix_tuples(case["mix"], case["queries"], case["mix_seed"]))
        out = sum(8 * (Engine.ngroups(abi.query(t, *p)) + 1) for t, p in qs)
        if kind == "batch":
            return {"bytes": _index_query_bytes(n, case["width4"], qs) + out, "flops": 0}
        total = 0.0
        for plan in case["plans"].split(","):
            for t, p in qs:
                total += (_scan_query_bytes(n, case["width4"], t, p) if plan in ("scan", "hash")
                          else _index_query_bytes(n, case["width4"], [(t, p)]))
            total += out
        return {"bytes": total, "flops": 0}
    if kind == "index":
        cols = sum(n * (4 if c in ("custcity", "partmfgr") or case["width4"] else
                        D.DevStar.NARROW.get(c, 4)) for c, _ in INDEX_LEVELS)
        k = case["k"]
        dims = 30_000 * k + 2 * 200_000 * (1 + int(math.log2(k)))
        return {"bytes": cols + dims + sum(len(b) - 1 for _, ls in INDEX_LEVELS for b in ls) * bm, "flops": 0}
    if kind == "flat":
        sel = 0.25 * 0.48 * (1 / 3 + 1 / 7 + 1 / 11) / 4.74  # b is Zipf(1) over 64 values
        return {"bytes": 3 * 4 * n + 214 * bm + 2 * _sectors(n, 4, sel), "flops": 0}
    if kind == "synth":
        f = case["permille"] / 1000
        sel = (1 - (1 - f) ** 2) / 3
        nb = {"perfect": 3, "many_or": 9, "candchk": 9}[case["recipe"]]
        return {"bytes": nb * bm + _sectors(n, 4, sel) + max(64, n // 100), "flops": 0}
    if kind == "wah":
        # stream words per 31-bit group, about: literals, plus fills between them
        fracs = {"ssb": (0.99, 0.99, 1.0), "dense": (1.0, 1.0), "sparse": (0.02, 0.02), "runs": (0.35, 0.35)}
        g = (n + 30) // 31 * 4
        ins, res = sum(fracs[case["data"]]), min(fracs[case["data"]])
        # bitmaps in, streams out; the streams in, the result out; the result in, its bitmap out
        return {"bytes": len(fracs[case["data"]]) * bm + g * (2 * ins + 2 * res) + bm, "flops": 0}
    h = case["hidden"]
    per = PL.NF * h + h * h + h * PL.NC
    return {"bytes": 4 * (n * (PL.NF + 3 * PL.NC) + 2 * per), "flops": 8 * n * per}
