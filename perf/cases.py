"""Timed cases of the oblivious operators, each through the call a user makes.

The listed cases are what a user of the library has it do: sorts and
compactions of plain rows, the query pipelines over lineitem-shaped and
dimension/fact tables, the relational operators behind a plan (ORDER BY, join,
GROUP BY, materialization), a planned batch, and a served batch of queries on
the persistent command queue.  Sizes are those of the benchmark's workloads and
tests or round numbers with a ragged remainder.  ``draw`` gives more cases of
the same kinds over the same ranges.

All results are integers (or moved bits), so every output has to be the same
bit for bit.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from velodb_b200 import capi
from velodb_b200._lib import VeloJoinPred, VeloJoinTables, VeloLineitem, VeloLineitemPred

# predicates of the two pipelines (selectivities of about 2 % and 25 %)
LI_PRED = dict(ship_lo=0, ship_hi=2504, disc_lo=10, disc_hi=10, qty_lo=1, qty_hi=11)
LI_PRED_WIDE = dict(ship_lo=100, ship_hi=2400, disc_lo=0, disc_hi=2_000_000_000, qty_lo=1, qty_hi=40)
JOIN_PRED = dict(date_hi=1278, price_hi=5_295_000)
GROUP_BOUND = 8
TOPK = 10

# velo_type numbers
INTEGER, BIGINT, FLOAT, DOUBLE, DATE = 4, 5, 6, 7, 10
ORDERINGS = {
    # one line per ORDER BY list: (type, ascending) of each column
    "price desc, date": ((DOUBLE, False), (DATE, True)),
    "date, quantity desc": ((DATE, True), (INTEGER, False)),
    "key": ((BIGINT, True),),
    "key desc, price, date": ((BIGINT, False), (DOUBLE, True), (DATE, False)),
}


def listed():
    return [
        # an ORDER BY of one small page of rows: launches and latency
        {"name": "sort_1k", "kind": "sort", "n": 1000},
        # the benchmark's plain sort
        {"name": "sort_1m", "kind": "sort", "n": 1 << 20},
        # the benchmark's sort beyond the L2 cache
        {"name": "sort_16m", "kind": "sort", "n": 1 << 24},
        # a WHERE clause that keeps 30 % of a table of some millions of rows
        {"name": "compact_3m", "kind": "compact", "n": 3_000_017, "keep": 0.3},
        # ORDER BY price DESC, date over the 1.5 M-row dimension table
        {"name": "orderby_1_5m", "kind": "orderby", "n": 1_500_000, "order": "price desc, date"},
        # the 6,001,215-row filter + group-by query
        {"name": "filter_groupby_6m", "kind": "filter_groupby", "n": 6_001_215, "wide": False},
        # the headline query: 1.5 M-row dimension, 6 M-row fact, top 10 groups
        {"name": "join_topk_7_5m", "kind": "join_topk", "n_dim": 1_500_000, "n_fact": 6_000_000, "k": TOPK},
        # the join operator: row-id pairs, BIGINT keys, a filter on either side
        {"name": "join_pkfk_1_2m", "kind": "join_pkfk", "n_build": 200_003, "n_probe": 1_000_017, "bigint": True,
         "masks": True},
        # the aggregate operator: GROUP BY a BIGINT key, SUM and COUNT, masked rows
        {"name": "groupby_2m", "kind": "groupby", "n": 2_000_003, "bigint": True, "n_sums": 1, "masks": True},
        # materialization: one column of a 1 M-row table by 500 k row ids
        {"name": "gather_1_5m", "kind": "gather", "n_table": 1_000_000, "n_req": 500_009},
        # 512 independent sorts and compactions of 2^10..2^22 rows, one launch
        {"name": "batch_512", "kind": "batch", "count": 512, "lo": 10.0, "hi": 22.0},
        # a served mix: 48 small queries at once on the persistent command queue
        {"name": "served_48", "kind": "served", "count": 48, "lo": 10.0, "hi": 18.0},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sort", "sort", "compact", "orderby", "filter_groupby", "join_topk", "join_pkfk", "groupby",
                       "gather", "batch", "served"])
    if kind == "sort":
        return {"kind": kind, "n": _log_uniform(rng, 500, 1 << 24)}
    if kind == "compact":
        return {"kind": kind, "n": _log_uniform(rng, 1000, 1 << 23), "keep": round(rng.uniform(0.02, 0.98), 3)}
    if kind == "orderby":
        return {"kind": kind, "n": _log_uniform(rng, 1000, 1 << 22), "order": rng.choice(sorted(ORDERINGS))}
    if kind == "filter_groupby":
        return {"kind": kind, "n": _log_uniform(rng, 1000, 8_000_000), "wide": rng.random() < 0.3}
    if kind == "join_topk":
        nd = _log_uniform(rng, 300, 1_500_000)
        return {"kind": kind, "n_dim": nd, "n_fact": int(nd * rng.uniform(1.0, 4.5)),
                "k": rng.choice([1, 10, 10, 10, 100])}
    if kind == "join_pkfk":
        nb = _log_uniform(rng, 300, 1_000_000)
        return {"kind": kind, "n_build": nb, "n_probe": int(nb * rng.uniform(0.5, 5.0)), "bigint": rng.random() < 0.5,
                "masks": rng.random() < 0.5}
    if kind == "groupby":
        return {"kind": kind, "n": _log_uniform(rng, 1000, 1 << 22), "bigint": rng.random() < 0.5,
                "n_sums": rng.choice([0, 1, 1]), "masks": rng.random() < 0.5}
    if kind == "gather":
        return {"kind": kind, "n_table": _log_uniform(rng, 1000, 2_000_000), "n_req": _log_uniform(rng, 1000, 2_000_000)}
    if kind == "batch":
        return {"kind": kind, "count": _log_uniform(rng, 8, 256), "lo": 10.0, "hi": round(rng.uniform(14.0, 22.0), 2)}
    return {"kind": kind, "count": rng.randrange(8, 65), "lo": 10.0, "hi": round(rng.uniform(14.0, 18.0), 2)}


# ---- inputs -----------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _ints(g, n, lo, hi, dtype):
    """n integers uniform over [lo, hi]."""
    return torch.randint(lo, hi + 1, (n,), generator=g, device="cuda", dtype=torch.int64).to(dtype)


def _u64(g, n):
    return torch.randint(-(2**63), 2**63 - 1, (n,), generator=g, device="cuda", dtype=torch.int64)


def _bernoulli(g, n, p):
    return (torch.rand(n, generator=g, device="cuda") < p).to(torch.uint8)


def _lineitem(g, n):
    return dict(qty=_ints(g, n, 1, 50, torch.int32), price=_ints(g, n, 90_000, 10_500_000, torch.int64),
                disc=_ints(g, n, 0, 10, torch.int32), tax=_ints(g, n, 0, 8, torch.int32),
                shipdate=_ints(g, n, 0, 2556, torch.int32), flag1=_ints(g, n, 0, 2, torch.uint8),
                flag2=_ints(g, n, 0, 1, torch.uint8))


def _join_tables(g, nd, nf):
    return dict(dim_key=(torch.randperm(nd, generator=g, device="cuda") + 1).to(torch.int32),
                dim_date=_ints(g, nd, 0, 2556, torch.int32), fact_fk=_ints(g, nf, 1, nd, torch.int32),
                fact_price=_ints(g, nf, 90_000, 10_500_000, torch.int64))


def _sizes(case):
    """Instance sizes of a batch or a served mix: a fixed spread over the
    case's range, from its own numbers (public sizes, not from the seed)."""
    r = np.random.RandomState(case["count"])
    return np.floor(np.exp2(r.uniform(case["lo"], case["hi"], case["count"]))).astype(np.int64)


def _orderby_columns(g, n, order):
    cols = []
    for t, _ in ORDERINGS[order]:
        if t == DOUBLE:
            cols.append(_ints(g, n, 90_000, 10_500_000, torch.int64).to(torch.float64) / 100.0)
        elif t == DATE:
            cols.append(_ints(g, n, 0, 2556, torch.int32))
        elif t == INTEGER:
            cols.append(_ints(g, n, 1, 50, torch.int32))
        else:
            cols.append(_ints(g, n, -(10**12), 10**12, torch.int64))
    return cols


def _padded(t, cap):
    out = torch.zeros(cap, dtype=t.dtype, device=t.device)
    out[: t.numel()] = t
    return out


def _pow2(n):
    return 1 << max(0, (n - 1).bit_length())


_queue = None


def _served_queue():
    """One persistent queue, as one program keeps it."""
    global _queue
    if _queue is None:
        _queue = capi.Queue(persistent=True)
    return _queue


def _served_slices(case):
    """(shape, offset, rows, dimension offset, dimension rows) of each query
    over tables of 2^20 fact and 2^18 dimension rows."""
    fact_n, dim_n = 1 << 20, 1 << 18
    r = np.random.RandomState(case["count"] + 1)
    out = []
    for i, n in enumerate(int(x) for x in _sizes(case)):
        o = int(r.randint(0, fact_n - n + 1))
        if i % 5 < 3:
            out.append(("filter", o, n, 0, 0))
        else:
            dn = max(1, n // 4)
            out.append(("join", o, n, int(r.randint(0, dim_n - dn + 1)), dn))
    return fact_n, dim_n, out


def _prepare_served(case, g):
    fact_n, dim_n, queries = _served_slices(case)
    li = _lineitem(g, fact_n)
    jt = _join_tables(g, dim_n, fact_n)
    nf = sum(q[0] == "filter" for q in queries)
    s = {"li": li, "jt": jt, "queries": queries, "keep": [], "cmds": [],
         "f_out": torch.zeros((nf, GROUP_BOUND, 6), dtype=torch.int64, device="cuda"),
         "f_counts": torch.zeros((nf, 2), dtype=torch.int64, device="cuda"),
         "j_out": torch.zeros((len(queries) - nf, TOPK, 3), dtype=torch.int64, device="cuda"),
         "j_counts": torch.zeros((len(queries) - nf, 2), dtype=torch.int64, device="cuda")}
    fi = ji = 0
    pred = VeloLineitemPred(*[LI_PRED[k] for k in ("ship_lo", "ship_hi", "disc_lo", "disc_hi", "qty_lo", "qty_hi")])
    jpred = VeloJoinPred(JOIN_PRED["date_hi"], 0, JOIN_PRED["price_hi"])
    for shape, o, n, do, dn in queries:
        if shape == "filter":
            cols = VeloLineitem(*[li[k][o:].data_ptr() for k in capi.LINEITEM_COLS])
            sc = torch.empty(capi.filter_groupby_scratch_bytes(n, GROUP_BOUND), dtype=torch.uint8, device="cuda")
            s["cmds"].append(capi.make_cmd("FILTER_GROUPBY", C.addressof(cols), n, C.addressof(pred), GROUP_BOUND,
                                           s["f_out"][fi], s["f_counts"][fi], sc, sc.numel()))
            fi += 1
            s["keep"].append((cols, pred, sc))
        else:
            tabs = VeloJoinTables(jt["dim_key"][do:].data_ptr(), jt["dim_date"][do:].data_ptr(), dn,
                                  jt["fact_fk"][o:].data_ptr(), jt["fact_price"][o:].data_ptr(), n)
            sc = torch.empty(capi.join_groupby_topk_scratch_bytes(dn, n), dtype=torch.uint8, device="cuda")
            s["cmds"].append(capi.make_cmd("JOIN_GROUPBY_TOPK", C.addressof(tabs), C.addressof(jpred), TOPK,
                                           s["j_out"][ji], s["j_counts"][ji], sc, sc.numel()))
            ji += 1
            s["keep"].append((tabs, jpred, sc))
    torch.cuda.synchronize()  # the queue is not ordered after torch's streams
    s["queue"] = _served_queue()
    return s


def _prepare_batch(case, g):
    sizes = [int(x) for x in _sizes(case)]
    caps = [_pow2(n) for n in sizes]
    rows = sum(caps)
    s = {"keys": _u64(g, rows), "pay": torch.arange(rows, device="cuda", dtype=torch.int32),
         "marks": _bernoulli(g, rows, 0.3), "counts": torch.zeros(len(sizes), dtype=torch.int64, device="cuda")}
    items, off = [], 0
    for i, (n, cap) in enumerate(zip(sizes, caps)):
        it = dict(kind="sort" if i % 2 == 0 else "compact", n=n, keys=s["keys"][off:off + cap],
                  pay=s["pay"][off:off + cap])
        if i % 2 == 1:
            it["marks"] = s["marks"][off:off + cap]
            it["count"] = s["counts"][i:i + 1]
        items.append(it)
        off += cap
    s["items"] = items
    torch.cuda.synchronize()
    s["batch"] = capi.Batch(items)
    return s


def prepare(case, seed):
    g = _gen(seed)
    k = case["kind"]
    if k == "sort":
        n, cap = case["n"], _pow2(case["n"])
        return {"case": case, "keys": _padded(_u64(g, n), cap),
                "pay": _padded(torch.arange(n, device="cuda", dtype=torch.int32), cap)}
    if k == "compact":
        n, cap = case["n"], _pow2(case["n"])
        return {"case": case, "keys": _padded(_u64(g, n), cap),
                "pay": _padded(torch.arange(n, device="cuda", dtype=torch.int32), cap),
                "marks": _padded(_bernoulli(g, n, case["keep"]), cap),
                "scratch": torch.empty(capi.compact_scratch_bytes(cap), dtype=torch.uint8, device="cuda")}
    if k == "orderby":
        cap = _pow2(case["n"])
        return {"case": case, "cols": [_padded(c, cap) for c in _orderby_columns(g, case["n"], case["order"])]}
    if k == "filter_groupby":
        return {"case": case, "cols": _lineitem(g, case["n"]),
                "scratch": torch.empty(capi.filter_groupby_scratch_bytes(case["n"], GROUP_BOUND), dtype=torch.uint8,
                                       device="cuda")}
    if k == "join_topk":
        return {"case": case, "tables": _join_tables(g, case["n_dim"], case["n_fact"]),
                "scratch": torch.empty(capi.join_groupby_topk_scratch_bytes(case["n_dim"], case["n_fact"]),
                                       dtype=torch.uint8, device="cuda")}
    if k == "join_pkfk":
        nb, np_ = case["n_build"], case["n_probe"]
        dt = torch.int64 if case["bigint"] else torch.int32
        bk = torch.randperm(2 * nb, generator=g, device="cuda")[:nb]  # unique, half of the domain
        pk = torch.randint(0, 2 * nb, (np_,), generator=g, device="cuda")
        if case["bigint"]:
            bk, pk = bk * 1_000_003, pk * 1_000_003
        return {"case": case, "bk": bk.to(dt), "pk": pk.to(dt),
                "bm": _bernoulli(g, nb, 0.5) if case["masks"] else None,
                "pm": _bernoulli(g, np_, 0.5) if case["masks"] else None}
    if k == "groupby":
        n = case["n"]
        keys = torch.randint(0, max(2, n // 20), (n,), generator=g, device="cuda")
        keys = (keys * 1_000_003 - 10**9) if case["bigint"] else keys.to(torch.int32)
        return {"case": case, "keys": keys,
                "sums": [_ints(g, n, 90_000, 10_500_000, torch.int64) for _ in range(case["n_sums"])],
                "mask": _bernoulli(g, n, 0.7) if case["masks"] else None}
    if k == "gather":
        return {"case": case, "table": _u64(g, case["n_table"]),
                "rids": torch.randint(0, case["n_table"], (case["n_req"],), generator=g, device="cuda").to(torch.int32),
                "out": torch.empty(case["n_req"], dtype=torch.int64, device="cuda")}
    s = _prepare_batch(case, g) if k == "batch" else _prepare_served(case, g)
    s["case"] = case
    return s


# ---- one pass ---------------------------------------------------------------


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "sort":
        capi.osort_kp(s["keys"], s["pay"], case["n"])
        return s["keys"], s["pay"]
    if k == "compact":
        count = capi.ocompact_kpm(s["keys"], s["pay"], s["marks"], case["n"], scratch=s["scratch"])
        return s["keys"], s["pay"], s["marks"], count
    if k == "orderby":
        spec = ORDERINGS[case["order"]]
        idx = capi.sort_columns(s["cols"], [t for t, _ in spec], [a for _, a in spec], case["n"])
        return s["cols"], idx
    if k == "filter_groupby":
        return capi.filter_groupby(s["cols"], case["n"], LI_PRED_WIDE if case["wide"] else LI_PRED, GROUP_BOUND,
                                   scratch=s["scratch"])
    if k == "join_topk":
        return capi.join_groupby_topk(s["tables"], JOIN_PRED, case["k"], scratch=s["scratch"])
    if k == "join_pkfk":
        return capi.ojoin_pkfk(s["bk"], s["bm"], s["pk"], s["pm"], BIGINT if case["bigint"] else INTEGER)
    if k == "groupby":
        keys, sums, cnt, counts = capi.ogroupby(s["keys"], BIGINT if case["bigint"] else INTEGER, case["n"],
                                                sums=s["sums"], with_count=True, mask=s["mask"])
        return keys, sums, cnt, counts
    if k == "gather":
        capi.ogather_u64(s["table"], case["n_table"], s["rids"], case["n_req"], s["out"])
        return s["out"]
    if k == "batch":
        s["batch"].launch()
        return s["keys"], s["pay"], s["marks"], s["counts"]
    q = s["queue"]
    for t in q.submit_batch(s["cmds"]):
        q.wait(t)
    return s["f_out"], s["f_counts"], s["j_out"], s["j_counts"]


# ---- what a pass cannot do without ------------------------------------------


def _li_bytes(n):
    return n * 26 + GROUP_BOUND * 48 + 16


def _join_bytes(nd, nf, k):
    return nd * 8 + nf * 12 + k * 24 + 16


def work(case):
    """Bytes of each input read once and each output written once; moving and
    comparing keys counts as no floating operations."""
    k = case["kind"]
    if k == "sort":
        b = case["n"] * 24
    elif k == "compact":
        b = case["n"] * 26 + 8
    elif k == "orderby":
        width = sum({DOUBLE: 8, BIGINT: 8}.get(t, 4) for t, _ in ORDERINGS[case["order"]])
        b = case["n"] * (2 * width + 8)
    elif k == "filter_groupby":
        b = _li_bytes(case["n"])
    elif k == "join_topk":
        b = _join_bytes(case["n_dim"], case["n_fact"], case["k"])
    elif k == "join_pkfk":
        w = (8 if case["bigint"] else 4) + (1 if case["masks"] else 0)
        b = (case["n_build"] + case["n_probe"]) * w + case["n_probe"] * 16 + 16
    elif k == "groupby":
        w = (8 if case["bigint"] else 4) + 8 * case["n_sums"] + (1 if case["masks"] else 0)
        b = case["n"] * w + case["n"] * (16 + 8 * case["n_sums"]) + 16
    elif k == "gather":
        b = case["n_table"] * 8 + case["n_req"] * 12
    elif k == "batch":
        b = int(sum(n * (24 if i % 2 == 0 else 26) for i, n in enumerate(_sizes(case))))
    else:
        b = sum(_li_bytes(n) if shape == "filter" else _join_bytes(dn, n, TOPK)
                for shape, _, n, _, dn in _served_slices(case)[2])
    return {"bytes": b, "flops": 0}


def tolerance(case):
    """Integers and moved bits: the same, bit for bit."""
    return "exact"


# ---- the same results by plain torch ----------------------------------------


def _exact_groupby_query(li, pred):
    ok = ((li["shipdate"] >= pred["ship_lo"]) & (li["shipdate"] <= pred["ship_hi"]) & (li["disc"] >= pred["disc_lo"])
          & (li["disc"] <= pred["disc_hi"]) & (li["qty"] >= pred["qty_lo"]) & (li["qty"] <= pred["qty_hi"]))
    c = {k: v[ok].to(torch.int64) for k, v in li.items()}
    key = c["flag1"] * 256 + c["flag2"]
    dp = c["price"] * (100 - c["disc"])
    vals = [torch.ones_like(key), c["qty"], c["price"], dp, dp * (100 + c["tax"])]
    sums = [torch.zeros(65536, dtype=torch.int64, device=key.device).scatter_add_(0, key, v) for v in vals]
    groups = torch.nonzero(sums[0]).reshape(-1)
    out = torch.zeros((GROUP_BOUND, 6), dtype=torch.int64, device=key.device)
    first = groups[:GROUP_BOUND]
    out[: first.numel(), 0] = first
    for i, v in enumerate(sums):
        out[: first.numel(), 1 + i] = v[first]
    counts = torch.tensor([int(ok.sum()), groups.numel()], dtype=torch.int64, device=key.device)
    return out, counts


def _exact_join_query(dim_key, dim_date, fk, price, k):
    top = int(max(dim_key.max(), fk.max())) + 1
    passes = torch.zeros(top, dtype=torch.bool, device=fk.device)
    passes[dim_key.long()] = dim_date < JOIN_PRED["date_hi"]
    joined = passes[fk.long()] & (price < JOIN_PRED["price_hi"])
    f = fk[joined].long()
    sums = torch.zeros(top, dtype=torch.int64, device=fk.device).scatter_add_(0, f, price[joined])
    cnt = torch.bincount(f, minlength=top)
    groups = torch.nonzero(cnt).reshape(-1)
    best = groups[torch.sort(sums[groups], descending=True, stable=True).indices[:k]]
    out = torch.zeros((k, 3), dtype=torch.int64, device=fk.device)
    out[: best.numel()] = torch.stack([best, sums[best], cnt[best]], dim=1)
    counts = torch.tensor([f.numel(), groups.numel()], dtype=torch.int64, device=fk.device)
    return out, counts


def _exact_compact(s, n):
    """ORCompact level by level over the padded rows."""
    cap = s["keys"].numel()
    rows = torch.arange(cap, device="cuda")
    live = rows < n
    key = torch.where(live, s["keys"], -1)
    pay = torch.where(live, s["pay"], -1)
    mark = torch.where(live, s["marks"], 0)
    pre = torch.zeros(cap + 1, dtype=torch.int64, device="cuda")
    pre[1:] = torch.cumsum(mark.long(), 0)
    pos = rows.clone()
    half = 1
    while half < cap:
        start = torch.arange(0, cap, 2 * half, device="cuda")
        off = pre[start] & (2 * half - 1)
        v = pos.view(-1, 2, half)
        if half == 1:
            m = mark[v.reshape(-1, 2)]
            swap = (((m[:, 0] == 0) & (m[:, 1] != 0)) != (off == 1)).view(-1, 1)
        else:
            left = pre[start + half] - pre[start]
            s0 = (((off & (half - 1)) + left) >= half) != (off >= half)
            swap = s0.view(-1, 1) != (torch.arange(half, device="cuda") >= ((off + left) & (half - 1)).view(-1, 1))
        a, b = v[:, 0].clone(), v[:, 1].clone()
        v[:, 0], v[:, 1] = torch.where(swap, b, a), torch.where(swap, a, b)
        half *= 2
    return key[pos], pay[pos], mark[pos], pre[cap:].clone()


def _exact_orderby(cols, spec, n):
    """The bitonic network in its (k, j) order with strict compares, on the
    rank of each row's key; the padding holds max() / lowest()."""
    cap = cols[0].numel()
    top = {DOUBLE: 1.7976931348623157e308, BIGINT: 2**63 - 1, INTEGER: 2**31 - 1, DATE: -1}
    low = {DOUBLE: -1.7976931348623157e308, BIGINT: -(2**63), INTEGER: -(2**31), DATE: 0}
    padded, rank = [], torch.zeros(cap, dtype=torch.int64, device="cuda")
    for c, (t, asc) in zip(cols, spec):
        p = c.clone()
        p[n:] = (top if asc else low)[t]
        padded.append(p)
        v = (p.long() & 0xFFFFFFFF) if t == DATE else p
        u, inv = torch.unique(v, return_inverse=True)
        rank = rank * u.numel() + (inv if asc else u.numel() - 1 - inv)
        rank = torch.unique(rank, return_inverse=True)[1]
    idx = torch.arange(cap, device="cuda")
    k = 2
    while k <= cap:
        j = k // 2
        while j:
            r, i = rank.view(-1, 2, j), idx.view(-1, 2, j)
            asc = ((torch.arange(r.shape[0], device="cuda") * 2 * j) & k).view(-1, 1) == 0
            a, b, x, y = r[:, 0].clone(), r[:, 1].clone(), i[:, 0].clone(), i[:, 1].clone()
            swap = torch.where(asc, a > b, a < b)
            r[:, 0], r[:, 1] = torch.where(swap, b, a), torch.where(swap, a, b)
            i[:, 0], i[:, 1] = torch.where(swap, y, x), torch.where(swap, x, y)
            j //= 2
        k *= 2
    return [p[idx] for p in padded], idx


def exact(case, seed):
    k = case["kind"]
    if k == "batch":
        return None
    s = prepare(case, seed)
    if k == "sort":
        n = case["n"]
        sign = -(2**63)
        order = torch.sort(s["keys"][:n] ^ sign, stable=True).indices  # unsigned order, row ids break ties
        keys, pay = torch.full_like(s["keys"], -1), torch.full_like(s["pay"], -1)
        keys[:n], pay[:n] = s["keys"][:n][order], s["pay"][:n][order]
        return keys, pay
    if k == "compact":
        return _exact_compact(s, case["n"])
    if k == "orderby":
        return _exact_orderby(s["cols"], ORDERINGS[case["order"]], case["n"])
    if k == "filter_groupby":
        return _exact_groupby_query(s["cols"], LI_PRED_WIDE if case["wide"] else LI_PRED)
    if k == "join_topk":
        t = s["tables"]
        return _exact_join_query(t["dim_key"], t["dim_date"], t["fact_fk"], t["fact_price"], case["k"])
    if k == "join_pkfk":
        bk, pk = s["bk"].long(), s["pk"].long()
        order = torch.argsort(bk)
        at = torch.searchsorted(bk[order], pk).clamp(max=bk.numel() - 1)
        hit = bk[order][at] == pk
        if s["bm"] is not None:
            hit &= s["bm"][order][at] != 0
            hit &= s["pm"] != 0
        rows = order[torch.sort(at[hit]).values]  # build rows in key order
        build = torch.full_like(pk, -1)
        build[: rows.numel()] = rows
        counts = torch.tensor([rows.numel(), 0], dtype=torch.int64, device="cuda")
        return build, None, counts  # probe rows of one key come in the network's order
    if k == "groupby":
        take = s["mask"] != 0 if s["mask"] is not None else torch.ones_like(s["keys"], dtype=torch.bool)
        u, inv, c = torch.unique(s["keys"][take].long(), return_inverse=True, return_counts=True)

        def padded(v):
            out = torch.zeros(case["n"], dtype=torch.int64, device="cuda")
            out[: v.numel()] = v
            return out

        sums = [padded(torch.zeros_like(u).scatter_add_(0, inv, v[take])) for v in s["sums"]]
        return padded(u), sums, padded(c), torch.tensor([u.numel(), 0], dtype=torch.int64, device="cuda")
    if k == "gather":
        return s["table"][s["rids"].long()]
    f, j = [], []
    for shape, o, n, do, dn in s["queries"]:
        if shape == "filter":
            f.append(_exact_groupby_query({c: v[o:o + n] for c, v in s["li"].items()}, LI_PRED))
        else:
            t = s["jt"]
            j.append(_exact_join_query(t["dim_key"][do:do + dn], t["dim_date"][do:do + dn], t["fact_fk"][o:o + n],
                                       t["fact_price"][o:o + n], TOPK))
    return (torch.stack([x[0] for x in f]), torch.stack([x[1] for x in f]), torch.stack([x[0] for x in j]),
            torch.stack([x[1] for x in j]))
