"""GPU parity of the trimmed and narrow-row paths at the sizes and values where
they can go wrong: the ends of tiles and of the trimmed blocks, keys and
prices at the ends of their types, repeated keys, and both sides of the rules
that choose a path.  Everything is integer, so the comparison is bit for bit."""
import numpy as np
import pytest
import torch

from velodb_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu

INTEGER, BIGINT, DOUBLE, DATE, SMALLINT = 4, 5, 7, 10, 3


# ---- trimmed sorts: one row around a tile (512 and 1024 rows for small sorts),
# ---- around 2^18 (the smaller tile's last size), in the last block of several
# ---- phases, and in the three-CTA form
@pytest.mark.parametrize("n", [3, 511, 512, 513, 1023, 1024, 1025, 2049, 4097, 6144, 6145, 12_289, (1 << 17) + 1, (1 << 18) - 2048, (1 << 18) + 1,
                               3 << 17, (3 << 17) + 4096, (1 << 19) + 4095, (1 << 20) + 1, 1_572_865, (1 << 21) + 5])
def test_trimmed_sort_and_padding(cuda, n):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    cap = capi.next_pow2(n)
    keys = torch.randint(-2**63, 2**63 - 1, (cap,), generator=g, device="cuda")
    keys[: n // 7] = -1  # the padding's own key
    keys[n // 3: n // 2] = 5
    pay = torch.randint(-2**31, 2**31 - 1, (cap,), generator=g, device="cuda").to(torch.int32)
    k, p = keys.clone(), pay.clone()
    capi.osort_kp(k, p, n)
    u = pay[:n].to(torch.int64) & 0xFFFFFFFF
    o = torch.argsort(u, stable=True)
    o = o[torch.argsort((keys[:n] ^ -2**63)[o], stable=True)]
    assert torch.equal(k[:n], keys[:n][o]) and torch.equal(p[:n], pay[:n][o])
    assert bool((k[n:] == -1).all()) and bool((p[n:] == -1).all())


def li_columns(n, seed, flags):
    rng = np.random.default_rng(seed)
    c = W.lineitem(n, seed=seed)
    c["flag1"] = rng.choice(np.array([f >> 8 for f in flags], np.uint8), n)
    c["flag2"] = rng.choice(np.array([f & 255 for f in flags], np.uint8), n)
    return c


def li_expected(c, pred, G):
    ok = ((c["shipdate"] >= pred["ship_lo"]) & (c["shipdate"] <= pred["ship_hi"]) & (c["disc"] >= pred["disc_lo"])
          & (c["disc"] <= pred["disc_hi"]) & (c["qty"] >= pred["qty_lo"]) & (c["qty"] <= pred["qty_hi"]))
    v = {k: x[ok].astype(np.int64) for k, x in c.items()}
    key = v["flag1"] * 256 + v["flag2"]
    uk, inv = np.unique(key, return_inverse=True)
    dp = v["price"] * (100 - v["disc"])
    out = np.zeros((G, 6), np.int64)
    m = min(G, len(uk))
    for i, x in enumerate([np.ones_like(key), v["qty"], v["price"], dp, dp * (100 + v["tax"])]):
        s = np.zeros(len(uk), np.int64)
        np.add.at(s, inv, x)
        out[:m, 1 + i] = s[:m]
    out[:m, 0] = uk[:m]
    return out, [int(ok.sum()), len(uk)]


ALL = dict(ship_lo=0, ship_hi=2556, disc_lo=0, disc_hi=10, qty_lo=1, qty_hi=50)


# key 0xFFFF is also the mark of a row that fails; 256 x 256 keys overflow every
# bound; sizes around the key pairs' tile (2 x 16,384 rows) and its multiples
@pytest.mark.parametrize("n", [1, 2, 3, 4097, 32_767, 32_769, 65_537, 98_305, 300_001])
@pytest.mark.parametrize("flags,G", [((0, 0xFFFF), 8), ((0xFFFF,), 1), (tuple(range(0, 65536, 257)), 16),
                                     ((0x00FF, 0x0100, 0xFF00, 0xFFFF), 9)])
def test_filter_groupby_keys(cuda, n, flags, G):
    c = li_columns(n, n + G, flags)
    d = capi.lineitem_to_device(c)
    for pred in (ALL, W.LINEITEM_PRED, dict(ALL, qty_hi=0)):
        out, counts = capi.filter_groupby(d, n, pred, G)
        want, wc = li_expected(c, pred, G)
        assert np.array_equal(out.cpu().numpy(), want) and counts.tolist() == wc


def test_filter_groupby_wide_values(cuda):
    n = 70_001
    rng = np.random.default_rng(5)
    c = li_columns(n, 9, (1, 2, 3))
    c["price"] = rng.integers(-2**62, 2**62, n)  # sums wrap modulo 2^64
    c["qty"] = rng.integers(-2**31, 2**31, n).astype(np.int32)
    c["disc"] = rng.integers(-2**31, 2**31, n).astype(np.int32)
    pred = dict(ALL, disc_lo=-2**31, disc_hi=2**31 - 1, qty_lo=-2**31, qty_hi=2**31 - 1)
    with np.errstate(over="ignore"):
        want, wc = li_expected(c, pred, 8)
    out, counts = capi.filter_groupby(capi.lineitem_to_device(c), n, pred, 8)
    assert np.array_equal(out.cpu().numpy(), want) and counts.tolist() == wc


def join_expected(dk, dd, fk, pr, pred, k):
    ok = np.isin(fk, dk[dd < pred["date_hi"]]) & (pr < pred["price_hi"])
    uk, inv = np.unique(fk[ok], return_inverse=True)
    s = np.zeros(len(uk), np.int64)
    np.add.at(s, inv, pr[ok])
    c = np.bincount(inv, minlength=len(uk))
    o = sorted(range(len(uk)), key=lambda i: (-int(s[i]), int(uk[i])))[:k]
    out = np.zeros((k, 3), np.int64)
    for r, i in enumerate(o):
        out[r] = uk[i], s[i], c[i]
    return out, [int(ok.sum()), len(uk)]


# price_hi = INT64_MAX takes the record form, anything below the 12-byte form;
# keys and prices at both ends, repeated and failing dimension rows
@pytest.mark.parametrize("nd,nf", [(1, 1), (1, 2047), (700, 1349), (1000, 3097), (5000, 20_000), (40_000, 100_000)])
@pytest.mark.parametrize("price_hi", [2**63 - 1, 2**63 - 2, 1000])
@pytest.mark.parametrize("k", [1, 16, 17, 300])
def test_join_topk_ends(cuda, nd, nf, price_hi, k):
    rng = np.random.default_rng(nd + nf + k)
    ends = np.array([-2**31, -2**31 + 1, -1, 0, 1, 2**31 - 2, 2**31 - 1])
    keys = np.concatenate([ends, rng.integers(-2**31, 2**31, max(nd // 2, 1))]).astype(np.int32)
    dk = rng.choice(keys, nd)  # keys repeat
    dd = rng.integers(0, 10, nd).astype(np.int32)
    fk = rng.choice(keys, nf)
    big = np.array([-2**63, -2**63 + 1, -5, 0, 999, 1000, 2**63 - 3, 2**63 - 2, 2**63 - 1])
    pr = np.where(rng.random(nf) < 0.01, rng.choice(big, nf), rng.integers(-10**6, 10**6, nf))
    if nf > 100:
        pr[rng.random(nf) < 0.2] = -7
    pred = dict(date_hi=5, price_hi=price_hi)
    with np.errstate(over="ignore"):
        want, wc = join_expected(dk, dd, fk, pr, pred, k)
    dt = {n: torch.from_numpy(v).cuda() for n, v in
          (("dim_key", dk), ("dim_date", dd), ("fact_fk", fk), ("fact_price", pr))}
    out, counts = capi.join_groupby_topk(dt, pred, k)
    assert counts.tolist() == wc and np.array_equal(out.cpu().numpy(), want)


# both routes there (table and sorted requests merged when at least three eighths
# of more than 2^18 rows are table rows) and back to request order (compaction when
# at most an eighth of the rows are requests, half above 2^18), repeated and
# out-of-range ids
@pytest.mark.parametrize("tn,rn", [(1, 1), (1, 4000), (5000, 5000), (5000, 4999), (5000, 5001), (4095, 1),
                                   (100_000, 3), (70_001, 300_007), (300_007, 70_001), (1024, 3072), (1025, 3072),
                                   (1024, 3073), (1023, 3074), (4097, 1), (8191, 1), (8192, 1), (4096, 4096),
                                   (4097, 12_287), (100_000, 31_072), (98_304, 163_841), (98_303, 163_842), (262_143, 1),
                                   (262_144, 1), (7000, 1000), (6999, 1001), (524_289, 2048), (700_001, 349_000),
                                   (1 << 20, 1 << 20), (524_288, 1_572_865)])
def test_gather_routes(cuda, tn, rn):
    rng = np.random.default_rng(tn + rn)
    table = rng.integers(-2**63, 2**63 - 1, tn)
    table[0] = -1
    rid = rng.integers(0, tn, rn).astype(np.int64)
    rid[rng.random(rn) < 0.1] = tn
    rid[rng.random(rn) < 0.05] = 2**32 - 1
    rid[rng.random(rn) < 0.05] = 0x7FFFFFFF
    out = torch.empty(rn, dtype=torch.int64, device="cuda")
    capi.ogather_u64(torch.from_numpy(table).cuda(), tn, torch.from_numpy(rid.astype(np.uint32).view(np.int32)).cuda(),
                     rn, out)
    want = np.where(rid < tn, table[np.minimum(rid, tn - 1)], 0)
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("nb,pn", [(1, 1), (3000, 1097), (1000, 3097), (20_000, 70_001), (100_001, 100_001)])
@pytest.mark.parametrize("bigint", [False, True])
def test_join_pkfk_ends(cuda, nb, pn, bigint):
    rng = np.random.default_rng(nb + pn)
    lim = 2**63 if bigint else 2**31
    dt = np.int64 if bigint else np.int32
    dom = np.unique(np.concatenate([[-lim, -lim + 1, -1, 0, lim - 2, lim - 1], rng.integers(-lim, lim, 2 * nb)]))
    bk = rng.permutation(dom)[:nb].astype(dt)  # unique
    pk = rng.choice(dom, pn).astype(dt)
    bm, pm = (rng.random(nb) < 0.7).astype(np.uint8), (rng.random(pn) < 0.7).astype(np.uint8)
    b, p, cnt = capi.ojoin_pkfk(torch.from_numpy(bk).cuda(), torch.from_numpy(bm).cuda(), torch.from_numpy(pk).cuda(),
                                torch.from_numpy(pm).cuda(), BIGINT if bigint else INTEGER)
    b, p, cnt = b.cpu().numpy(), p.cpu().numpy(), cnt.tolist()
    o = np.argsort(bk)
    at = np.minimum(np.searchsorted(bk[o], pk), nb - 1)
    hit = (bk[o][at] == pk) & (pm != 0) & (bm[o][at] != 0)
    c = int(hit.sum())
    assert cnt == [c, 0] and (b[c:] == -1).all() and (p[c:] == -1).all()
    assert sorted(p[:c].tolist()) == np.flatnonzero(hit).tolist()
    assert (b[:c] == o[at[p[:c]]]).all() and (np.diff(pk[p[:c]]) >= 0).all()


# BIGINT groups: the key 2^63 - 1 shares its word with the rows left out
@pytest.mark.parametrize("n", [1, 4095, 4097, 12_289, 100_003])
@pytest.mark.parametrize("ns,with_count", [(0, True), (1, True), (1, False), (2, False)])
def test_groupby_bigint_last_key(cuda, n, ns, with_count):
    rng = np.random.default_rng(n + ns)
    top = 2**63 - 1
    for share, masked in ((0.0, 0.5), (0.3, 0.5), (1.0, 0.5), (0.3, 1.0), (0.3, 0.0)):
        keys = np.where(rng.random(n) < share, top, rng.choice(np.array([-2**63, -1, 0, 7, top - 1]), n))
        vals = [rng.integers(-2**62, 2**62, n) for _ in range(ns)]
        mask = rng.random(n) >= masked
        ok, osum, ocnt, cnt = capi.ogroupby(torch.from_numpy(keys).cuda(), BIGINT, n,
                                            [torch.from_numpy(v).cuda() for v in vals], with_count,
                                            torch.from_numpy(mask.astype(np.uint8)).cuda())
        uk, inv = np.unique(keys[mask], return_inverse=True)
        g = len(uk)
        assert cnt.tolist() == [g, 0]
        ok = ok.cpu().numpy()
        assert np.array_equal(ok[:g], uk) and not ok[g:].any()
        with np.errstate(over="ignore"):
            for a, v in zip(osum, vals):
                s = np.zeros(g, np.int64)
                np.add.at(s, inv, v[mask])
                a = a.cpu().numpy()
                assert np.array_equal(a[:g], s) and not a[g:].any()
        if with_count:
            c = ocnt.cpu().numpy()
            assert np.array_equal(c[:g], np.bincount(inv, minlength=g)) and not c[g:].any()


# ORDER BY in each record form (key bits <= 32, <= 64, <= 96, <= 128), few
# distinct values so that the network's arrangement of ties shows, against the
# network itself with strict compares
@pytest.mark.parametrize("n", [1, 2, 100, 4095, 4097, 20_000])
@pytest.mark.parametrize("types", [(SMALLINT,), (INTEGER,), (SMALLINT, SMALLINT), (BIGINT,), (DATE, INTEGER),
                                   (BIGINT, DATE), (DATE, BIGINT), (INTEGER, SMALLINT, INTEGER),
                                   (BIGINT, BIGINT), (BIGINT, SMALLINT, INTEGER)])
def test_sort_columns_forms(cuda, n, types):
    rng = np.random.default_rng(n + len(types))
    dts = {SMALLINT: np.int16, INTEGER: np.int32, BIGINT: np.int64, DATE: np.uint32}
    cap = capi.next_pow2(n)
    for flip in (False, True):
        asc = [(i % 2 == 0) != flip for i in range(len(types))]
        host, rank = [], np.zeros(cap, np.int64)
        for t, a in zip(types, asc):
            ii = np.iinfo(dts[t])
            pool = np.array([ii.min, ii.min + 1, ii.max - 1, ii.max, 0, 3], dts[t])
            c = np.full(cap, ii.max if a else ii.min, dts[t])
            c[:n] = rng.choice(pool, n)
            host.append(c)
            u, inv = np.unique(c, return_inverse=True)
            rank = rank * len(u) + (inv if a else len(u) - 1 - inv)
        idx = np.arange(cap)
        k = 2
        while k <= cap:
            j = k // 2
            while j:
                r, x = rank.reshape(-1, 2, j), idx.reshape(-1, 2, j)
                up = ((np.arange(r.shape[0]) * 2 * j) & k)[:, None] == 0
                swap = np.where(up, r[:, 0] > r[:, 1], r[:, 0] < r[:, 1])
                for y in (r, x):
                    lo, hi = y[:, 0].copy(), y[:, 1].copy()
                    y[:, 0], y[:, 1] = np.where(swap, hi, lo), np.where(swap, lo, hi)
                j //= 2
            k *= 2
        signed = {SMALLINT: np.int16, INTEGER: np.int32, BIGINT: np.int64, DATE: np.int32}
        dev = [torch.from_numpy(c.view(signed[t]).copy()).cuda() for c, t in zip(host, types)]
        got = capi.sort_columns(dev, types, asc, n)
        assert np.array_equal(got.cpu().numpy(), idx), (types, asc)
        for d, c, t in zip(dev, host, types):
            assert np.array_equal(d.cpu().numpy(), c[idx].view(signed[t]))


# a batch's sorts of more than 2^20 rows run outside its persistent launch
def test_batch_large_sort(cuda):
    import velodb_b200
    from velodb_b200._lib import check

    def items():
        out = []
        for i, n in enumerate([(1 << 20) + 1, 5000, 1 << 20, 1_500_000]):
            g = torch.Generator(device="cuda")
            g.manual_seed(n)
            cap = capi.next_pow2(n)
            it = dict(kind="compact" if i == 1 else "sort", n=n,
                      keys=torch.randint(-2**63, 2**63 - 1, (cap,), generator=g, device="cuda"),
                      pay=torch.arange(cap, device="cuda", dtype=torch.int32))
            if i == 1:
                it["marks"] = (torch.rand(cap, generator=g, device="cuda") < 0.3).to(torch.uint8)
                it["count"] = torch.zeros(1, dtype=torch.int64, device="cuda")
            out.append(it)
        return out

    a, ref = items(), items()
    b = capi.Batch(a)
    b.launch()
    b.status()
    for x, r in zip(a, ref):
        if r["kind"] == "sort":
            capi.osort_kp(r["keys"], r["pay"], r["n"])
            assert torch.equal(x["keys"], r["keys"]) and torch.equal(x["pay"], r["pay"])
    L = velodb_b200.lib()
    check(L.velo_batch_set_timeout(b.ptr, 2_000_000), "velo_batch_set_timeout")
    check(L.velo_batch_inject_unmet_wait(b.ptr, 3), "velo_batch_inject_unmet_wait")  # a large one
    b.launch()
    with pytest.raises(velodb_b200.VeloError) as e:
        b.status()
    assert e.value.status == -4  # VELO_ETIMEDOUT
    b.close()


# plain compactions around the rule that gives one more fused level (2^20 rows)
@pytest.mark.parametrize("n", [(1 << 19) + 3, (1 << 20) - 5, 1 << 20, (1 << 20) + 3])
def test_compaction_level_rule(cuda, n):
    rng = np.random.default_rng(n)
    cap = capi.next_pow2(n)
    keys, pay = W.sort_kp(n, seed=n)
    marks = (rng.random(n) < 0.4).astype(np.uint8)
    k, p, m = capi.to_dev_u64(keys, cap), capi.to_dev_u32(pay, cap), capi.to_dev_u8(marks, cap)
    cnt = capi.ocompact_kpm(k, p, m, n)
    c = int(marks.sum())
    keep = marks != 0
    assert int(cnt.item()) == c
    assert np.array_equal(capi.host_u64(k, c), keys[keep]) and np.array_equal(capi.host_u32(p, c), pay[keep])
    tail = capi.host_u64(k, cap)[c:]  # the other rows and the padding, re-routed
    assert np.array_equal(np.sort(tail), np.sort(np.concatenate([keys[~keep], np.full(cap - n, ~np.uint64(0))])))


# blocks of padding alone are passed over: one and a few rows past a power of
# two (whole blocks of every phase are padding), the last row of a block, and
# the three-CTA form; the passes' results over all 2^k rows
@pytest.mark.parametrize("n", [4097, 8191, (9 << 13) + 3, (1 << 17) + 5, 5 << 16, (5 << 16) + 1, (1 << 21) - (1 << 18),
                               (1 << 20) + 4097, (5 << 19) + 1])
def test_blocks_of_padding(cuda, orc, n):
    rng = np.random.default_rng(n)
    cap = capi.next_pow2(n)
    rec, marks = np.full((cap, 16), 255, np.uint8), np.zeros(cap, np.uint8)
    keys, pay = rng.integers(0, 2**63, n).astype(np.uint64), np.arange(n, dtype=np.uint32)
    rec[:n, :8] = keys.view(np.uint8).reshape(n, 8)
    rec[:n, 8:12] = pay.view(np.uint8).reshape(n, 4)
    for density in (0.3, 1.0):
        marks[:n] = rng.random(n) < density
        want, wm, wc = orc.ocompact(rec, marks)
        k, p, m = capi.to_dev_u64(keys, cap), capi.to_dev_u32(pay, cap), capi.to_dev_u8(marks[:n], cap)
        count = int(capi.ocompact_kpm(k, p, m, n).item())
        assert count == wc and np.array_equal(m.cpu().numpy(), wm)
        assert np.array_equal(capi.host_u64(k), np.ascontiguousarray(want[:, :8]).view(np.uint64).reshape(-1))
        assert np.array_equal(capi.host_u32(p), np.ascontiguousarray(want[:, 8:12]).view(np.uint32).reshape(-1))
    for types, asc in (((BIGINT,), (True,)), ((INTEGER, DATE), (False, True)), ((BIGINT, DATE), (False, False))):
        dts = {INTEGER: np.int32, BIGINT: np.int64, DATE: np.uint32}
        cols = [rng.integers(0, 50, n).astype(dts[t]) for t in types]
        cols[0][: n // 3] = np.iinfo(dts[types[0]]).max  # the padding's own key
        want, widx = orc.bitonic_sort_cols(cols, types, asc, n)
        dev = []
        for c in cols:
            x = np.zeros(cap, c.dtype)
            x[:n] = c
            dev.append(torch.from_numpy(x.view(np.int32) if x.dtype == np.uint32 else x).cuda())
        idx = capi.sort_columns(dev, types, asc, n)
        assert np.array_equal(idx.cpu().numpy(), widx), (types, asc)
        for d, w in zip(dev, want):
            assert np.array_equal(d.cpu().numpy(), w.view(d.cpu().numpy().dtype))
