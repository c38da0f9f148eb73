"""GPU parity of the network sorts with each load tune switched on: the
bulk-copy merge prefetch (velo_set_merge_pipeline) and the tensor-map tile
loads of the merge and fused global passes (velo_set_tensor_tile_loads).
Both keep the network, so the results are bit-exact against the oracle, and
the pipelines that sort inside (join, group-by) equal their plain runs."""
import numpy as np
import pytest
import torch

from velodb_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu

ALL_ONES = 2**64 - 1


@pytest.fixture(params=sorted(capi.TUNES))
def tune(request):
    switch = capi.TUNES[request.param]
    switch(True)
    try:
        yield request.param
    finally:
        switch(False)
    assert capi.tensor_tile_status() == 0


def gpu_sort_kp(keys, pay):
    n = len(keys)
    cap = capi.next_pow2(n)
    k, p = capi.to_dev_u64(keys, cap), capi.to_dev_u32(pay, cap)
    capi.osort_kp(k, p, n)
    torch.cuda.synchronize()
    return capi.host_u64(k, cap), capi.host_u32(p, cap)


def gpu_sort_records(words, mask, strict):
    n = len(words[0])
    cap = capi.next_pow2(n)
    ds = [capi.to_dev_u64(w, cap) for w in words]
    capi.osort_records(ds, n, mask, strict=strict)
    torch.cuda.synchronize()
    return [capi.host_u64(d, cap) for d in ds]


# 2^13 rows: one global pass of one level; 65,537 and 300,001 rows: a
# partial last tile; 2^20: global passes of 1..8 levels
@pytest.mark.parametrize("n", [8192, 65_537, 300_001, 1 << 20])
def test_sort_kp_with_tune(cuda, orc, tune, n):
    keys, pay = W.sort_kp(n, seed=W.SEED_SORT + 3 * n)
    keys[: n // 3] = keys[n // 2]  # ties: the arrangement of equal keys is the network's
    gk, gp = gpu_sort_kp(keys, pay)
    ok, op = orc.bitonic_kp(keys, pay)
    assert np.array_equal(gk, ok) and np.array_equal(gp, op)


def record_case(words, seed):
    n = (1 << 19) + 123
    ws = [W.splitmix64(seed + x, n, x) for x in range(words)]
    ws[0] = ws[0] & np.uint64(0xFFFF0000FFFFFFFF)  # equal masked keys
    return ws


# Strict record sorts order ties as the oracle's network does, so they are
# bit-exact against it; the default (non-strict) sorts may exchange equal keys
# in descending blocks, so their keys match the oracle's and their whole rows
# match the same sort with the tune off.
@pytest.mark.parametrize("words,mask", [(2, 0xFFFFFFFF00000000), (2, ALL_ONES), (3, 0xFFFF800000000000)])
@pytest.mark.parametrize("strict", [True, False])
def test_sort_records_with_tune(cuda, orc, tune, words, mask, strict):
    ws = record_case(words, 11)
    got = gpu_sort_records(ws, mask, strict)
    want = orc.bitonic_records(ws, 1, [mask], [ALL_ONES] * words)
    if strict:
        for g, w in zip(got, want):
            assert np.array_equal(g, w)
        return
    assert np.array_equal(got[0] & np.uint64(mask), want[0] & np.uint64(mask))
    capi.TUNES[tune](False)
    plain = gpu_sort_records(ws, mask, strict)
    for g, w in zip(got, plain):
        assert np.array_equal(g, w)


@pytest.mark.parametrize("words,mask", [(1, ALL_ONES), (2, 0xFFFFFFFF00000000), (3, 0xFFFF800000000000)])
def test_sort_records_strict_without_tune(cuda, orc, words, mask):
    ws = record_case(words, 29)
    got = gpu_sort_records(ws, mask, True)
    want = orc.bitonic_records(ws, 1, [mask], [ALL_ONES] * words)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


def test_join_and_groupby_with_tune(cuda, tune):
    dim, fact = W.join_tables()
    dt = capi.join_to_device(dim, fact)
    cols = W.lineitem()
    dc = capi.lineitem_to_device(cols)
    n = W.LINEITEM_ROWS

    def both():
        jo, jc = capi.join_groupby_topk(dt, W.JOIN_PRED, W.JOIN_TOPK)
        go, gc = capi.filter_groupby(dc, n, W.LINEITEM_PRED, W.LINEITEM_GROUP_BOUND)
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in (jo, jc, go, gc)]

    with_tune = both()
    capi.TUNES[tune](False)
    plain = both()
    for a, b in zip(with_tune, plain):
        assert np.array_equal(a, b)


# the kernel of each tune, and one call of every operator whose sort runs in
# 4096-row tiles of 12-byte rows or records of up to three words: n leaves
# whole tiles of padding, so the networks are trimmed or pass over padding
KERNEL = {"merge_pipeline": "k_merge_pipe", "tensor_tile_loads": "k_sort_pass_tma"}


def _i64(n, seed, span):
    return torch.from_numpy((W.splitmix64(seed, n, 0) % np.uint64(span)).astype(np.int64)).cuda()


def op_sort():
    keys, pay = W.sort_kp(300_001, seed=5)
    return gpu_sort_kp(keys, pay)


def op_order_by(types):
    n = 300_001
    cap = capi.next_pow2(n)
    dt = {5: torch.int64, 7: torch.float64, 10: torch.int32}
    cols = []
    for i, t in enumerate(types):
        c = torch.zeros(cap, dtype=dt[t], device="cuda")
        c[:n] = _i64(n, 31 + i, 5000).to(dt[t])  # equal keys: their order is seen
        cols.append(c)
    idx = capi.sort_columns(cols, types, [i % 2 == 0 for i in range(len(types))], n)
    return cols + [idx]


def op_join_topk():
    dim, fact = W.join_tables(70_000, 300_001, seed=9)
    return capi.join_groupby_topk(capi.join_to_device(dim, fact), W.JOIN_PRED, 10)


def op_join_topk_records():
    dim, fact = W.join_tables(70_000, 300_001, seed=9)
    return capi.join_groupby_topk(capi.join_to_device(dim, fact), dict(W.JOIN_PRED, price_hi=2**63 - 1), 10)


def op_join_pkfk():
    return capi.ojoin_pkfk(torch.randperm(50_000, device="cuda", generator=_gen(3)), None, _i64(300_001, 8, 60_000),
                           None, 5)


def op_join_mn():
    return capi.ojoin_mn(_i64(50_000, 7, 50_000), None, _i64(250_001, 8, 50_000), None, 5, 400_000)


def op_join_hash():
    return capi.ohash_join(torch.randperm(50_000, device="cuda", generator=_gen(4)), None, _i64(250_001, 8, 60_000),
                           None, 5)


def op_group_by(key_type, n_sums):
    n = 300_001
    keys = _i64(n, 2, 9000).to(torch.int64 if key_type == 5 else torch.int32)
    out = capi.ogroupby(keys, key_type, n, sums=[_i64(n, 20 + i, 1000) for i in range(n_sums)])
    return [out[0], *out[1], out[2], out[3]]


def op_gather():
    n_table, n_req = 300_001, 100_003
    out = torch.empty(n_req, dtype=torch.int64, device="cuda")
    capi.ogather_u64(_i64(n_table, 1, 2**40), n_table, _i64(n_req, 2, n_table + 2).to(torch.int32), n_req, out)
    return [out]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


TUNED_OPS = {
    "sort": op_sort,
    "order by 32 bits": lambda: op_order_by([10]),
    "order by 64 bits": lambda: op_order_by([5]),
    "order by 96 bits": lambda: op_order_by([7, 10]),
    "order by 128 bits": lambda: op_order_by([5, 7]),
    "join top-k": op_join_topk,
    "join top-k, no price bound": op_join_topk_records,
    "PK-FK join": op_join_pkfk,
    "many-to-many join": op_join_mn,
    "hash join": op_join_hash,
    "GROUP BY BIGINT, sum": lambda: op_group_by(5, 1),
    "GROUP BY INTEGER": lambda: op_group_by(4, 0),
    "gather": op_gather,
}


@pytest.mark.parametrize("op", sorted(TUNED_OPS))
def test_tuned_kernels_run(cuda, tune, op):
    from torch.profiler import ProfilerActivity, profile

    def call():
        out = TUNED_OPS[op]()
        torch.cuda.synchronize()
        return [np.asarray(t.cpu()) if torch.is_tensor(t) else t for t in out]

    call()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        tuned = call()
    names = {e.key for e in prof.key_averages()}
    assert any("k_sort_pass" in x for x in names)
    assert any(KERNEL[tune] in x for x in names), sorted(names)
    capi.TUNES[tune](False)
    for a, b in zip(tuned, call()):
        assert np.array_equal(a, b)
