"""GPU parity of the oblivious filter + group-by pipeline against the oracle
(exact int64 sums), through the C ABI."""
import numpy as np
import pytest
import torch

from velodb_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu


def run_gpu(cols, pred, G=8, reveal=False):
    n = len(cols["qty"])
    d = capi.lineitem_to_device(cols)
    out, counts = capi.filter_groupby(d, n, pred, G, reveal_count=reveal)
    torch.cuda.synchronize()
    return out.cpu().numpy(), counts.cpu().numpy()


def check(orc, cols, pred, G=8, reveal=False):
    out, counts = run_gpu(cols, pred, G, reveal)
    g, keys, sums = orc.filter_groupby(cols, pred, max_groups=G)
    mask = ((cols["shipdate"] >= pred["ship_lo"]) & (cols["shipdate"] <= pred["ship_hi"])
            & (cols["disc"] >= pred["disc_lo"]) & (cols["disc"] <= pred["disc_hi"])
            & (cols["qty"] >= pred["qty_lo"]) & (cols["qty"] <= pred["qty_hi"]))
    assert int(counts[0]) == int(mask.sum())
    assert int(counts[1]) == g
    m = min(g, G)
    assert np.array_equal(out[:m, 0], keys[:m].astype(np.int64))
    assert np.array_equal(out[:m, 1:], sums[:m])
    assert not out[m:].any()


@pytest.mark.parametrize("n", [1, 7, 100, 2047, 2048, 4096, 5000, 65536, 100_003])
def test_filter_groupby_small(cuda, orc, n):
    cols = W.lineitem(n, seed=W.SEED_LINEITEM + n)
    check(orc, cols, W.LINEITEM_PRED)
    check(orc, cols, dict(ship_lo=0, ship_hi=2556, disc_lo=0, disc_hi=10, qty_lo=1, qty_hi=50))  # everything


def test_filter_groupby_selectivities(cuda, orc):
    cols = W.lineitem(300_000, seed=99)
    for pred in [dict(ship_lo=0, ship_hi=-1, disc_lo=0, disc_hi=10, qty_lo=1, qty_hi=50),  # nothing passes
                 dict(ship_lo=5, ship_hi=6, disc_lo=3, disc_hi=3, qty_lo=1, qty_hi=2),      # a handful
                 W.LINEITEM_PRED]:
        check(orc, cols, pred)
        check(orc, cols, pred, reveal=True)


def test_filter_groupby_bound_smaller_than_groups(cuda, orc):
    cols = W.lineitem(50_000, seed=5)
    check(orc, cols, W.LINEITEM_PRED, G=4)  # 6 groups, 4 slots: first 4 in key order, count says 6


def test_filter_groupby_config1_full(cuda, orc):
    cols = W.lineitem()  # 6,001,215 rows
    check(orc, cols, W.LINEITEM_PRED)
    check(orc, cols, W.LINEITEM_PRED, reveal=True)


def test_filter_groupby_wide_bands_use_three_word_records(cuda, orc):
    # bands too wide for the packed two-word layout: the three-word path
    cols = W.lineitem(70_000, seed=17)
    check(orc, cols, dict(ship_lo=0, ship_hi=2000, disc_lo=-(1 << 20), disc_hi=1 << 20, qty_lo=-(2**31),
                          qty_hi=2**31 - 1))


def test_filter_groupby_band_edges_in_packed_layout(cuda, orc):
    # qty band of 10 bits and disc band of 5 bits (15 packed bits, the limit),
    # with values at both edges of each band
    n = 20_000
    rng = np.random.default_rng(4)
    cols = W.lineitem(n, seed=23)
    cols["qty"] = rng.choice(np.array([-7, -7 + 1023, 100], np.int32), n)
    cols["disc"] = rng.choice(np.array([3, 3 + 31, 10], np.int32), n)
    check(orc, cols, dict(ship_lo=0, ship_hi=2556, disc_lo=3, disc_hi=34, qty_lo=-7, qty_hi=1016))


def test_stage_timing_reports_four_stages(cuda):
    cols = W.lineitem(100_000, seed=3)
    d = capi.lineitem_to_device(cols)
    capi.set_stage_timing(True)
    try:
        capi.filter_groupby(d, 100_000, W.LINEITEM_PRED)
        t = capi.last_stage_times()
    finally:
        capi.set_stage_timing(False)
    assert len(t) == 4 and all(x >= 0 for x in t) and sum(t) > 0


def rows_passing(n, rows, flags, seed):
    """Lineitem columns of which `rows` rows pass the whole-range predicate."""
    rng = np.random.default_rng(seed)
    c = W.lineitem(n, seed=seed)
    c["shipdate"][:] = 5000
    c["shipdate"][rng.permutation(n)[:rows]] = 10
    key = rng.choice(np.array(flags), n)
    c["flag1"], c["flag2"] = (key >> 8).astype(np.uint8), (key & 255).astype(np.uint8)
    return c


ANY = dict(ship_lo=0, ship_hi=2556, disc_lo=0, disc_hi=10, qty_lo=1, qty_hi=50)


def key_sort_rows(d, n, G, reveal):
    """log2 rows of the call's sort passes, and whether it compacts."""
    capi.set_pass_timing(True)
    try:
        capi.clear_pass_times()
        capi.filter_groupby(d, n, ANY, G, reveal_count=reveal)
        t = capi.last_pass_times()
    finally:
        capi.set_pass_timing(False)
    return max(x[1] for x in t if not x[0].startswith("compact")), any(x[0].startswith("compact") for x in t)


# with the count revealed, few passing rows are sorted alone: the sort works on
# next_pow2(rows) key words (4096 at least, one tile), not on n / 2
@pytest.mark.parametrize("n,rows", [(1_000_001, 10_000), (3_000_001, 60_000), (6_001_215, 300_000)])
def test_revealed_count_sorts_fewer_rows(cuda, n, rows):
    d = capi.lineitem_to_device(rows_passing(n, rows, (65, 66, 300), seed=n))
    assert key_sort_rows(d, n, 8, True) == (max(12, (rows - 1).bit_length()), True)
    assert key_sort_rows(d, n, 8, False) == (((n + 1) // 2 - 1).bit_length(), False)


# the rule's edges (2^19..2^22 key words: next_pow2(rows) up to half of them; no
# more than 2^18 words are sorted whole), no row, one row, every row; 0xFFFF is
# also the mark of a row that fails
@pytest.mark.parametrize("n,rows", [(600_001, 0), (600_001, 1), (600_001, 1 << 18), (600_001, (1 << 18) + 1),
                                    (600_001, 600_001), (1_200_003, 1 << 19), (1_200_003, (1 << 19) + 1),
                                    (2_300_001, 1 << 20), (2_300_001, (1 << 20) + 1), (4_300_001, 70_000),
                                    (4_300_001, 1 << 21), ((1 << 21) + 1, 100), (1 << 20, 100), ((1 << 19) + 1, 100),
                                    (1 << 19, 100)])
@pytest.mark.parametrize("flags,G", [((65, 0xFFFF), 1), ((0xFFFF,), 8), (tuple(range(0, 65536, 257)), 16)])
def test_revealed_count_changes_no_result(cuda, n, rows, flags, G):
    c = rows_passing(n, rows, flags, seed=n + rows + G)
    d = capi.lineitem_to_device(c)
    plain = capi.filter_groupby(d, n, ANY, G)
    revealed = capi.filter_groupby(d, n, ANY, G, reveal_count=True)
    torch.cuda.synchronize()
    for a, b in zip(plain, revealed):
        assert torch.equal(a, b)
    key = c["flag1"].astype(np.int64) * 256 + c["flag2"]
    keys, counts = np.unique(key[c["shipdate"] == 10], return_counts=True)
    m = min(G, len(keys))
    out = plain[0].cpu().numpy()
    assert plain[1].tolist() == [rows, len(keys)]
    assert np.array_equal(out[:m, 0], keys[:m]) and np.array_equal(out[:m, 1], counts[:m]) and not out[m:].any()


def test_revealed_count_in_a_captured_stream(cuda):
    # a stream that is being captured cannot wait for the count: the whole sort
    n = 1_000_001
    d = capi.lineitem_to_device(rows_passing(n, 5000, (65, 66), seed=1))
    want = capi.filter_groupby(d, n, ANY, 8)
    sc = torch.empty(capi.filter_groupby_scratch_bytes(n, 8), dtype=torch.uint8, device="cuda")
    out, counts = torch.zeros_like(want[0]), torch.zeros_like(want[1])
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        capi.filter_groupby(d, n, ANY, 8, reveal_count=True, scratch=sc, out=out, counts=counts)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want[0]) and torch.equal(counts, want[1])


# key words at the edges of the tile rules (2^11, 2^12 of one tile; with the count
# revealed 2^18 | 2^19 and 2^21 | 2^22 of the next tile)
@pytest.mark.parametrize("words", [2047, 2048, 2049, 4096, 4097, 8193, 1 << 18, (1 << 18) + 1, 1 << 21, (1 << 21) + 1])
@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("reveal", [False, True])
def test_filter_groupby_key_tiles(cuda, words, odd, reveal):
    n = 2 * words - odd
    c = rows_passing(n, n - n // 5, tuple(range(0, 65536, 4369)), seed=n)
    out, counts = run_gpu(c, ANY, 16, reveal)
    key = c["flag1"].astype(np.int64) * 256 + c["flag2"]
    ok = c["shipdate"] == 10
    keys, num = np.unique(key[ok], return_counts=True)
    assert counts.tolist() == [int(ok.sum()), len(keys)] and len(keys) == 16
    assert np.array_equal(out[:, 0], keys) and np.array_equal(out[:, 1], num)
    price = np.zeros(65536, np.int64)
    np.add.at(price, key[ok], c["price"][ok].astype(np.int64))
    assert np.array_equal(out[:, 3], price[keys])
